"""The FP64 projector products of small blocks (one and many k-points, spinors) against numpy on the host: band and
projector counts around the tiles of 8, 16 and 32, plane-wave counts that are no multiple of 4 or 16, several slices.

Bound: a sum of K products of n-bit values errs by at most about K u |a| |b| (u = 2^-53); the two products chain, so
the result is compared at (npw + nkb) u times the sum of magnitudes."""
from __future__ import annotations

import numpy as np
import pytest

U = 2.0 ** -53


def _setup(pkg, nat, nh, nks, npol=1, seed=1):
    import torch
    P = pkg.pwdft
    rng = np.random.default_rng(seed)
    k = rng.uniform(-0.5, 0.5, size=(nks, 3))
    b = P.PWBasisK(5.13, np.diag([1.0, 1.1, 0.9]), 24.0, k)
    ld = b.npwk_max + 2
    h = P.HamiltPW(b, P.PREC_FP64)
    vkb = [rng.standard_normal((nat * nh, ld)) + 1j * rng.standard_normal((nat * nh, ld)) for _ in range(nks)]
    if npol == 1:
        d = rng.uniform(-1, 1, size=(1, nat, nh, nh))
        h.set_veff(torch.zeros(b.nxyz, dtype=torch.float64, device="cuda"))
        h.set_deeq([nat], [nh], torch.from_numpy(d).cuda())
    else:
        d = rng.standard_normal((4, nat, nh, nh)) + 1j * rng.standard_normal((4, nat, nh, nh))
        h.set_veff_nc(torch.zeros(4, b.nxyz, dtype=torch.float64, device="cuda"))
        h.set_deeq_nc([nat], [nh], torch.from_numpy(d).cuda())
    for ik in range(nks):
        h.set_vkb(ik, torch.from_numpy(vkb[ik]).cuda())
    return b, h, vkb, d, ld


def _psi(b, ik, rows, ld, seed):
    rng = np.random.default_rng(seed)
    psi = np.zeros((rows, ld), dtype=np.complex128)
    n = int(b.npwk[ik])
    psi[:, :n] = rng.standard_normal((rows, n)) + 1j * rng.standard_normal((rows, n))
    return psi


def _want(b, ik, vkb, d, psi):
    """(H_nl psi, bound on its error): ps_k = sum_x D(x, k) becp_x."""
    n, (nat, nh) = int(b.npwk[ik]), d.shape[1:3]
    v, p = vkb[:, :n], psi[:, :n]
    becp = (p @ v.conj().T).reshape(len(p), nat, nh)
    ps = np.einsum("axk,bax->bak", d[0], becp).reshape(len(p), -1)
    mag = np.einsum("axk,bax->bak", np.abs(d[0]), (np.abs(p) @ np.abs(v).T).reshape(len(p), nat, nh)).reshape(len(p), -1)
    return ps @ v, 8 * (n + nat * nh) * U * (mag @ np.abs(v))


@pytest.mark.gpu
@pytest.mark.parametrize("nat,nh,nb", [(1, 1, 1), (1, 4, 8), (2, 8, 9), (3, 5, 16), (2, 13, 17), (5, 8, 33), (3, 18, 47),
                                       (2, 33, 3), (2, 8, 48), (4, 9, 61), (1, 6, 130), (2, 18, 47), (2, 17, 31), (4, 8, 1)])
def test_small_products(pkg, nat, nh, nb):
    torch = pytest.importorskip("torch")
    b, h, vkb, d, ld = _setup(pkg, nat, nh, 1)
    psi = _psi(b, 0, nb, ld, 7)
    pd = torch.from_numpy(psi).cuda()
    hd = torch.zeros_like(pd)
    for _ in range(2):  # the second call finds the tile counters as the first one left them
        hd.zero_()
        h.hpsi_part(0, pd, hd, nb, ld, 2)
    want, bound = _want(b, 0, vkb[0], d, psi)
    assert np.all(np.abs(hd.cpu().numpy()[:, :want.shape[1]] - want) <= bound)


@pytest.mark.gpu
@pytest.mark.parametrize("nk,nb", [(2, 1), (3, 12), (5, 31), (128, 3)])
def test_small_products_of_a_batch(pkg, nk, nb):
    torch = pytest.importorskip("torch")
    b, h, vkb, d, ld = _setup(pkg, 2, 8, nk)
    psis = [_psi(b, ik, nb, ld, ik) for ik in range(nk)]
    pd = [torch.from_numpy(p).cuda() for p in psis]
    hd = [torch.zeros_like(p) for p in pd]
    h.hpsi_kbatch(range(nk), pd, hd, nb, ld)
    for ik in range(0, nk, max(1, nk // 3)):
        want, bound = _want(b, ik, vkb[ik], d, psis[ik])
        n = want.shape[1]
        kin = b.gk2_k(ik) * b.tpiba2 * psis[ik][:, :n]
        assert np.all(np.abs(hd[ik].cpu().numpy()[:, :n] - (want + kin)) <= bound + 8 * U * np.abs(kin))


@pytest.mark.gpu
@pytest.mark.parametrize("nb", [1, 5, 20])
def test_small_products_of_spinors(pkg, nb):
    torch = pytest.importorskip("torch")
    b, h, vkb, d, ld = _setup(pkg, 2, 7, 1, npol=2)
    psi = _psi(b, 0, 2 * nb, ld, 11)
    pd = torch.from_numpy(psi).cuda()
    hd = torch.zeros_like(pd)
    h.hpsi_nc(0, pd, hd, nb, ld)
    n = int(b.npwk[0])
    v, p = vkb[0][:, :n], psi[:, :n]
    becp = (p @ v.conj().T).reshape(nb, 2, 2, 7)
    mag = (np.abs(p) @ np.abs(v).T).reshape(nb, 2, 2, 7)
    up = np.einsum("akx,bax->bak", d[0], becp[:, 0]) + np.einsum("akx,bax->bak", d[1], becp[:, 1])
    dn = np.einsum("akx,bax->bak", d[2], becp[:, 0]) + np.einsum("akx,bax->bak", d[3], becp[:, 1])
    mu = np.einsum("akx,bax->bak", abs(d[0]), mag[:, 0]) + np.einsum("akx,bax->bak", abs(d[1]), mag[:, 1])
    md = np.einsum("akx,bax->bak", abs(d[2]), mag[:, 0]) + np.einsum("akx,bax->bak", abs(d[3]), mag[:, 1])
    want = np.stack([up, dn], 1).reshape(2 * nb, -1) @ v + b.gk2_k(0) * b.tpiba2 * p
    bound = 16 * (n + 14) * U * (np.stack([mu, md], 1).reshape(2 * nb, -1) @ np.abs(v) + np.abs(want))
    assert np.all(np.abs(hd.cpu().numpy()[:, :n] - want) <= bound)
