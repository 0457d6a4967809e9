"""The local part of H|psi> on two-pass line transforms, every compiled edge as x, as z and on square planes,
run-time edges, odd band counts and several k-points, against the oracle (FP64 within 1e-12 relative, FP32 within
2e-5, the bars of test_gpu_hpsi.py).  The run descriptors it relies on: test_line_plan.py, on the host."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import hamilt_ref as H
from oracle.pw_basis_ref import PWBasisKRef

# (grid, bands): square and rectangular planes; the second factor of an edge is exercised as y and as z
GRIDS = [((16, 12, 15), 1), ((20, 20, 18), 3), ((24, 24, 27), 2), ((27, 27, 20), 5), ((30, 30, 32), 2),
         ((32, 25, 30), 3), ((36, 36, 40), 4), ((40, 40, 36), 1), ((45, 45, 50), 3), ((48, 48, 45), 2),
         ((50, 50, 48), 2), ((54, 54, 60), 2), ((60, 60, 54), 3), ((72, 36, 108), 3), ((75, 75, 72), 2),
         ((80, 80, 75), 1), ((81, 81, 80), 2), ((90, 90, 81), 1), ((100, 100, 90), 1), ((108, 108, 100), 1),
         ((120, 120, 24), 1), ((125, 125, 25), 1), ((135, 135, 27), 1), ((144, 144, 32), 1), ((150, 150, 30), 1),
         ((96, 64, 120), 1), ((64, 96, 125), 1), ((32, 125, 135), 1), ((125, 32, 144), 1), ((18, 150, 150), 1),
         ((25, 18, 160), 1), ((128, 16, 16), 2), ((8, 8, 8), 2)]
SPACING = 0.28  # bohr: the sphere's diameter is then about half of each edge at 30 Ry


def _setup(pkg, grid, nks=1):
    lat = np.diag(np.array(grid, dtype=float))
    k = np.array([[0.125, -0.375, 0.375], [0.0, 0.0, 0.0], [-0.25, 0.4, 0.1]])[:nks]
    b = pkg.pwdft.PWBasisK(SPACING, lat, 30.0, k, grid=grid)
    return b, PWBasisKRef(SPACING, lat, 30.0, k, grid=grid)


def _inputs(b, ik, nb, seed=3):
    rng = np.random.default_rng(seed)
    ld = b.npwk_max + 3
    npw = int(b.npwk[ik])
    psi = np.zeros((nb, ld), dtype=np.complex128)
    psi[:, :npw] = rng.standard_normal((nb, npw)) + 1j * rng.standard_normal((nb, npw))
    return rng.uniform(-2.0, 0.5, size=b.nxyz), psi, ld


def _oracle(ref, ik, veff, psi, nb, ld):
    h = H.HamiltPWRef(ref, ik, veff, np.zeros((0, ld), dtype=np.complex128), np.zeros((1, 0, 0, 0)), [], [])
    return h.hpsi_local(psi.reshape(-1), nb, ld)


def rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("grid,nb", GRIDS)
def test_local_pass_matches_oracle(pkg, grid, nb, prec):
    torch = pytest.importorskip("torch")
    P = pkg.pwdft
    b, ref = _setup(pkg, grid)
    veff, psi, ld = _inputs(b, 0, nb)
    h = P.HamiltPW(b, prec)
    h.set_veff(torch.from_numpy(veff).cuda())
    pd = torch.from_numpy(psi).to("cuda", torch.complex64 if prec else torch.complex128)
    hd = torch.full_like(pd, 7.0)
    h.hpsi_part(0, pd, hd, nb, ld, 1)
    torch.cuda.synchronize()
    out = hd.cpu().numpy().reshape(-1)
    assert rel(out, _oracle(ref, 0, veff, psi, nb, ld)) < (2e-5 if prec else 1e-12)
    assert np.all(out.reshape(nb, ld)[:, int(b.npwk[0]):] == 0)


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("grid", [(36, 36, 40), (72, 36, 108), (25, 18, 160)])
def test_kbatch_on_lines_matches_oracle(pkg, grid, prec):
    torch = pytest.importorskip("torch")
    P = pkg.pwdft
    b, ref = _setup(pkg, grid, 3)
    h = P.HamiltPW(b, prec)
    dt = torch.complex64 if prec else torch.complex128
    ins = [_inputs(b, ik, 5, seed=ik) for ik in range(3)]
    veff, ld = ins[0][0], ins[0][2]
    h.set_veff(torch.from_numpy(veff).cuda())
    h.set_chunk(2)  # 5 bands in chunks of 2, 2 and 1
    pd = [torch.from_numpy(i[1]).to("cuda", dt) for i in ins]
    hd = [torch.full_like(p, 7.0) for p in pd]
    h.hpsi_kbatch([0, 1, 2], pd, hd, 5, ld)
    torch.cuda.synchronize()
    for ik in range(3):
        assert rel(hd[ik].cpu().numpy().reshape(-1), _oracle(ref, ik, veff, ins[ik][1], 5, ld)) < (2e-5 if prec else 1e-12)


@pytest.mark.gpu
def test_kbatch_of_more_bands_than_a_launch_takes(pkg):
    """12 x 12 x 12 in FP32: the stick buffer holds more bands than gridDim.y; 70 000 bands of seven vectors."""
    torch = pytest.importorskip("torch")
    P = pkg.pwdft
    b, ref = _setup(pkg, (12, 12, 12))
    veff, psi, ld = _inputs(b, 0, 7)
    h = P.HamiltPW(b, P.PREC_MIXED)
    h.set_veff(torch.from_numpy(veff).cuda())
    pd = torch.from_numpy(psi).to("cuda", torch.complex64).repeat(10000, 1)
    hd = torch.full_like(pd, 7.0)
    h.hpsi_kbatch([0], [pd], [hd], len(pd), ld)
    want = torch.from_numpy(_oracle(ref, 0, veff, psi, 7, ld).reshape(7, ld)).cuda()
    diff = (hd.view(10000, 7, ld) - want).abs().max()
    assert float(diff / want.abs().max()) < 2e-5


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("grid,nb", [((18, 18, 18), 3), ((36, 45, 20), 2), ((75, 75, 16), 1), ((90, 96, 25), 1)])
def test_spinor_local_pass_matches_oracle(pkg, grid, nb, prec):
    torch = pytest.importorskip("torch")
    P = pkg.pwdft
    b, ref = _setup(pkg, grid)
    _, psi, ld = _inputs(b, 0, 2 * nb)
    v4 = np.random.default_rng(9).uniform(-1.0, 1.0, size=(4, b.nxyz))
    want = H.HamiltPWRefNC(ref, 0, list(v4), np.zeros((0, ld), dtype=np.complex128),
                           np.zeros((4, 0, 0, 0), dtype=np.complex128), [], []).hpsi(psi.reshape(-1), nb, ld)
    h = P.HamiltPW(b, prec)
    h.set_veff_nc(torch.from_numpy(v4).cuda())
    pd = torch.from_numpy(psi).to("cuda", torch.complex64 if prec else torch.complex128)
    hd = torch.full_like(pd, 7.0)
    h.hpsi_nc(0, pd, hd, nb, ld)
    torch.cuda.synchronize()
    assert rel(hd.cpu().numpy().reshape(-1), want) < (2e-5 if prec else 1e-12)
