"""psi -> rho on the line transforms against the oracle's loop over bands (1e-12 relative in FP64, 2e-5 in FP32):
square and rectangular planes, sums in shared memory and in the partial planes, bands without weight (skipped, also
when they hold NaN), rho added to, more partial planes than a later run of bands fills."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import hamilt_ref as H
from oracle.pw_basis_ref import PWBasisKRef

CASES = [((18, 18, 18), 1), ((20, 25, 32), 7), ((36, 36, 45), 33), ((72, 36, 50), 4), ((96, 96, 27), 3), ((125, 125, 16), 2),
         ((128, 128, 18), 3), ((144, 144, 16), 1), ((135, 64, 20), 2)]


@pytest.mark.gpu
def test_band_counts_on_one_handle(pkg):
    """The scratch of a handle serves both precisions and every band count (24 and 40 bands cut a plane into more
    partial sums than 25 or 48): the same bits as the call on a handle of its own, in any order."""
    torch = pytest.importorskip("torch")
    grid = (36, 36, 36)
    lat, k = np.diag(np.array(grid, dtype=float)), np.array([[0.125, -0.375, 0.375]])
    rng = np.random.default_rng(6)

    def basis():
        return pkg.pwdft.PWBasisK(0.28, lat, 30.0, k, grid=grid)
    shared = basis()
    ld = int(shared.npwk[0])
    psi = rng.standard_normal((48, ld)) + 1j * rng.standard_normal((48, ld))
    w = rng.uniform(0.1, 2.0, size=48)

    def rho(b, nb, prec):
        out = torch.zeros(b.nxyz, dtype=torch.float32 if prec else torch.float64, device="cuda")
        b.psi_to_rho(0, torch.from_numpy(psi).to("cuda", torch.complex64 if prec else torch.complex128), nb, ld, w[:nb], out)
        return out
    for nb, prec in ((25, 0), (24, 0), (3, 1), (40, 1), (1, 0), (48, 0), (40, 0), (48, 1), (24, 1)):
        assert torch.equal(rho(shared, nb, prec), rho(basis(), nb, prec)), (nb, prec)


@pytest.mark.gpu
def test_more_bands_than_a_launch_takes(pkg):
    """A 12 x 12 x 12 grid's stick buffer holds more bands than gridDim.y: seven bands, each 10 000 times."""
    torch = pytest.importorskip("torch")
    grid, nb, times = (12, 12, 12), 7, 10000
    lat, k = np.diag(np.array(grid, dtype=float)), np.array([[0.125, -0.375, 0.375]])
    b = pkg.pwdft.PWBasisK(0.28, lat, 30.0, k, grid=grid)
    ref = PWBasisKRef(0.28, lat, 30.0, k, grid=grid)
    rng = np.random.default_rng(8)
    npw = int(b.npwk[0])
    psi = rng.standard_normal((nb, npw)) + 1j * rng.standard_normal((nb, npw))
    want = sum(np.abs(H.recip_to_real(ref, p, 0)) ** 2 for p in psi)
    rho = torch.zeros(b.nxyz, dtype=torch.float64, device="cuda")
    b.psi_to_rho(0, torch.from_numpy(psi).cuda().repeat(times, 1), nb * times, npw, np.full(nb * times, 1.0 / times), rho)
    assert np.max(np.abs(rho.cpu().numpy() - want)) / np.max(want) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("grid,nb", CASES)
def test_rho_matches_oracle(pkg, grid, nb, prec):
    torch = pytest.importorskip("torch")
    lat, k = np.diag(np.array(grid, dtype=float)), np.array([[0.125, -0.375, 0.375]])
    b = pkg.pwdft.PWBasisK(0.28, lat, 30.0, k, grid=grid)
    ref = PWBasisKRef(0.28, lat, 30.0, k, grid=grid)
    rng = np.random.default_rng(5)
    npw, ld = int(b.npwk[0]), int(b.npwk[0]) + 1
    psi = np.zeros((nb, ld), dtype=np.complex128)
    psi[:, :npw] = rng.standard_normal((nb, npw)) + 1j * rng.standard_normal((nb, npw))
    w = rng.uniform(0.1, 2.0, size=nb)
    rho0 = rng.uniform(0.0, 1.0, size=b.nxyz)
    want = rho0.copy()
    if nb > 4:
        w[2] = w[nb - 2] = 0.0
    for ib in range(nb):
        if w[ib]:
            want += w[ib] * np.abs(H.recip_to_real(ref, psi[ib, :npw], 0)) ** 2
    if nb > 4:
        psi[2] = np.nan
    pd = torch.from_numpy(psi).to("cuda", torch.complex64 if prec else torch.complex128)
    rho = torch.from_numpy(rho0).to("cuda", torch.float32 if prec else torch.float64)
    b.psi_to_rho(0, pd, nb, ld, w, rho)
    torch.cuda.synchronize()
    assert np.max(np.abs(rho.cpu().numpy() - want)) / np.max(want) < (2e-5 if prec else 1e-12)
