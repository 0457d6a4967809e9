"""recip_to_real / real_to_recip on the line transforms against the oracle's transforms, FP64 within 1e-12 relative and
FP32 within 2e-5 (the bars of test_gpu_transforms.py): tiles of z, sticks and threads with remainders, add and factor."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import hamilt_ref as H
from oracle.pw_basis_ref import PWBasisKRef

GRIDS = [(8, 8, 8), (16, 12, 15), (18, 18, 18), (25, 36, 20), (45, 90, 50), (72, 30, 27), (90, 45, 81), (125, 24, 40),
         (20, 125, 96), (32, 20, 125), (128, 64, 100), (150, 135, 16), (160, 40, 54)]


def rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("grid", GRIDS)
def test_box_transforms(pkg, grid, prec):
    torch = pytest.importorskip("torch")
    lat, k = np.diag(np.array(grid, dtype=float)), np.array([[0.125, -0.375, 0.375]])
    b = pkg.pwdft.PWBasisK(0.28, lat, 30.0, k, grid=grid)
    ref = PWBasisKRef(0.28, lat, 30.0, k, grid=grid)
    rng = np.random.default_rng(2)
    npw, bar = int(b.npwk[0]), 2e-5 if prec else 1e-12
    dt = torch.complex64 if prec else torch.complex128
    c = rng.standard_normal(npw) + 1j * rng.standard_normal(npw)
    box = rng.standard_normal(b.nxyz) + 1j * rng.standard_normal(b.nxyz)
    want_r, want_g = H.recip_to_real(ref, c, 0), H.real_to_recip(ref, box, 0)
    cd, bd = torch.from_numpy(c).to("cuda", dt), torch.from_numpy(box).to("cuda", dt)
    out_r, out_g = torch.full_like(bd, 3.0), torch.full_like(cd, 3.0)
    b.recip_to_real(cd, out_r, 0)
    b.real_to_recip(bd, out_g, 0)
    assert rel(out_r.cpu().numpy(), want_r) < bar
    assert rel(out_g.cpu().numpy(), want_g) < bar
    b.recip_to_real(cd, out_r, 0, add=True, factor=-0.5)
    b.real_to_recip(bd, out_g, 0, add=True, factor=0.25)
    assert rel(out_r.cpu().numpy(), 0.5 * want_r) < 2 * bar
    assert rel(out_g.cpu().numpy(), 1.25 * want_g) < 2 * bar
