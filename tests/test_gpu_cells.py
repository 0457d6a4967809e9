"""The local operator, the box transforms, psi -> rho and k batches against the oracle (FP64 within 1e-12 relative, FP32
within 2e-5) where the line transforms meet other runs than an orthorhombic cell's, and on the grids that they leave to
the Stockham kernels: skewed cells; an edge without two of their factors (162); a plane whose spinor components do not
fit in shared memory (128 x 128 in FP64); a grid so tight that sticks and columns outgrow the auxiliary box."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import hamilt_ref as H
from oracle.pw_basis_ref import PWBasisKRef

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

K3 = np.array([[0.125, -0.375, 0.375], [0.0, 0.0, 0.0], [-0.25, 0.4, 0.5]])
_S = 0.28  # bohr a grid point: the sphere's diameter is then about half of each edge at 30 Ry


def _grid(*n, s=_S):
    return s, np.diag(np.array(n, dtype=float)), n


CELLS = {"fcc": (10.26, [[0, 0.5, 0.5], [0.5, 0, 0.5], [0.5, 0.5, 0]], None),
         "bcc": (8.0, [[-0.5, 0.5, 0.5], [0.5, -0.5, 0.5], [0.5, 0.5, -0.5]], None),
         "hex": (6.0, [[1, 0, 0], [-0.5, 3 ** 0.5 / 2, 0], [0, 0, 1.633]], None),
         "tri": (9.0, [[1, 0.1, -0.2], [0.3, 1.1, 0.05], [-0.15, 0.25, 0.9]], None),
         "thin": (7.0, [[1, 0.9, 0], [0, 1, 0.9], [0, 0, 1]], None),
         "162_x": _grid(162, 20, 18), "162_y": _grid(18, 162, 20), "162_z": _grid(20, 18, 162), "tight": _grid(24, 24, 24, s=0.5)}


SPINOR_CELLS = dict(CELLS, **{"128_plane": _grid(128, 128, 16)})


def rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


class _Case:
    def __init__(self, pkg, name, prec, nb=5):
        lat0, lat, grid = SPINOR_CELLS[name]
        lat = np.asarray(lat, dtype=float)
        self.b = pkg.pwdft.PWBasisK(lat0, lat, 30.0, K3, grid=grid)
        self.ref = PWBasisKRef(lat0, lat, 30.0, K3, grid=grid)
        self.rng = np.random.default_rng(7)
        self.nb, self.ld, self.bar = nb, self.b.npwk_max + 1, 2e-5 if prec else 1e-12
        self.ct = torch.complex64 if prec else torch.complex128
        self.rt = torch.float32 if prec else torch.float64
        self.veff = self.rng.uniform(-2.0, 0.5, size=self.b.nxyz)
        self.psi = []
        for ik in range(3):
            p = np.zeros((nb, self.ld), dtype=np.complex128)
            n = int(self.b.npwk[ik])
            p[:, :n] = self.rng.standard_normal((nb, n)) + 1j * self.rng.standard_normal((nb, n))
            self.psi.append(p)

    def dev(self, a):
        return torch.from_numpy(a).to("cuda", self.ct)

    def local(self, ik):
        h = H.HamiltPWRef(self.ref, ik, self.veff, np.zeros((0, self.ld), dtype=np.complex128), np.zeros((1, 0, 0, 0)), [], [])
        return h.hpsi_local(self.psi[ik].reshape(-1), self.nb, self.ld)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("name", CELLS)
def test_local_operator_and_kbatch(pkg, name, prec):
    c = _Case(pkg, name, prec)
    h = pkg.pwdft.HamiltPW(c.b, prec)
    h.set_veff(torch.from_numpy(c.veff).cuda())
    pd = [c.dev(p) for p in c.psi]
    hd = [torch.full_like(p, 7.0) for p in pd]
    h.hpsi_kbatch([0, 1, 2], pd, hd, c.nb, c.ld)
    for ik in range(3):
        want = c.local(ik)
        one = torch.full_like(pd[ik], 7.0)
        h.hpsi_part(ik, pd[ik], one, c.nb, c.ld, 1)
        assert rel(one.cpu().numpy().reshape(-1), want) < c.bar
        assert rel(hd[ik].cpu().numpy().reshape(-1), want) < c.bar


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("name", CELLS)
def test_transforms_and_rho(pkg, name, prec):
    c = _Case(pkg, name, prec)
    for ik in range(3):
        n = int(c.b.npwk[ik])
        g = c.psi[ik][0, :n]
        box = c.rng.standard_normal(c.b.nxyz) + 1j * c.rng.standard_normal(c.b.nxyz)
        out_r, out_g = torch.full((c.b.nxyz,), 3.0, dtype=c.ct, device="cuda"), torch.full((n,), 3.0, dtype=c.ct, device="cuda")
        c.b.recip_to_real(c.dev(g), out_r, ik)
        c.b.real_to_recip(c.dev(box), out_g, ik, add=True, factor=0.5)
        assert rel(out_r.cpu().numpy(), H.recip_to_real(c.ref, g, ik)) < c.bar
        assert rel(out_g.cpu().numpy(), 3.0 + 0.5 * H.real_to_recip(c.ref, box, ik)) < c.bar
        w = np.array([0.5, 0.0, 1.0, 2.0, 0.25])
        rho = torch.full((c.b.nxyz,), 0.1, dtype=c.rt, device="cuda")
        want = 0.1 + sum(w[i] * np.abs(H.recip_to_real(c.ref, c.psi[ik][i, :n], ik)) ** 2 for i in range(c.nb))
        c.b.psi_to_rho(ik, c.dev(c.psi[ik]), c.nb, c.ld, w, rho)
        assert rel(rho.cpu().numpy(), want) < c.bar


@pytest.mark.parametrize("name,prec", [("fcc", 0), ("hex", 1), ("162_x", 0), ("162_y", 1), ("162_z", 0), ("128_plane", 0),
                                       ("tight", 1)])
def test_spinors(pkg, name, prec):
    c = _Case(pkg, name, prec, nb=4)
    v4 = c.rng.uniform(-1.0, 1.0, size=(4, c.b.nxyz))
    want = H.HamiltPWRefNC(c.ref, 0, list(v4), np.zeros((0, c.ld), dtype=np.complex128),
                           np.zeros((4, 0, 0, 0), dtype=np.complex128), [], []).hpsi(c.psi[0].reshape(-1), 2, c.ld)
    h = pkg.pwdft.HamiltPW(c.b, prec)
    h.set_veff_nc(torch.from_numpy(v4).cuda())
    pd = c.dev(c.psi[0])
    hd = torch.full_like(pd, 7.0)
    h.hpsi_nc(0, pd, hd, 2, c.ld)
    assert rel(hd.cpu().numpy().reshape(-1), want) < c.bar
