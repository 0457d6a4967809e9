"""Performance cases of the plane-wave H|psi> / band-solver path.

Each case is one call (or the short sequence of calls) that a plane-wave program makes through this package's
public entry points: H|psi> of a block of bands in both precisions, with one or many k-points and with spinors;
the functor sequence of the local operator; psi -> rho; the projectors of a k-point; a whole band solve.  Cells
are displaced diamond supercells at lat0 = 10.26 bohr per cubic repetition (the package's own workloads), FFT
grids follow the plane-wave basis's rule (2-, 3-, 5-smooth sizes) unless a case gives one.

A case is a dict of plain values:
  kind      hpsi | kbatch | hpsi_nc | local_functors | rho | projectors | solve
  rx ry rz  repetitions of the 8-atom cubic cell (0 0 0: the 2-atom cell of half the edge)
  ecut      wavefunction cut-off (Ry);  n: edge of an explicit cubic FFT grid (0: the basis's rule)
  kx ky kz  k-point in direct coordinates;  nk: k-points of a batch (1 elsewhere)
  nb        bands;  mixed: FP32 transforms and 3xTF32 products (False: FP64)
"""
from __future__ import annotations

import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

LAT0 = 10.26
NH = 8  # projectors per atom: (r_c = 0.8, 1.2) x (s, p_z, p_x, p_y)
_DIAMOND8 = np.array([[0.0, 0.0, 0.0], [0.0, 0.5, 0.5], [0.5, 0.0, 0.5], [0.5, 0.5, 0.0],
                      [0.25, 0.25, 0.25], [0.25, 0.75, 0.75], [0.75, 0.25, 0.75], [0.75, 0.75, 0.25]])


def _package():
    name = "abacus_develop_b200"
    if name not in sys.modules:
        d = Path.cwd() / "abacus-develop_b200"
        spec = importlib.util.spec_from_file_location(name, d / "__init__.py", submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return importlib.import_module(name + ".pwdft")


def _case(name, kind, reps, ecut, nb, mixed=False, k=(0.0, 0.0, 0.0), nk=1, n=0):
    c = dict(kind=kind, rx=reps[0], ry=reps[1], rz=reps[2], ecut=float(ecut), n=n, kx=float(k[0]), ky=float(k[1]),
             kz=float(k[2]), nk=nk, nb=nb, mixed=mixed)
    if name:
        c["name"] = name
    return c


def listed():
    k = (0.125, -0.375, 0.375)
    return [
        # the primitive cell: one call is latency; an iterative solver makes hundreds of them
        _case("hpsi_2atom_fp64", "hpsi", (0, 0, 0), 30, 8, k=k),
        # a Monkhorst-Pack pool of the cubic cell in one batched call
        _case("hpsi_8atom_64k_fp64", "kbatch", (1, 1, 1), 30, 32, nk=64),
        # a double cell: 45 x 45 x 90 grid, the unconverged bands of one Davidson step (an odd count)
        _case("hpsi_16atom_fp64", "hpsi", (1, 1, 2), 40, 61, k=k),
        # an elongated supercell on a grid with three different edges (72 x 36 x 108)
        _case("hpsi_48atom_fp64", "hpsi", (2, 1, 3), 30, 120, k=k),
        # the 64-atom cell (96^3) in both precisions: the benchmark's headline workload
        _case("hpsi_64atom_fp64", "hpsi", (2, 2, 2), 50, 160),
        _case("hpsi_64atom_mixed", "hpsi", (2, 2, 2), 50, 160, mixed=True),
        # the 216-atom cell (128^3, 480 bands, 1728 projectors): the largest block, mixed as its solver runs it
        _case("hpsi_216atom_mixed", "hpsi", (3, 3, 3), 40, 480, mixed=True, n=128),
        # non-collinear spinors
        _case("hpsi_nc_16atom_fp64", "hpsi_nc", (1, 1, 2), 40, 40, k=k),
        # the local operator as an unfused program calls it: transform, product, transform, per band
        _case("local_functors_32atom_fp64", "local_functors", (2, 2, 1), 40, 6, k=k),
        # the charge density of a k-point's occupied bands
        _case("rho_64atom_fp64", "rho", (2, 2, 2), 50, 128),
        # the projectors of a new k-point
        _case("projectors_64atom", "projectors", (2, 2, 2), 50, 160, k=k),
        # a whole band solve of the cubic cell and the density of its bands
        _case("solve_8atom_mixed", "solve", (1, 1, 1), 30, 16, mixed=True, k=k),
    ]


def _grid_edge(r, ecut):
    """Grid edge the basis's rule gives a cell edge of r lattice constants (2-, 3-, 5-smooth)."""
    m = 2 * int(math.sqrt(4.0 * ecut) * LAT0 * r / (2 * math.pi)) + 1
    while True:
        b = m
        for p in (2, 3, 5):
            while b % p == 0:
                b //= p
        if b == 1:
            return m
        m += 1


def draw(rng):
    while True:
        kind = rng.choice(["hpsi", "hpsi", "hpsi", "hpsi", "kbatch", "hpsi_nc", "local_functors", "rho", "projectors",
                           "solve"])
        reps = rng.choice([(0, 0, 0), (1, 1, 1), (1, 1, 2), (1, 2, 2), (2, 1, 3), (2, 2, 2), (1, 3, 2), (3, 2, 2),
                           (3, 3, 1), (2, 3, 3), (3, 3, 3)])
        mixed = rng.random() < 0.4
        ecut = round(rng.uniform(20.0, 60.0), 1)
        nat = 8 * reps[0] * reps[1] * reps[2] or 2
        edges = [_grid_edge(r or 0.5, ecut) for r in reps]
        vol = edges[0] * edges[1] * edges[2]
        nb = max(1, int(round(math.exp(rng.uniform(math.log(1.0), math.log(4.0 * nat))))))
        nk = 1
        if kind == "kbatch":
            nk = rng.randint(2, 64)
        elif kind == "local_functors":
            nb = min(nb, 12)
        elif kind == "projectors":
            nb, mixed = 1, False
        elif kind == "solve":
            nb = 2 * nat
        k = tuple(round(rng.uniform(-0.5, 0.5), 3) for _ in range(3))
        # within the largest listed case's work and the plane sizes every pass accepts
        if max(edges) > 150 or nk * nb * vol * (1 if mixed else 3) > 480 * 128 ** 3:
            continue
        if kind == "solve" and (nat > 8 or vol > 48 ** 3):
            continue
        if kind == "hpsi_nc" and 4 * nb * vol > 480 * 128 ** 3:
            continue
        if nk * nat * vol > 216 * 128 ** 3 or (kind == "projectors" and nat * vol > 64 * 96 ** 3):
            continue
        return _case("", kind, reps, ecut, nb, mixed=mixed, k=k, nk=nk)


# ------------------------------------------------------------------ inputs from the case and the seed alone
class _Cell:
    """Cell, atoms, grid and k-point spheres (restated here so that exact() needs nothing of the package)."""

    def __init__(self, case, seed):
        r = (case["rx"], case["ry"], case["rz"])
        rng = np.random.Generator(np.random.PCG64(seed))
        if r == (0, 0, 0):
            self.lat = np.array([0.5, 0.5, 0.5])
            frac = np.array([[0.0, 0.0, 0.0], [0.25, 0.25, 0.25]])
        else:
            self.lat = np.array(r, dtype=float)
            frac = np.array([(f + np.array([i, j, l])) / self.lat for i in range(r[0]) for j in range(r[1])
                             for l in range(r[2]) for f in _DIAMOND8])
        self.edge = self.lat * LAT0
        self.tau = frac * self.edge + rng.normal(0.0, 0.05, size=frac.shape)
        self.nat = len(self.tau)
        self.nkb = NH * self.nat
        self.omega = float(np.prod(self.edge))
        d = rng.uniform(-1.0, 1.0, size=(self.nat, NH, NH))
        self.deeq = 0.5 * (d + d.transpose(0, 2, 1)) + np.eye(NH) * rng.uniform(-2.0, 2.0, size=(self.nat, 1, NH))
        self.gen_seed = int(rng.integers(1 << 40))
        self.grid = (case["n"],) * 3 if case["n"] else tuple(_grid_edge(x, case["ecut"]) for x in self.lat)
        k0 = np.array([case["kx"], case["ky"], case["kz"]])
        if case["nk"] == 1:
            self.kpts = k0[None, :]
        else:  # the shifted 4 x 4 x 4 Monkhorst-Pack grid, in its order, displaced by the case's k
            u = (np.arange(4) + 0.5) / 4
            u = np.where(u >= 0.5, u - 1.0, u)
            self.kpts = (np.array([[x, y, z] for x in u for y in u for z in u]) + k0)[:case["nk"]]
        nx, ny, nz = self.grid
        ax = [np.where(np.arange(n) > n // 2, np.arange(n) - n, np.arange(n)) for n in self.grid]
        g = [a[:, None] * 0 + a[:, None] for a in ax]
        self.q, self.idx, self.mil = [], [], []
        two_pi = 2 * math.pi
        for kd in self.kpts:
            qx, qy, qz = [two_pi * (g[i][:, 0] + kd[i]) / self.edge[i] for i in range(3)]
            q2 = qx[:, None, None] ** 2 + qy[None, :, None] ** 2 + qz[None, None, :] ** 2
            ix, iy, iz = np.nonzero(q2 <= case["ecut"])
            order = np.argsort((ix * ny + iy).astype(np.int64) * (2 * nz) + ax[2][iz] + nz, kind="stable")
            ix, iy, iz = ix[order], iy[order], iz[order]
            self.q.append(np.stack([qx[ix], qy[iy], qz[iz]], axis=1))
            self.idx.append((ix.astype(np.int64) * ny + iy) * nz + iz)
            self.mil.append(np.stack([ax[0][ix], ax[1][iy], ax[2][iz]], axis=1))
        self.npw = [len(i) for i in self.idx]
        self.ld = max(self.npw)

    def gen(self, salt):
        g = torch.Generator(device="cuda")
        g.manual_seed(self.gen_seed + salt)
        return g

    def qd(self, ik):
        return torch.from_numpy(self.q[ik]).cuda()

    def veff(self):
        """V(r) = -2 Ry sum_atoms exp(-|r - R|^2 / 2), minimum image; r = (x ny + y) nz + z."""
        e = []
        for ax, n in enumerate(self.grid):
            x = torch.arange(n, dtype=torch.float64, device="cuda") * (self.edge[ax] / n)
            d = x[None, :] - torch.from_numpy(self.tau[:, ax]).cuda()[:, None]
            d -= self.edge[ax] * torch.round(d / self.edge[ax])
            e.append(torch.exp(-0.5 * d * d))
        exy = (e[0][:, :, None] * e[1][:, None, :]).reshape(self.nat, -1)
        return (-2.0 * exy.T @ e[2]).reshape(-1).contiguous()

    def vkb(self, ik):
        """Projectors (nkb, ld): c (-i)^l q^l exp(-q^2 r_c^2 / 2) Y_lm exp(-i q R)."""
        q = self.qd(ik)
        q2 = (q * q).sum(1)
        rows = []
        for rc in (0.8, 1.2):
            for l, comp in ((0, 0), (1, 2), (1, 0), (1, 1)):
                integ = math.gamma(l + 1.5) / (2.0 * rc ** (2 * l + 3))
                c = math.sqrt((2 * math.pi) ** 3 / self.omega / integ)
                rad = c * torch.exp(-0.5 * q2 * rc * rc)
                ang = q[:, comp] * math.sqrt(3.0 / (4 * math.pi)) if l else 1.0 / math.sqrt(4 * math.pi)
                rows.append((rad * ang).to(torch.complex128) * ((-1j) ** l))
        ch = torch.stack(rows)                                            # (NH, npw)
        ph = torch.from_numpy(self.tau).cuda() @ q.T                      # (nat, npw)
        out = torch.zeros(self.nkb, self.ld, dtype=torch.complex128, device="cuda")
        v = out.view(self.nat, NH, self.ld)
        for a0 in range(0, self.nat, 32):
            sk = torch.polar(torch.ones_like(ph[a0:a0 + 32]), -ph[a0:a0 + 32])
            v[a0:a0 + 32, :, :self.npw[ik]] = ch[None] * sk[:, None, :]
        return out

    def psi(self, ik, rows, dtype):
        """Random vectors / (1 + |q|^2), zero past the sphere."""
        w = 1.0 / (1.0 + (self.qd(ik) ** 2).sum(1))
        out = torch.zeros(rows, self.ld, dtype=dtype, device="cuda")
        out[:, :self.npw[ik]] = torch.randn(rows, self.npw[ik], dtype=dtype, device="cuda", generator=self.gen(ik)) * w
        return out

    def spinor(self):
        """A non-collinear cell: V_eff's four components and D's four spin blocks D_s(atom, k, x), applied as
        ps_k = sum_x D(k, x) becp_x."""
        v0 = self.veff()
        rng = np.random.Generator(np.random.PCG64(self.gen_seed + 7))
        v4 = torch.stack([v0] + [float(c) * v0 for c in rng.uniform(-0.2, 0.2, size=3)])
        d = self.deeq.astype(np.complex128)
        off = 0.1 * (rng.standard_normal(d.shape) + 1j * rng.standard_normal(d.shape))
        dnc = np.stack([d, off, off.conj().transpose(0, 2, 1), 0.8 * d])
        return v4, torch.from_numpy(np.ascontiguousarray(dnc)).cuda()

    def tables(self, ecut):
        """getvnl's radial tables of the projectors: 4 radial functions on a 0.01 bohr^-1 grid."""
        dq = 0.01
        x = np.arange(int(math.sqrt(ecut) / dq + 4) + 1) * dq
        tab = np.zeros((1, 4, len(x)))
        for ib, (rc, l) in enumerate(((0.8, 0), (0.8, 1), (1.2, 0), (1.2, 1))):
            integ = math.gamma(l + 1.5) / (2.0 * rc ** (2 * l + 3))
            tab[0, ib] = math.sqrt((2 * math.pi) ** 3 / self.omega / integ) * x ** l * np.exp(-0.5 * x * x * rc * rc)
        ch = np.array([[0, 1, 1, 1, 2, 3, 3, 3]])
        return tab, ch, np.array([[0, 1, 1, 1, 0, 1, 1, 1]]), np.array([[0, 1, 2, 3, 0, 1, 2, 3]]), dq


def prepare(case, seed):
    P = _package()
    cell = _Cell(case, seed)
    kind, nb, mixed = case["kind"], case["nb"], case["mixed"]
    dtype = torch.complex64 if mixed else torch.complex128
    real = torch.float32 if mixed else torch.float64
    grid = cell.grid if case["n"] else None
    basis = P.PWBasisK(LAT0, np.diag(cell.lat), case["ecut"], cell.kpts, grid=grid)
    if (basis.nx, basis.ny, basis.nz) != cell.grid or list(basis.npwk) != cell.npw:
        raise RuntimeError("the basis differs from the case's")
    st = {"kind": kind, "P": P, "basis": basis, "nb": nb, "ld": cell.ld, "case": case}
    if kind == "rho":
        st["psi"] = cell.psi(0, nb, dtype)
        st["w"] = np.full(nb, 2.0 / cell.omega)
        st["rho"] = torch.zeros(basis.nxyz, dtype=real, device="cuda")
        return st
    if kind == "local_functors":
        st["psi"] = cell.psi(0, nb, dtype)
        st["veff"] = cell.veff().to(real)
        st["box"] = torch.zeros(basis.nxyz, dtype=dtype, device="cuda")
        st["hpsi"] = torch.zeros_like(st["psi"])
        return st
    h = P.HamiltPW(basis, P.PREC_MIXED if mixed else P.PREC_FP64)
    st["h"] = h
    if kind == "hpsi_nc":
        v4, dnc = cell.spinor()
        h.set_veff_nc(v4)
        h.set_deeq_nc([cell.nat], [NH], dnc)
    else:
        h.set_veff(cell.veff())
        h.set_deeq([cell.nat], [NH], torch.from_numpy(cell.deeq[None]).cuda())
    if kind == "projectors":
        tab, indv, nhtol, nhtolm, dq = cell.tables(case["ecut"])
        h.set_projectors(P.ProjectorSet(1, [cell.nat], [4], [NH], NH, 1, indv, nhtol, nhtolm, tab, dq),
                         cell.tau / LAT0)
        st["vkb"] = torch.zeros(cell.nkb, cell.ld, dtype=torch.complex128, device="cuda")
        return st
    for ik in range(len(cell.npw)):
        h.set_vkb(ik, cell.vkb(ik))
    torch.cuda.empty_cache()  # the library keeps its own copy of the projectors
    if kind == "solve":
        st["start"] = cell.psi(0, nb, torch.complex128)
        st["x"] = torch.zeros_like(st["start"])
        st["dav"] = P.DiagoDavid(P.precondition_d(basis, 0), nb, cell.ld, 4, P.PREC_MIXED if mixed else P.PREC_FP64)
        st["w"] = np.full(nb, 2.0 / cell.omega)
        st["rho"] = torch.zeros(basis.nxyz, dtype=torch.float64, device="cuda")
    elif kind == "kbatch":
        st["psi"] = [cell.psi(ik, nb, dtype) for ik in range(len(cell.npw))]
        st["hpsi"] = [torch.zeros_like(p) for p in st["psi"]]
    else:
        st["psi"] = cell.psi(0, nb * (2 if kind == "hpsi_nc" else 1), dtype)
        st["hpsi"] = torch.zeros_like(st["psi"])
    return st


def run(st):
    kind, nb, ld = st["kind"], st["nb"], st["ld"]
    if kind == "hpsi":
        st["h"].hpsi(0, st["psi"], st["hpsi"], nb, ld)
        return st["hpsi"]
    if kind == "kbatch":
        st["h"].hpsi_kbatch(range(len(st["psi"])), st["psi"], st["hpsi"], nb, ld)
        return st["hpsi"]
    if kind == "hpsi_nc":
        st["h"].hpsi_nc(0, st["psi"], st["hpsi"], nb, ld)
        return st["hpsi"]
    if kind == "local_functors":
        st["hpsi"].zero_()
        for ib in range(nb):
            st["basis"].recip_to_real(st["psi"][ib], st["box"], 0)
            st["P"].veff_pw_op(st["basis"].nxyz, st["box"], st["veff"])
            st["basis"].real_to_recip(st["box"], st["hpsi"][ib], 0, add=True)
        return st["hpsi"], st["box"]
    if kind == "rho":
        st["rho"].zero_()
        st["basis"].psi_to_rho(0, st["psi"], nb, ld, st["w"], st["rho"])
        return st["rho"]
    if kind == "projectors":
        st["h"].build_vkb(0)
        st["h"].copy_vkb(0, st["vkb"])
        return st["vkb"]
    # solve: from the start vectors to the eigenpairs, then the density of the bands
    e = np.zeros(nb)
    st["x"].copy_(st["start"])
    st["dav"].diag_hamilt(st["h"], 0, ld, st["x"], e, 1e-9, 100)
    st["rho"].zero_()
    st["basis"].psi_to_rho(0, st["x"], nb, ld, st["w"], st["rho"])
    return e, st["rho"]


def work(case):
    """Bytes: psi, V_eff and the projectors read once, H|psi> (rho, vkb) written once.  Flops: 5 n log2 n per
    line of the transforms over the occupied sticks and columns, 8 per complex product term."""
    kind, nb, nk = case["kind"], case["nb"], case["nk"]
    reps = [case["rx"] or 0.5, case["ry"] or 0.5, case["rz"] or 0.5]
    nat = 2 if case["rx"] == 0 else 8 * case["rx"] * case["ry"] * case["rz"]
    nx, ny, nz = (case["n"],) * 3 if case["n"] else tuple(_grid_edge(r, case["ecut"]) for r in reps)
    rad = [math.sqrt(case["ecut"]) * LAT0 * r / (2 * math.pi) for r in reps]  # sphere radius in G per axis
    npw = 4.0 / 3.0 * math.pi * rad[0] * rad[1] * rad[2]
    nst, nxc = math.pi * rad[0] * rad[1], min(nx, 2 * rad[0] + 1)
    c, r = (8, 4) if case["mixed"] else (16, 8)
    vol = nx * ny * nz
    fft = 5.0 * (nst * nz * math.log2(nz) + nxc * nz * ny * math.log2(ny) + vol * math.log2(nx))  # one direction
    nl = 16.0 * npw * NH * nat
    if kind == "rho":
        return {"bytes": nb * npw * c + vol * r, "flops": nb * (fft + 4.0 * vol)}
    if kind == "local_functors":
        # three calls per band, each with its own inputs and outputs: the real-space box crosses memory four times
        return {"bytes": nb * (2 * npw * c + 4 * vol * c + vol * r), "flops": nb * (2 * fft + 2.0 * vol)}
    if kind == "projectors":
        return {"bytes": npw * NH * nat * 16.0, "flops": npw * NH * nat * 8.0}
    if kind == "solve":
        # at least ten applications of H to each band
        return {"bytes": 2 * nb * npw * 16 + vol * 8 + npw * NH * nat * 16, "flops": 10.0 * nb * (2 * fft + nl)}
    cols = nb * nk * (2 if kind == "hpsi_nc" else 1)
    return {"bytes": 2 * cols * npw * c + nk * npw * NH * nat * c + vol * r * (4 if kind == "hpsi_nc" else 1),
            "flops": cols * (2 * fft + nl * (1.5 if kind == "hpsi_nc" else 1.0))}


def tolerance(case):
    if case["kind"] == "solve":
        # eigenvalues and density of bands converged to |d lambda| < 1e-9 Ry
        return {"rel": 3e-5}
    if case["kind"] == "projectors":
        return {"rel": 1e-14}
    if case["mixed"]:
        # FP32 transforms; projector products in 3xTF32
        return {"rel": 8e-7}
    return {"rel": 2e-15}


# ------------------------------------------------------------------ the same results in plain torch, 64 bits
def _to_real(cell, ik, c):
    box = torch.zeros(c.shape[0], int(np.prod(cell.grid)), dtype=torch.complex128, device="cuda")
    box[:, torch.from_numpy(cell.idx[ik]).cuda()] = c
    return torch.fft.ifftn(box.view(-1, *cell.grid), dim=(1, 2, 3), norm="forward").reshape(c.shape[0], -1)


def _to_recip(cell, ik, box):
    g = torch.fft.fftn(box.view(-1, *cell.grid), dim=(1, 2, 3), norm="forward").reshape(box.shape[0], -1)
    return g[:, torch.from_numpy(cell.idx[ik]).cuda()]


def _bands_at_once(cell):
    return max(1, int(2e8 // np.prod(cell.grid)))


def _exact_hpsi(cell, ik, psi, veff, deeq, nonlocal_part=True, kinetic=True):
    n = cell.npw[ik]
    out = torch.zeros(psi.shape, dtype=torch.complex128, device="cuda")
    g2 = (cell.qd(ik) ** 2).sum(1)
    step = _bands_at_once(cell)
    for b in range(0, len(psi), step):
        c = psi[b:b + step, :n].to(torch.complex128)
        out[b:b + step, :n] = _to_recip(cell, ik, _to_real(cell, ik, c) * veff)
        if kinetic:
            out[b:b + step, :n] += g2 * c
    if nonlocal_part:
        vkb = cell.vkb(ik)[:, :n]
        p = psi[:, :n].to(torch.complex128)
        becp = (p @ vkb.conj().T).view(len(p), cell.nat, NH)                # (nb, nat, k)
        ps = torch.einsum("axk,bak->bax", deeq.to(torch.complex128), becp)
        out[:, :n] += ps.reshape(len(p), -1) @ vkb
    return out


def _exact_nc(cell, psi):
    n = cell.npw[0]
    v4, dnc = cell.spinor()
    out = torch.zeros(psi.shape, dtype=torch.complex128, device="cuda")
    g2 = (cell.qd(0) ** 2).sum(1)
    step = max(2, _bands_at_once(cell) // 2 * 2)
    for b in range(0, len(psi), step):
        c = psi[b:b + step, :n].to(torch.complex128)
        r = _to_real(cell, 0, c)
        up, dn = r[0::2], r[1::2]
        a = up * (v4[0] + v4[3]) + dn * torch.complex(v4[1], -v4[2])
        d = dn * (v4[0] - v4[3]) + up * torch.complex(v4[1], v4[2])
        r = torch.stack([a, d], 1).reshape(r.shape)
        out[b:b + step, :n] = _to_recip(cell, 0, r) + g2 * c
    vkb = cell.vkb(0)[:, :n]
    becp = (psi[:, :n].to(torch.complex128) @ vkb.conj().T).view(-1, 2, cell.nat, NH)
    up = torch.einsum("akx,bax->bak", dnc[0], becp[:, 0]) + torch.einsum("akx,bax->bak", dnc[1], becp[:, 1])
    dn = torch.einsum("akx,bax->bak", dnc[2], becp[:, 0]) + torch.einsum("akx,bax->bak", dnc[3], becp[:, 1])
    ps = torch.stack([up, dn], 1).reshape(len(psi), -1)
    out[:, :n] += ps @ vkb
    return out


def _exact_rho(cell, psi, w):
    rho = torch.zeros(int(np.prod(cell.grid)), dtype=torch.float64, device="cuda")
    step = _bands_at_once(cell)
    for b in range(0, len(psi), step):
        r = _to_real(cell, 0, psi[b:b + step, :cell.npw[0]].to(torch.complex128))
        rho += w * (r.real ** 2 + r.imag ** 2).sum(0)
    return rho


def _exact_projectors(cell, ecut):
    """getvnl's definition: the tables at |q| by 4-point Lagrange interpolation, (-i)^l, exp(-i q R) and the real
    spherical harmonics with getvnl's sign (m = +-1 carry a minus)."""
    tab, ch, nhtol, nhtolm, dq = cell.tables(ecut)
    q = cell.qd(0)
    qn = torch.sqrt((q * q).sum(1))
    pos = qn / dq
    i = pos.long()
    x0 = pos - i
    x1, x2, x3 = 1.0 - x0, 2.0 - x0, 3.0 - x0
    t = torch.from_numpy(tab[0]).cuda()
    vq = (t[:, i] * x1 * x2 * x3 / 6.0 + t[:, i + 1] * x0 * x2 * x3 / 2.0 - t[:, i + 2] * x1 * x0 * x3 / 2.0
          + t[:, i + 3] * x1 * x2 * x0 / 6.0)
    c = math.sqrt(3.0 / (4 * math.pi))
    u = torch.where(qn[:, None] > 0, q / qn.clamp(min=1e-300)[:, None], torch.zeros_like(q))
    ylm = torch.stack([torch.full_like(qn, 1.0 / math.sqrt(4 * math.pi)), c * u[:, 2], -c * u[:, 0], -c * u[:, 1]])
    rows = [(ylm[int(nhtolm[0, j])] * vq[int(ch[0, j])]).to(torch.complex128) * ((-1j) ** int(nhtol[0, j]))
            for j in range(NH)]
    ph = torch.from_numpy(cell.tau).cuda() @ q.T
    sk = torch.polar(torch.ones_like(ph), -ph)
    out = torch.zeros(cell.nkb, cell.ld, dtype=torch.complex128, device="cuda")
    out.view(cell.nat, NH, cell.ld)[:, :, :cell.npw[0]] = torch.stack(rows)[None] * sk[:, None, :]
    return out


def _exact_solve(cell, nb):
    """Dense diagonalisation: H(G, G') = |k+G|^2 delta + V(G - G') + vkb D vkb^H."""
    nx, ny, nz = cell.grid
    v = torch.fft.fftn(cell.veff().view(nx, ny, nz).to(torch.complex128), norm="forward").reshape(-1)
    m = torch.from_numpy(cell.mil[0]).cuda()
    d = m[:, None, :] - m[None, :, :]
    h = v[(d[..., 0] % nx * ny + d[..., 1] % ny) * nz + d[..., 2] % nz]
    h += torch.diag((cell.qd(0) ** 2).sum(1)).to(torch.complex128)
    vkb = cell.vkb(0)[:, :cell.npw[0]]
    dv = torch.einsum("axk,akg->axg", torch.from_numpy(cell.deeq).cuda().to(torch.complex128),
                      vkb.conj().view(cell.nat, NH, -1)).reshape(cell.nkb, -1)
    h += vkb.T @ dv
    e, x = torch.linalg.eigh(0.5 * (h + h.conj().T))
    return e[:nb].cpu().numpy(), _exact_rho(cell, x[:, :nb].T.contiguous(), 2.0 / cell.omega)


def exact(case, seed):
    cell = _Cell(case, seed)
    kind, nb = case["kind"], case["nb"]
    dtype = torch.complex64 if case["mixed"] else torch.complex128
    if kind == "solve":
        return _exact_solve(cell, nb)
    if kind == "projectors":
        return _exact_projectors(cell, case["ecut"])
    if kind == "rho":
        return _exact_rho(cell, cell.psi(0, nb, dtype), 2.0 / cell.omega)
    if kind == "hpsi_nc":
        return _exact_nc(cell, cell.psi(0, 2 * nb, dtype))
    deeq = torch.from_numpy(cell.deeq).cuda()
    if kind == "local_functors":
        psi, veff = cell.psi(0, nb, dtype), cell.veff()
        box = _to_real(cell, 0, psi[nb - 1:, :cell.npw[0]].to(torch.complex128))[0] * veff
        return _exact_hpsi(cell, 0, psi, veff, deeq, nonlocal_part=False, kinetic=False), box
    out = [_exact_hpsi(cell, ik, cell.psi(ik, nb, dtype), cell.veff(), deeq) for ik in range(len(cell.npw))]
    return out if kind == "kbatch" else out[0]
