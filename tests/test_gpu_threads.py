"""Several host threads on one basis: their launches share kernels, whose state (the limit of dynamic shared memory) no
thread may change under another.  At 96 x 96 the plane pass's launch shape, and with it the shared memory, changes with
the band count, so threads with different band counts meet each other's sizes at every call."""
from __future__ import annotations

import dataclasses
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _run_threads(jobs):
    errors = []

    def guard(job):
        try:
            job()
        except BaseException as e:  # noqa: BLE001 - reported by the caller
            errors.append(e)
    threads = [threading.Thread(target=guard, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_local_pass_with_different_band_counts(pkg, prec):
    """Three handles of one basis, a thread and a stream each, bands 1 to 8 in different orders: bit for bit the
    results of the same calls alone, of the local part and of the whole H|psi> (each handle with projector scratch and
    a second stream of its own)."""
    P = pkg.pwdft
    n = 96
    b = P.PWBasisK(0.28, np.diag([float(n)] * 3), 30.0, np.array([[0.125, -0.375, 0.375]]), grid=(n, n, n))
    rng = np.random.default_rng(4)
    ld = int(b.npwk_max)
    ct = torch.complex128 if prec == "fp64" else torch.complex64
    psi = torch.from_numpy(rng.standard_normal((8, ld)) + 1j * rng.standard_normal((8, ld))).to("cuda", ct)
    veff = torch.from_numpy(rng.uniform(-2.0, 0.5, size=b.nxyz)).cuda()
    hs = [P.HamiltPW(b, P.PREC_FP64 if prec == "fp64" else P.PREC_MIXED) for _ in range(3)]
    vkb = torch.from_numpy(rng.standard_normal((8, ld)) + 1j * rng.standard_normal((8, ld))).cuda()
    deeq = torch.from_numpy(rng.standard_normal((1, 1, 8, 8))).cuda()
    for h in hs:
        h.set_veff(veff)
        h.set_deeq([1], [8], deeq)
        h.set_vkb(0, vkb)

    def call(h, whole, nb, out):
        if whole:
            h.hpsi(0, psi, out, nb, ld)
        else:
            h.hpsi_part(0, psi, out, nb, ld, 1)
    want = {(nb, whole): torch.zeros_like(psi[:nb]) for nb in (1, 2, 3, 4, 5, 7, 8) for whole in (False, True)}
    for (nb, whole), out in want.items():
        call(hs[0], whole, nb, out)
    torch.cuda.synchronize()

    def job(h, counts):
        def run():
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                out = torch.zeros_like(psi)
                for i in range(400):
                    nb, whole = counts[i % len(counts)], i >= 200
                    call(h, whole, nb, out)
                    if i % 25 < len(counts):
                        assert torch.equal(out[:nb], want[nb, whole]), (i, nb, whole)
                s.synchronize()
        return run
    _run_threads([job(hs[0], (1, 5, 2)), job(hs[1], (8, 1, 4)), job(hs[2], (3, 7))])


def test_concurrent_mixed_solves_at_96(pkg):
    """Four workers on one Hamiltonian, so that their unconverged bands differ: each k-point's eigenvalues and iteration
    count of its solve alone."""
    P = pkg.pwdft
    spec = dataclasses.replace(pkg.synth.config(0), grid=(96, 96, 96))
    wl = P.build_workload(spec, kpts=pkg.synth.mp_grid(2, True)[:4])
    h = P.device_hamilt(wl, P.PREC_FP64)
    nband, ld = 6, wl.basis.npwk_max
    iks = list(range(4))
    pcs = [P.precondition_d(wl.basis, ik) for ik in iks]
    start = [torch.from_numpy(wl.psi0_h[ik][:nband].reshape(-1).copy()).cuda() for ik in iks]
    alone, its_alone = [], []
    for ik in iks:
        dav = P.DiagoDavid(pcs[ik], nband, int(wl.basis.npwk[ik]), 4, P.PREC_MIXED)
        e = np.zeros(nband)
        its_alone.append(dav.diag_hamilt(h, ik, ld, start[ik].clone(), e, 1e-9, 100))
        alone.append(e)
    for _ in range(5):
        eig, its = h.solve_kpoints(iks, pcs, [x.clone() for x in start], ld, nband, 1e-9, 100, precision=P.PREC_MIXED,
                                   nworkers=4)
        assert np.max(np.abs(np.asarray(eig) - np.asarray(alone))) < 1e-9
        assert list(its) == its_alone


def test_workers_share_the_stick_buffer(pkg):
    """64-atom sized blocks (2.6 MB of sticks a band): four workers hold 128 MB of sticks each where one takes all bands
    in one chunk, which shows in the kernels launched; the eigenvalues are the same."""
    P = pkg.pwdft
    rng = np.random.default_rng(1)
    nk, nband = 4, 96
    b = P.PWBasisK(20.52, np.eye(3), 50.0, rng.uniform(-0.2, 0.2, size=(nk, 3)), grid=(96, 96, 96))
    ld = int(b.npwk_max)
    h = P.HamiltPW(b, P.PREC_FP64)
    h.set_veff(torch.from_numpy(rng.uniform(-2.0, 0.5, size=b.nxyz)).cuda())
    h.set_deeq([1], [1], torch.ones(1, 1, 1, 1, dtype=torch.float64, device="cuda"))
    for ik in range(nk):
        h.set_vkb(ik, torch.full((1, ld), 0.01 + 0j, dtype=torch.complex128, device="cuda"))
    pcs = [P.precondition_d(b, ik) for ik in range(nk)]
    gen = torch.Generator(device="cuda")
    launches, eig = [], []
    for workers in (1, 4):
        gen.manual_seed(3)
        x = [torch.randn(nband, ld, dtype=torch.complex128, device="cuda", generator=gen) for _ in range(nk)]
        for ik in range(nk):
            x[ik][:, int(b.npwk[ik]):] = 0
        n0 = pkg._lib.load().b200_kernel_launches()
        eig.append(h.solve_kpoints(range(nk), pcs, x, ld, nband, 1e9, 3, nworkers=workers)[0])
        launches.append(pkg._lib.load().b200_kernel_launches() - n0)
    assert launches[1] > launches[0]
    assert np.max(np.abs(eig[1] - eig[0])) < 1e-9 * np.max(np.abs(eig[0]))
