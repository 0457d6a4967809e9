"""The line transforms' plan on the host: factors and pads of every edge, and, for orthorhombic and skewed cells, the
runs of occupied x, of each column's sticks and of each stick's plane waves against the maps they stand for
(line_plan_check.cu, compiled against the library)."""
from __future__ import annotations

import importlib.util
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent
PKG = ROOT / "abacus-develop_b200"

LATTICES = {"sc": np.eye(3), "ortho": np.diag([2.0, 1.0, 3.0]),
            "fcc": [[0, 0.5, 0.5], [0.5, 0, 0.5], [0.5, 0.5, 0]], "bcc": [[-0.5, 0.5, 0.5], [0.5, -0.5, 0.5], [0.5, 0.5, -0.5]],
            "hex": [[1, 0, 0], [-0.5, 3 ** 0.5 / 2, 0], [0, 0, 1.633]],
            "tri": [[1, 0.1, -0.2], [0.3, 1.1, 0.05], [-0.15, 0.25, 0.9]],
            "thin": [[1, 0.9, 0], [0, 1, 0.9], [0, 0, 1]]}
KPTS = {"gamma": [[0, 0, 0]], "k": [[0.125, -0.375, 0.375]], "edge": [[0.5, 0.5, 0.5], [0.5, 0, 0]],
        "mp": [[x, y, z] for x in (-0.375, 0.125) for y in (-0.125, 0.375) for z in (0.0, 0.5)]}


@pytest.fixture(scope="module")
def plan_check(tmp_path_factory):
    spec = importlib.util.spec_from_file_location("_line_plan_build", PKG / "build.py")
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    exe = tmp_path_factory.mktemp("line_plan") / "check"
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(build.CSRC),
                    str(Path(__file__).with_name("line_plan_check.cu")), "-o", str(exe), "-L", str(PKG), "-labacus_b200",
                    "-Xlinker", f"-rpath={PKG}"], check=True, capture_output=True, text=True)
    return exe


def _run(plan_check, cells):
    text = "".join("%s %r %s %r %d %d %d %d %s\n" % (name, lat0, " ".join(map(repr, np.asarray(lat, float).ravel().tolist())),
                                                    ecut, *grid, len(k), " ".join(map(repr, np.asarray(k, float).ravel().tolist())))
                   for name, lat0, lat, ecut, grid, k in cells)
    r = subprocess.run([str(plan_check)], input=text, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return {f[0]: (int(f[1]), int(f[2])) for f in (line.split() for line in r.stdout.splitlines())}, r.stderr


def test_runs_of_cells(plan_check):
    cells = [(f"{l}-{k}-{e}", 10.26, LATTICES[l], e, (0, 0, 0), KPTS[k]) for l in LATTICES for k in KPTS for e in (11.0, 30.0)]
    got, err = _run(plan_check, cells)
    assert got.pop("geometry") == (1, 0), err
    assert len(got) == len(cells)
    assert all(v == (1, 0) for v in got.values()), ({n: v for n, v in got.items() if v != (1, 0)}, err)


def test_grids_that_fall_back(plan_check):
    """An edge without two of the factors leaves the plan empty; a tight grid, whose runs fill whole lines, does not."""
    cells = [(f"n{n}{a}", 0.28, np.diag([float(x) for x in g]), 30.0, g, KPTS["k"])
             for n in (162, 180, 192, 216, 243) for a, g in (("x", (n, 20, 18)), ("y", (20, n, 18)), ("z", (18, 20, n)))]
    cells.append(("tight", 0.5, np.diag([24.0, 24.0, 24.0]), 30.0, (24, 24, 24), KPTS["gamma"]))
    got, err = _run(plan_check, cells)
    got.pop("geometry")
    assert got.pop("tight") == (1, 0), err
    assert all(v == (0, 0) for v in got.values()), got
