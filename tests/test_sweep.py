"""Sweeps: several steps per launch (csrc/lbm_sweep.cuh). The CPU test replays
the block order of the plans; the GPU tests compare run(n), which sweeps, with
n calls of run(1), which takes single steps: bit for bit."""
import os
import subprocess

import numpy as np
import pytest

import lbmb200 as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sweep_order(tmp_path):
    exe = tmp_path / "probe"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "lbm-bench_b200", "csrc"),
                    os.path.join(ROOT, "tests", "sweep_order_probe.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout


def _solver(dims, kind, pattern, precision, compact):
    if kind == "porous":
        flags, _, _ = L.porous_channel(dims, 0.25, 2.0, 5.0, seed=3)
        per = (1, 0, 0)
    else:  # fully periodic
        flags, per, _ = L.geometry("fluid", dims)
    s = L.Solver(flags, per, pattern, precision, compact=compact)
    s.set_params(1.3, 3 / 16, 1e-5, kind == "porous")
    s.init_equilibrium(seed=5, amplitude=1e-3)
    return s


# step-major: lattices in the L2, down to planes smaller than a block and
# fewer planes than steps; fronts: larger ones, one and two slabs of y, with
# rows of one word, ragged words and a periodic z
RESIDENT = [(20, 18, 40), (3, 61, 33), (130, 7, 12), (64, 30, 65)]
FRONTS = {L.F64: [(41, 131, 141), (10, 301, 300)], L.F32: [(80, 131, 141), (10, 421, 420)],
          L.F16: [(70, 221, 203)]}
CASES = [(d, p, c) for d in RESIDENT for p in (L.F64, L.F32, L.F16) for c in (True, False)]
CASES += [(d, p, c) for p, dims in FRONTS.items() for d in dims for c in (True, False)]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["porous", "periodic"])
@pytest.mark.parametrize("pattern", ["aa", "pull", "push"])
@pytest.mark.parametrize("dims,precision,compact", CASES)
def test_sweeps_equal_single_steps(dims, precision, compact, pattern, kind):
    if kind == "porous" and min(dims[1:]) < 12:
        kind = "periodic"  # walls alone would fill it
    with _solver(dims, kind, pattern, precision, compact) as s:
        for _ in range(9):
            s.run(1)
        ref = s.get_state()
        singles = s.launch_count
    with _solver(dims, kind, pattern, precision, compact) as s:
        s.run(3)  # AA is left at an odd step: the next call starts with a single one
        s.run(6)
        got = s.get_state()
        assert s.steps_done == 9 and singles == 9
        # large FP16 lattices keep the single steps that are faster there
        if not (precision == L.F16 and compact and pattern == "aa" and
                dims in FRONTS[L.F16]):
            assert s.launch_count < 9
    assert np.array_equal(got, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("dims,precision", [((24, 30, 40), L.F64), ((41, 131, 141), L.F64),
                                            ((24, 30, 41), L.F32), ((80, 131, 141), L.F32)])
@pytest.mark.parametrize("pattern", ["aa", "push"])
def test_brinkman_sweeps_equal_single_steps(pattern, dims, precision):
    por = np.random.default_rng(4).uniform(0, 1, dims).astype(np.float32)
    out = []
    for steps in ((1,) * 6, (6,)):
        with _solver(dims, "porous", pattern, precision, False) as s:
            s.set_porosity(por, 0.1)
            for n in steps:
                s.run(n)
            out.append(s.get_state())
    assert np.array_equal(out[0], out[1])


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [L.F64, L.F32])
@pytest.mark.parametrize("dims", [(24, 30, 41), (81, 131, 141)])
def test_gradient_does_not_depend_on_sweeps(dims, precision):
    """checkpoint_every = 1 recomputes single steps; longer segments sweep
    (even and odd lengths), saving each step's momentum."""
    por = np.random.default_rng(4).uniform(0, 1, dims).astype(np.float32)
    out = []
    for k in (1, 4, 5, 11):
        with _solver(dims, "porous", "aa", precision, False) as s:
            s.set_porosity(por, 0.1)
            out.append(s.adjoint_gradient(11, k)[:2])
            again = s.adjoint_gradient(11, k)[:2]  # in the kept workspace
            assert again[0] == out[-1][0] and np.array_equal(again[1], out[-1][1])
    for j, g in out[1:]:
        assert j == out[0][0] and np.array_equal(g, out[0][1])
