"""Sweeps against single steps, bit for bit, at edges that test_sweep.py's boxes
do not have: run(n) sweeps, n calls of run(1) do not."""
import numpy as np
import pytest

import lbmb200 as L

pytestmark = pytest.mark.gpu


def _states(flags, per, pattern, precision, compact, runs, force=True, porosity=None):
    """State after each list of runs, and the launches it took."""
    out = []
    for steps in runs:
        with L.Solver(flags, per, pattern, precision, compact=compact) as s:
            s.set_params(1.3, 3 / 16, 1e-5, force)
            if porosity is not None:
                s.set_porosity(porosity, 0.1)
            s.init_equilibrium(seed=5, amplitude=1e-3)
            for n in steps:
                s.run(n)
            out.append((s.get_state(), s.launch_count))
    return out


@pytest.mark.parametrize("pattern", ["aa", "pull", "push"])
@pytest.mark.parametrize("precision", [L.F64, L.F32, L.F16])
@pytest.mark.parametrize("dims", [(70, 90, 1), (60, 60, 2), (16, 20, 31), (16, 20, 32),
                                  (16, 20, 33), (12, 20, 64), (12, 20, 65), (8, 20, 96)])
def test_rows_that_wrap_in_z(dims, precision, pattern):
    """Compact layout, periodic z: first and last cells of rows of one cell, of
    part of a word, of whole words and of one cell more, with walls on them."""
    flags = (np.random.default_rng(sum(dims)).uniform(size=dims[::-1]) > 0.3).astype(np.int32)
    (ref, singles), (got, launches) = _states(flags, (1, 1, 1), pattern, precision, True,
                                              ((1,) * 8, (8,)))
    assert singles == 8 and launches == 1
    assert np.array_equal(got, ref)


@pytest.mark.slow
@pytest.mark.parametrize("kind", ["fluid", "channel"])
def test_wide_offsets(kind):
    """Compact FP64 lattices of more than 2^32 elements, compared on the
    device: sweeps of AA and pull against single AA steps."""
    dims = (2048, 336, 336)
    flags, per, fluid = L.geometry(kind, dims, (1, 0, 0))
    assert 19 * int((flags != 0).sum()) >= 2 ** 32

    def make(pattern):
        s = L.Solver(flags, per, pattern, L.F64, compact=True)
        s.set_params(1.3, 3 / 16, 1e-5, True)
        s.init_equilibrium(seed=5, amplitude=1e-3)
        return s

    with make("aa") as ref:
        for _ in range(4):
            ref.run(1)
        assert ref.launch_count == 4
        for pattern in ("aa", "pull"):
            with make(pattern) as s:
                s.run(4)
                assert s.launch_count == 2
                out = s.compare(ref)
                assert out[0] == out[2] == out[4] == 0.0 and out[3] > 0.0


@pytest.mark.parametrize("compact", [False, True])
@pytest.mark.parametrize("precision", [L.F64, L.F32])
def test_a_wait_that_runs_out_is_reported(monkeypatch, precision, compact):
    """With no polls allowed, blocks of later steps that run beside the first give
    up at their sixteenth: the kernel ends, the call says so, and the solver goes
    on in single steps from the state it is given next."""
    flags, per, _ = L.geometry("channel", (20, 20, 40), (1, 0, 0))
    f0 = L.perturbed_equilibrium(flags, seed=4, amplitude=2e-3)
    with L.Solver(flags, per, "aa", precision, compact=compact) as s:
        s.set_state(f0)
        for _ in range(8):
            s.run(1)
        ref = s.get_state()
    monkeypatch.setenv("LBM_B200_SWEEP_SPIN", "0")
    with L.Solver(flags, per, "aa", precision, compact=compact) as s:
        s.set_state(f0)
        s.run(8)
        with pytest.raises(L.LbmError, match="gave up waiting"):
            s.synchronize()
        s.set_state(f0)
        s.run(8)
        assert np.array_equal(s.get_state(), ref)
        assert s.launch_count == 1 + 8


@pytest.mark.parametrize("dims", [(12, 10, 64), (9, 11, 128), (8, 9, 256)])
@pytest.mark.parametrize("per", [(1, 0, 0), (1, 1, 1), (0, 1, 1)])
@pytest.mark.parametrize("precision", [L.F64, L.F32, L.F16])
def test_rows_of_whole_segments(monkeypatch, precision, per, dims):
    """For nz a multiple of 64 (128) the single steps of the dense layout run
    shuffle-aligned (four-cell) kernels: they, the generic two-cell kernels,
    the compact layout's and the sweeps agree, odd and even steps, with walls."""
    flags = (np.random.default_rng(sum(dims) + sum(per)).uniform(size=dims[::-1]) > 0.25)
    flags = flags.astype(np.int32)
    for axis in range(3):
        if not per[axis]:
            face = [slice(None)] * 3
            face[2 - axis] = [0, -1]
            flags[tuple(face)] = 0
    assert flags.sum() >= 4096
    for pattern in ("aa", "pull", "push"):
        out = {}
        for switch in ("", "LBM_B200_NO_SHUFFLE", "LBM_B200_NO_QUAD"):
            for name in ("LBM_B200_NO_SHUFFLE", "LBM_B200_NO_QUAD"):
                monkeypatch.setenv(name, "1" if name == switch else "0")
            out[switch or "aligned"], = _states(flags, per, pattern, precision, False, ((1,) * 7,))
        out["compact"], = _states(flags, per, pattern, precision, True, ((1,) * 7,))
        assert all(launches == 7 for _, launches in out.values())
        for compact in (False, True):
            out["sweep", compact], = _states(flags, per, pattern, precision, compact, ((7,),))
            assert out["sweep", compact][1] == 2
        ref = out["aligned"][0]
        for name, (state, _) in out.items():
            assert np.array_equal(state, ref), (pattern, name)


@pytest.mark.parametrize("per", [(1, 1, 1), (1, 1, 0)])
@pytest.mark.parametrize("precision,dims,compact,patterns", [
    (L.F16, (8, 600, 600), False, ("aa", "push", "pull")),
    (L.F16, (8, 600, 600), True, ("push", "pull")),  # AA keeps single steps there
    (L.F32, (8, 500, 431), False, ("aa", "push", "pull")),
    (L.F32, (8, 500, 431), True, ("aa", "push", "pull"))])
def test_fronts_in_two_slabs(precision, dims, compact, patterns, per):
    """Planes of more than 9 MB: two y slabs, whose rows the second step shifts
    by one; two cells of a pair can belong to different slabs."""
    flags = (np.random.default_rng(7).uniform(size=dims[::-1]) > 0.05).astype(np.int32)
    for pattern in patterns:
        (ref, singles), (got, launches) = _states(flags, per, pattern, precision, compact,
                                                  ((1,) * 4, (4,)))
        assert singles == 4 and launches == 2
        assert np.array_equal(got, ref), pattern


@pytest.mark.parametrize("pattern", ["aa", "push"])
@pytest.mark.parametrize("dims,launches", [((24, 30, 41), 1), ((70, 221, 203), 3)])
def test_fp16_brinkman_sweeps(dims, launches, pattern):
    flags, _, _ = L.porous_channel(dims, 0.25, 2.0, 5.0, seed=3)
    por = np.random.default_rng(4).uniform(0, 1, dims).astype(np.float32)
    (ref, singles), (got, n) = _states(flags, (1, 0, 0), pattern, L.F16, False,
                                       ((1,) * 6, (6,)), porosity=por)
    assert singles == 6 and n == launches
    assert np.array_equal(got, ref)
