"""Host paths of the solver without a GPU: the library's own objects linked
with a CUDA runtime that counts launches and limits memory (fake_cudart.cpp)."""
import ctypes
import glob
import importlib.util
import os
import subprocess
import sys

import numpy as np
import pytest

import lbmb200

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "lbm-bench_b200")


@pytest.fixture(scope="module")
def L(tmp_path_factory):
    """The binding over the fake runtime, with .fake (the library)."""
    subprocess.run(["make", "-C", PKG, "-j8"], check=True, capture_output=True)
    objs = [o for o in sorted(glob.glob(os.path.join(PKG, "_build", "lbm_*.o")))
            if not o.endswith("_sp.o")]
    so = tmp_path_factory.mktemp("fake") / "libfake.so"
    subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "fake_cudart.cpp"), *objs, "-o", str(so),
                    "-Wl,-Bsymbolic", "-fopenmp", "-ldl"], check=True, capture_output=True)
    spec = importlib.util.spec_from_file_location("lbmb200_fake", lbmb200.__file__)
    mod = importlib.util.module_from_spec(spec)
    sys.modules["lbmb200_fake"] = mod
    spec.loader.exec_module(mod)
    mod.LIB_PATH = str(so)
    mod.fake = mod.lib()
    mod.fake.fake_limit.argtypes = [ctypes.c_size_t]
    mod.fake.fake_raise.argtypes = [ctypes.c_uint]
    mod.fake.fake_used.restype = ctypes.c_size_t
    mod.fake.fake_launches.restype = ctypes.c_long
    mod.fake.fake_mapped.restype = ctypes.c_long
    yield mod
    mod.fake.fake_limit(1 << 40)


def _porous_solver(L, dims, precision=None):
    flags = np.ones(dims[::-1], np.int32)
    s = L.Solver(flags, (1, 1, 1), "aa", L.F64 if precision is None else precision)
    s.set_porosity(np.full(dims, 0.5, np.float32), 0.1)
    return s


def test_failed_staging_growth_leaves_the_solver_usable(L):
    """A slice of the moments of 1 x 1500 x 1500 (72 MB) is larger than the
    staging the solver was created with: growing it fails, and the gradient's
    download, which needs no more than before, still has its buffer."""
    with _porous_solver(L, (1, 1500, 1500)) as s:
        before = s.device_bytes
        L.fake.fake_limit(L.fake.fake_used() + (1 << 20))
        with pytest.raises(L.LbmError):
            s.moments()
        L.fake.fake_limit(1 << 40)
        assert s.device_bytes == before
        s.adjoint_gradient(2, 1)
        s.set_porosity(np.zeros((1, 1500, 1500), np.float32), 0.0)
        assert s.device_bytes == before
        s.moments()
        assert s.device_bytes > before


@pytest.mark.parametrize("pattern,lattices", [("aa", 1), ("push", 2)])
@pytest.mark.parametrize("compact", [False, True])
def test_creation_maps_memory_for_the_lattices_only(L, compact, pattern, lattices):
    """A small solver's other buffers come out of memory that is mapped anyway."""
    flags, per, _ = L.geometry("box", (20, 20, 20))
    before = L.fake.fake_mapped()
    with L.Solver(flags, per, L.PATTERNS[pattern], L.F64, compact=compact) as s:
        s.set_state(np.zeros((19, 20, 20, 20)))
        s.run(8)
        s.get_state()
        s.moments()
        assert L.fake.fake_mapped() - before <= lattices
    assert L.fake.fake_used() == 0


@pytest.mark.parametrize("dims", [(512, 16, 32), (128, 32, 32)])
@pytest.mark.parametrize("compact", [False, True])
def test_creation_needs_no_memory_for_what_it_can_do_without(L, compact, dims):
    """On a nearly full device a solver is created without the sweeps'
    counters and with staging for one dense plane, and takes single steps."""
    flags = np.ones(dims[::-1], np.int32)
    cells = dims[0] * dims[1] * dims[2]

    def make():
        return L.Solver(flags, (1, 1, 1), "aa", L.F64, compact=compact)

    with make() as s:
        s.run(8)
        assert s.launch_count == 1
        full = s.device_bytes
        assert full == L.fake.fake_used()
    # state, link masks, staging plane, the build's fluid bytes; compact: the
    # index and the build's dense masks; 64 KB of reduction partials and padding
    least = 19 * 8 * cells + 4 * cells + 8 * cells + cells + (1 << 16)
    if compact:
        least += 8 * cells // 32 + 4 * cells
    assert least < full
    try:
        for limit in range(least, full + 1, (full - least) // 16):
            L.fake.fake_limit(limit)
            with make() as s:
                s.run(8)
                assert s.steps_done == 8
                assert s.launch_count == 8 or limit > least or dims[0] == 128
                s.get_state()
                s.moments()
    finally:
        L.fake.fake_limit(1 << 40)
    assert L.fake.fake_used() == 0


# (box, geometry, pattern, precision, compact, whether run(8) sweeps): boxes at
# which sweeps measured slower than single steps, each beside one of the same
# kind at which they are faster
ROUTES = [
    ((16384, 3, 3), "fluid", "push", "fp32", True, False),  # thin planes
    ((4096, 8, 8), "fluid", "push", "fp32", True, True),
    ((16384, 3, 3), "fluid", "push", "fp64", False, False),
    ((8192, 10, 10), "channel", "aa", "fp64", True, False),
    ((2048, 24, 24), "channel", "aa", "fp64", True, True),
    ((2, 300, 300), "channel", "aa", "fp64", True, False),  # few planes
    ((2, 300, 300), "fluid", "pull", "fp64", False, False),
    ((16, 128, 128), "fluid", "pull", "fp64", True, True),
    ((1024, 24, 24), "channel", "push", "fp16", True, False),  # rows of one word
    ((1024, 40, 40), "channel", "push", "fp16", True, True),
    ((200, 200, 33), "pipe", "aa", "fp64", False, False),   # mostly solid box
    ((200, 100, 33), "channel", "aa", "fp64", False, True),
    ((128, 128, 128), "fluid", "pull", "fp16", False, False),  # rows of whole segments
    ((96, 96, 96), "fluid", "pull", "fp16", False, True),
    ((64, 64, 64), "channel", "aa", "fp64", False, True),
]


@pytest.mark.parametrize("dims,kind,pattern,precision,compact,sweeps", ROUTES)
def test_sweeps_run_where_they_are_faster(L, dims, kind, pattern, precision, compact, sweeps):
    flags, per, _ = L.geometry(kind, dims, (1, 0, 0))
    with L.Solver(flags, per, L.PATTERNS[pattern], L.PRECISIONS[precision], compact=compact) as s:
        s.run(8)
        assert s.steps_done == 8
        assert (s.launch_count < 8) == sweeps


def test_counters_stay_small(L):
    """31 counters of a cache line for each plane of a long thin box would be
    more memory than its lattice."""
    for dims in ((60000, 3, 3), (4096, 4, 4), (2900, 3, 3)):
        flags = np.ones(dims[::-1], np.int32)
        for compact in (False, True):
            with L.Solver(flags, (1, 1, 1), "aa", L.F64, compact=compact) as s:
                s.run(64)
                state = 19 * 8 * flags.size
                assert s.device_bytes < 3 * state + (16 << 20)


@pytest.mark.parametrize("dims,kind,sweeps", [((16384, 6, 6), "channel", False),
                                              ((300, 200, 16), "pipe", False),
                                              ((64, 64, 64), "channel", True),
                                              ((128, 64, 64), "channel", True)])
def test_reverse_sweeps_run_where_they_are_faster(L, dims, kind, sweeps):
    flags, per, _ = L.geometry(kind, dims, (1, 0, 0))
    with L.Solver(flags, per, "aa", L.F64) as s:
        s.set_porosity(np.full(dims, 0.5, np.float32), 0.1)
        L.fake.fake_launches(b"", 1)
        s.adjoint_gradient(8, 8)
        assert (L.fake.fake_launches(b"SweepAdjoint", 0) > 0) == sweeps
        assert (L.fake.fake_launches(b"adjoint_step_kernel", 0) == 8) != sweeps


@pytest.mark.slow
def test_wide_offsets_sweep_in_fp64_only(L):
    """Lattices of 2^32 elements and more (here by a few planes) need 64-bit
    offsets, with which the two-cell sweeps spill and are slower."""
    dims = (2048, 332, 333)
    assert 19 * dims[0] * dims[1] * dims[2] >= 2 ** 32
    flags = np.ones(dims[::-1], np.int32)
    for precision, sweeps in ((L.F64, True), (L.F32, False)):
        with L.Solver(flags, (1, 1, 1), "pull", precision, compact=True) as s:
            s.run(8)
            assert (s.launch_count < 8) == sweeps


def test_a_sweep_that_gave_up_leaves_single_steps(L):
    """The error word set by a sweep's kernel: the next call that waits reports
    it, and later steps and gradients run as single steps."""
    with _porous_solver(L, (64, 64, 64)) as s:
        s.run(8)
        assert s.launch_count == 1
        L.fake.fake_raise(1 << 31)
        with pytest.raises(L.LbmError, match="gave up waiting"):
            s.synchronize()
        s.synchronize()
        s.run(8)
        assert s.launch_count == 1 + 8
        L.fake.fake_launches(b"", 1)
        s.adjoint_gradient(8, 8)
        assert L.fake.fake_launches(b"sweep_kernel", 0) == 0


def test_synchronize_always_looks_at_the_error_word(L):
    """A sweep or pipelined step in a graph captured by the caller may run after
    the launch's own check."""
    flags, per, _ = L.geometry("channel", (64, 64, 64), (1, 0, 0))
    for call in ("synchronize", "run_timed", "time_launches"):
        with L.Solver(flags, per, "aa", L.F64) as s:
            s.run(8)
            s.synchronize()
            L.fake.fake_raise(1 << 30)
            with pytest.raises(L.LbmError, match="bulk copies"):
                getattr(s, call)(*(() if call == "synchronize" else (1,)))
            s.run(9)
            assert s.launch_count < s.steps_done  # not a sweep's fault: it still sweeps


def test_no_sweep_switch(L, monkeypatch):
    monkeypatch.setenv("LBM_B200_NO_SWEEP", "1")
    with _porous_solver(L, (64, 64, 64)) as s:
        s.run(8)
        assert s.launch_count == 8
        L.fake.fake_launches(b"", 1)
        s.adjoint_gradient(8, 8)
        assert L.fake.fake_launches(b"sweep_kernel", 0) == 0


def test_kept_adjoint_workspace_is_given_back(L):
    """A solver keeps its workspace between gradients; a second gradient or a
    second solver that would not fit without that memory gets it, and switching
    the porosity off gives it back."""
    dims = (64, 64, 64)
    with _porous_solver(L, dims) as a:
        own = a.device_bytes
        g = a.adjoint_gradient(30, 30)[2]
        kept = a.device_bytes - own
        assert kept == g["extra_bytes"] > 4 * own and g["peak_bytes"] == own + kept
        try:
            # room for a second solver, but not for its gradient
            L.fake.fake_limit(L.fake.fake_used() + own + (8 << 20))
            with _porous_solver(L, dims) as b:
                # AUTO: the longest interval, with what a keeps counted as free
                assert b.adjoint_gradient(9, L.CKPT_AUTO)[2]["interval"] == 9
                assert a.device_bytes == own < b.device_bytes
                a.adjoint_gradient(30, 30)  # and the other way round
                assert b.device_bytes == own and a.device_bytes == own + kept
                with _porous_solver(L, dims):
                    assert a.device_bytes == own
                a.adjoint_gradient(30, 30)
            assert a.device_bytes == own + kept == L.fake.fake_used()
        finally:
            L.fake.fake_limit(1 << 40)
        a.set_porosity(np.zeros(dims, np.float32), 0.0)
        assert a.device_bytes == own == L.fake.fake_used()
    assert L.fake.fake_used() == 0


@pytest.mark.parametrize("dims,kind,pattern,precision,compact,least", [
    ((20, 20, 20), "channel", "aa", "fp64", False, 4),
    ((32, 32, 32), "channel", "push", "fp32", True, 4),
    ((200, 64, 64), "channel", "aa", "fp16", True, 4),
    ((64, 64, 64), "channel", "push", "fp64", False, 2),
    ((20, 20, 40), "fluid", "pull", "fp16", True, 2),
    ((128, 128, 128), "channel", "aa", "fp64", True, 2)])
def test_short_calls(L, dims, kind, pattern, precision, compact, least):
    """Calls of two or three steps sweep where that is faster."""
    flags, per, _ = L.geometry(kind, dims, (1, 0, 0))
    with L.Solver(flags, per, L.PATTERNS[pattern], L.PRECISIONS[precision], compact=compact) as s:
        s.run(2)
        assert s.launch_count == (1 if least == 2 else 2)
        s.run(least)
        assert s.launch_count == (2 if least == 2 else 3)
