"""State transfers in chunks of slices (stream_slices in csrc/lbm_solver.cu):
round trips and moments at sizes below one chunk, across chunk boundaries and
with a slice larger than half the staging buffer."""
import numpy as np
import pytest

import lbmb200 as L

DIMS = [(3, 4, 5),        # a few KB: one kernel, one copy
        (37, 61, 53),     # 18 MB: several chunks of uneven slices
        (1, 300, 310),    # one x plane: a slice is a whole plane
        (2, 1500, 1400),  # slices of 17 MB
        (150, 160, 170)]  # 620 MB: chunks of the largest size


@pytest.mark.gpu
@pytest.mark.parametrize("compact", [False, True])
@pytest.mark.parametrize("pattern", ["pull", "aa"])
@pytest.mark.parametrize("dims", DIMS)
def test_chunked_round_trip(dims, pattern, compact):
    rng = np.random.default_rng(2)
    flags = (rng.uniform(size=dims[::-1]) > 0.2).astype(np.int32)
    fluid = np.transpose(flags, (2, 1, 0)) != 0
    f = rng.uniform(0.01, 0.4, (19,) + dims)
    f[:, ~fluid] = 0.0
    with L.Solver(flags, (1, 1, 1), pattern, L.F64, compact=compact) as s:
        s.set_state(f)
        assert np.array_equal(s.get_state(), f)
        rho, ux, uy, uz = s.moments()
    c = np.array([(0, 1, 0), (0, -1, 0), (1, 0, 0), (-1, 0, 0), (1, 1, 0), (1, -1, 0),
                  (-1, 1, 0), (-1, -1, 0), (0, 0, 1), (0, 1, 1), (1, 0, 1), (-1, 0, 1),
                  (0, -1, 1), (0, 0, -1), (0, -1, -1), (0, 1, -1), (-1, 0, -1), (1, 0, -1),
                  (0, 0, 0)])
    # sums of 19 values below 0.4: 19 roundings of partial sums below 8
    tol = 19 * 8 * 2.0 ** -53
    assert np.max(np.abs(rho - f.sum(0))) <= tol
    for a, u in enumerate((ux, uy, uz)):
        assert np.max(np.abs(u - np.tensordot(c[:, a], f, 1))) <= tol
