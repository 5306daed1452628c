"""Widths whose half is no power of two, on either side of the lines between a row pair in one block and the
passes through global memory, which each lane draws for one level and for the bank: both in blocks (1500),
the bank alone (a prime radix, 488 and 1320; a long chain of radices over few rows, 3200; Bluestein, 1301 x 5),
FP64's one level alone and the reverse in FP32 (2000 x 600, whose rows fill the SMs more than once; 1301 x 200),
and neither (1830, and rows too long for an SM's shared memory). Against the oracle, bounds as
test_widths_gpu's: mean level 1e-10, bank 1e-8, FP32 5e-5."""
import numpy as np
import pytest

from deeptime_gpu import _lib as L
from deeptime_gpu import flexure as F
from deeptime_gpu import inputs as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("w,h", [(1500, 64), (488, 300), (1320, 16), (3200, 16), (1301, 5), (1301, 200), (2000, 600), (1830, 16),
                                 (2053, 4), (6480, 3), (12870, 2)])
def test_both_routes_match_the_oracle(w, h):
    dx = 20_000.0
    d, c, _ = I.flexure_problem(w, h, 2.0, w + 13 * h)
    r = np.random.default_rng(w + h).standard_normal((h, w)) * 1e4
    sv = F.Solver(w, h, dx)
    for precond, bound in ((L.PRECOND_MEAN_D, 1e-10), (L.PRECOND_REFERENCE, 1e-8)):
        want = O.flex_precondition(d, c, r, dx, precond)
        assert rel_l2(sv.precondition(d, c, r, precond, L.PREC_FP64), want) < bound
        assert rel_l2(sv.precondition(d, c, r, precond, L.PREC_MIXED), want) < 5e-5


def test_long_rows_keep_the_speed_of_the_passes():
    # FP32 rows of 9000 in blocks made an iteration 1.38 ms, the passes 0.60; the power-of-two kernels at 8192,
    # 0.21 on the same rows, are the measure of the machine: 6.6 and 2.9 times, the line between them
    h, times = 512, {}
    for w in (9000, 8192):
        d, c, b = I.flexure_problem(w, h, 2.0, w)
        sv = F.Solver(w, h, 20_000.0)
        p = F.params(precond=L.PRECOND_REFERENCE, stop=L.STOP_REL_RESIDUAL, precision=L.PREC_MIXED_RELIABLE, tol=1e-300,
                     max_iterations=20)
        times[w] = min(sv.solve_with(d, c, b, p)[1].device_ms for _ in range(4))
    assert times[9000] < 4.4 * times[8192], times


def test_blocks_allocate_no_buffers_for_the_passes():
    # 1500 x 750: the passes' buffers would be 3 levels x 2 x 375 x 1500 complex values in each lane, 81 MB;
    # the handle without them takes 328 MB (allocations round up to 2 MB)
    torch = pytest.importorskip("torch")
    w, h = 1500, 750
    F.Solver(64, 32, 20_000.0).close()  # the context and the library's modules
    before = torch.cuda.mem_get_info()[0]
    sv = F.Solver(w, h, 20_000.0)
    used = before - torch.cuda.mem_get_info()[0]
    sv.close()
    assert used < 370e6, used
