"""Widths whose half is no power of two, transformed a row pair a block in shared memory: each radix (2 to 7,
a larger prime, a power of two next to odd factors), Bluestein, an odd last row, and in FP64 widths on
either side of the shared-memory limit (6400 values), against the oracle. Bounds as test_widths_gpu's:
mean level 1e-10, bank 1e-8, FP32 5e-5."""
import numpy as np
import pytest

from deeptime_gpu import _lib as L
from deeptime_gpu import flexure as F
from deeptime_gpu import inputs as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("w,h", [(3, 2), (10, 7), (14, 16), (24, 9), (122, 11), (131, 8), (750, 16), (1000, 17), (1920, 8), (1997, 4),
                                 (3125, 3), (6300, 4), (6500, 4), (4099, 2)])
def test_row_pairs_in_a_block_match_the_oracle(w, h):
    dx = 20_000.0
    d, c, _ = I.flexure_problem(w, h, 2.0, w + 11 * h)
    r = np.random.default_rng(abs(w - h)).standard_normal((h, w)) * 1e4
    sv = F.Solver(w, h, dx)
    for precond, bound in ((L.PRECOND_MEAN_D, 1e-10), (L.PRECOND_REFERENCE, 1e-8)):
        want = O.flex_precondition(d, c, r, dx, precond)
        assert rel_l2(sv.precondition(d, c, r, precond, L.PREC_FP64), want) < bound
        assert rel_l2(sv.precondition(d, c, r, precond, L.PREC_MIXED), want) < 5e-5
