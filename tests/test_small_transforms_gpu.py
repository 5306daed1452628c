"""The transforms of small rasters (up to 2^19 cells, lengths up to 1024: eight values a thread, few
columns a block, the bank's levels side by side) at the shortest and longest rows and columns
that take them and on either side of the cell limit, against the oracle. Bounds as
test_flexure_gpu's: the mean level 1e-10, the bank 1e-8, FP32 5e-5."""
import numpy as np
import pytest

from deeptime_gpu import _lib as L
from deeptime_gpu import flexure as F
from deeptime_gpu import inputs as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("w,h", [(4, 16), (8, 16), (8, 8), (16, 1024), (128, 33), (512, 128), (2048, 16), (2048, 256),
                                 (1024, 512), (512, 1024), (1024, 1024), (4096, 64)])
def test_small_transforms_match_the_oracle(w, h):
    dx = 20_000.0
    d, c, _ = I.flexure_problem(w, h, 2.0, 3 * w + h)
    r = np.random.default_rng(w + h).standard_normal((h, w)) * 1e4
    sv = F.Solver(w, h, dx)
    for precond, bound in ((L.PRECOND_MEAN_D, 1e-10), (L.PRECOND_REFERENCE, 1e-8)):
        want = O.flex_precondition(d, c, r, dx, precond)
        assert rel_l2(sv.precondition(d, c, r, precond, L.PREC_FP64), want) < bound
        assert rel_l2(sv.precondition(d, c, r, precond, L.PREC_MIXED), want) < 5e-5
