"""The row solve along y (heights that are not powers of two, and the row metric) at the edges of its
kernel's ranges: part-filled last chunks of 16 rows, one chunk, the heights where a block goes from 8
wavenumbers to 4 (1024 rows; shared memory bounds the FP64 block earlier) and where the passes
over chunks of 64 rows take over (beyond 2048 rows), against the oracle. Bounds as
test_flexure_gpu's and test_metric_gpu's: the mean level 1e-10, the bank 1e-8, FP32 5e-5."""
import numpy as np
import pytest

from deeptime_gpu import _lib as L
from deeptime_gpu import flexure as F
from deeptime_gpu import inputs as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("w,h", [(64, 3), (64, 15), (64, 17), (32, 33), (16, 1000), (16, 1025), (16, 1935), (16, 1937),
                                 (16, 2047), (16, 2049), (16, 4000)])
def test_heights_at_the_edges_of_the_row_solve(w, h):
    dx = 20_000.0
    d, c, _ = I.flexure_problem(w, h, 4.0, w + h)
    r = np.random.default_rng(h).standard_normal((h, w)) * 1e4
    sv = F.Solver(w, h, dx)
    for precond, bound in ((L.PRECOND_MEAN_D, 1e-10), (L.PRECOND_REFERENCE, 1e-8)):
        want = O.flex_precondition(d, c, r, dx, precond)
        assert rel_l2(sv.precondition(d, c, r, precond, L.PREC_FP64), want) < bound
        assert rel_l2(sv.precondition(d, c, r, precond, L.PREC_MIXED), want) < 5e-5


@pytest.mark.parametrize("h", [17, 1024, 2048])
def test_the_row_metric_at_the_same_edges(h):
    w, dx = 16, 50_000.0
    d, c, _ = I.flexure_problem(w, h, 4.0, h)
    metric = O.row_metric_from_sin_faces(np.clip((0.5 * h - np.arange(h + 1)) / (0.6 * h), -1.0, 1.0), 1)
    r = np.random.default_rng(h).standard_normal((h, w)) * 1e4
    sv = F.Solver(w, h, dx, metric)
    want = O.flex_precondition(d, c, r, dx, L.PRECOND_MEAN_D, metric)
    assert rel_l2(sv.precondition(d, c, r, L.PRECOND_MEAN_D), want) < 1e-10
    assert rel_l2(sv.precondition(d, c, r, L.PRECOND_MEAN_D, L.PREC_MIXED), want) < 5e-5
