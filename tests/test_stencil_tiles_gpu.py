"""The loop's stencils over register tiles (60 columns by 28 or 60 rows of output) at the edges of their
tiles: rasters narrower than a tile's 64-column region (columns that repeat), odd widths, one row, a
last row or column alone in its tile, and 64-row regions, through solves and the preconditioner. Bounds as
test_flexure_gpu's and test_metric_gpu's: the bank 1e-8 (FP32 5e-5), solves to 1e-10 at 1e-8."""
import numpy as np
import pytest

from deeptime_gpu import _lib as L
from deeptime_gpu import flexure as F
from deeptime_gpu import inputs as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("w,h", [(6, 2), (7, 29), (60, 28), (61, 29), (62, 57), (64, 3), (120, 61), (121, 16), (1800, 1500)])
def test_the_sandwich_matches_the_oracle(w, h):
    dx = 20_000.0
    d, c, _ = I.flexure_problem(w, h, 2.0, 5 * w + h)
    r = np.random.default_rng(w + 3 * h).standard_normal((h, w)) * 1e4
    sv = F.Solver(w, h, dx)
    want = O.flex_precondition(d, c, r, dx, O.PRECOND_REFERENCE)
    assert rel_l2(sv.precondition(d, c, r, L.PRECOND_REFERENCE, L.PREC_FP64), want) < 1e-8
    assert rel_l2(sv.precondition(d, c, r, L.PRECOND_REFERENCE, L.PREC_MIXED), want) < 5e-5


@pytest.mark.parametrize("metric", [False, True])
@pytest.mark.parametrize("w,h", [(62, 57), (61, 30), (244, 90)])
def test_solves_on_ragged_tiles_match_the_oracle(w, h, metric):
    dx = 40_000.0
    d, c, b = I.flexure_problem(w, h, 2.0, 7 * w + h)
    m = O.row_metric_from_sin_faces(np.clip((0.5 * h - np.arange(h + 1)) / (0.6 * h), -1.0, 1.0), 1) if metric else None
    want, orep = O.flex_solve(d, c, b, dx, 1e-12, 20000, stop=O.STOP_REL_RESIDUAL, metric=m)
    assert orep["converged"]
    sv = F.Solver(w, h, dx, m)
    for prec in (L.PREC_FP64, L.PREC_MIXED_RELIABLE):
        x, rep = sv.solve_with(d, c, b, F.params(stop=L.STOP_REL_RESIDUAL, precision=prec, tol=1e-10, max_iterations=20000))
        assert rep.converged and rel_l2(x, want) < 1e-8
