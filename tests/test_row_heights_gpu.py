"""The last height whose FP64 columns k_row_solve's block holds, 1952 rows (122 chunks of 16 in 232,064 bytes of
shared memory), and the first that takes the passes over chunks of 64 rows, against the oracle with
test_row_solve_gpu's bounds."""
import numpy as np
import pytest

from deeptime_gpu import _lib as L
from deeptime_gpu import flexure as F
from deeptime_gpu import inputs as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [1952, 1953])
def test_the_fp64_block_ends_at_1952_rows(h):
    w, dx = 16, 20_000.0
    d, c, _ = I.flexure_problem(w, h, 4.0, w + h)
    r = np.random.default_rng(h).standard_normal((h, w)) * 1e4
    sv = F.Solver(w, h, dx)
    for precond, bound in ((L.PRECOND_MEAN_D, 1e-10), (L.PRECOND_REFERENCE, 1e-8)):
        want = O.flex_precondition(d, c, r, dx, precond)
        for precision, most in ((L.PREC_FP64, bound), (L.PREC_MIXED, 5e-5)):
            got = sv.precondition(d, c, r, precond, precision)
            assert np.linalg.norm(got - want) < most * np.linalg.norm(want)


@pytest.mark.parametrize("h,dx,most", [(1500, 2500.0, 4e-4), (3000, 1250.0, 1.9e-3)])
def test_fp32_factors_carry_the_fp64_chain_s_error(h, dx, most):
    # The factors' chain amplifies rounding by the dominant wavenumber's contrast (k = 0): restated in numpy, an
    # FP32 chain leaves the solve off by 1.5e-2 and 6.6e-2, an FP64 one rounded once by 1.1e-5 and 5.4e-5; the
    # bounds are the geometric means. In one block (1500 rows) and by the chunk passes (3000).
    w = 16
    d, c = np.full((h, w), 10.0**22.8 / 9.81), np.full((h, w), 3300.0)
    r = np.random.default_rng(h).standard_normal((h, w))
    want = O.flex_precondition(d, c, r, dx, L.PRECOND_MEAN_D)
    got = F.Solver(w, h, dx).precondition(d, c, r, L.PRECOND_MEAN_D, L.PREC_MIXED)
    assert np.linalg.norm(got - want) < most * np.linalg.norm(want)
