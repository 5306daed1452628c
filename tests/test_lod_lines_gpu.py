"""The LOD first guess (k_lod_lines) at the edges of its chunks (16 unknowns), of a column segment (1024)
and of a row segment (8192), with blocks whose last line or chunk is partly empty, against the oracle.
Bound as test_diffusion_gpu's: 1e-12 of the largest value."""
import numpy as np
import pytest

from deeptime_gpu import diffusion as D
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,wrap", [(3, 1, True), (16, 16, True), (17, 15, True), (33, 31, True), (31, 17, False), (100, 1023, True),
                                      (9, 1024, True), (10, 1025, True), (5, 2049, True), (8191, 5, True), (8192, 3, True),
                                      (8193, 4, True), (16400, 2, True), (512, 640, True), (2, 40, True), (1, 33, False)])
def test_the_first_guess_matches_the_oracle(w, h, wrap):
    rng = np.random.default_rng(w * 31 + h)
    b = 500.0 * rng.standard_normal((h, w))
    kd = 10.0 ** rng.uniform(-2.0, 1.5, (h, w))
    got = D.Workspace(D.Dims(w, h, 2400.0, wrap)).lod(b, kd, 2.0e6)
    want = O.diff_lod(b, kd, 2.0e6, 2400.0, wrap)
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
