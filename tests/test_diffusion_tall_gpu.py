"""Rasters taller than the tiled smoothing's grid reaches (65535 rows of tiles of 24 or 28 cells): the cycle
takes one launch per sweep or colour pass there, bit for bit those of DT_MG_FUSED=0, and the solve meets its
tolerance."""
import numpy as np
import pytest

from deeptime_gpu import _lib as L
from deeptime_gpu import diffusion as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,wrap", [(4, 1_840_000, True), (3, 1_600_000, False)])
@pytest.mark.parametrize("cycle", [L.CYCLE_JACOBI, L.CYCLE_RBGS])
def test_tall_rasters_are_still_taken(w, h, wrap, cycle, monkeypatch):
    rng = np.random.default_rng(h)
    kd = 10.0 ** rng.uniform(-2.0, 1.0, (h, w))
    r = rng.random((h, w)) - 0.5
    ws = D.Workspace(D.Dims(w, h, 2400.0, wrap))
    monkeypatch.setenv("DT_MG_FUSED", "0")
    apart = D.Workspace(D.Dims(w, h, 2400.0, wrap))
    zf, lf = ws.vcycle(kd, 2.0e6, r, cycle)
    za, la = apart.vcycle(kd, 2.0e6, r, cycle)
    assert lf == la and np.array_equal(zf, za), float(np.abs(zf - za).max())
    x, rep = ws.solve_with(500.0 * r, kd, 2.0e6, D.params(cycle=cycle, tol=1e-5))
    assert rep.converged and rep.error_m <= 1e-5
