"""The register-tiled smoothing of both cycles and the one-block coarse levels (the default) against one
launch per sweep or colour pass (DT_MG_FUSED=0 at create): each update takes the same terms in the
same order, so the FP32 cycles give the same bits. Rasters with ragged last tiles, odd widths (the Jacobi
cycle wraps them; one column at a time instead of two), widths below a tile's 64 columns, one row of
tiles, and 64-row regions."""
import numpy as np
import pytest

from deeptime_gpu import _lib as L
from deeptime_gpu import diffusion as D

pytestmark = pytest.mark.gpu

RASTERS = [(2048, 656, True), (257, 129, True), (301, 77, False), (300, 201, True), (96, 48, True), (63, 40, True), (58, 61, True),
           (7, 9, True), (1, 300, False), (3001, 1501, True), (3000, 1999, False)]


def pair(monkeypatch, w, h, wrap):
    fused = D.Workspace(D.Dims(w, h, 2400.0, wrap))
    monkeypatch.setenv("DT_MG_FUSED", "0")
    apart = D.Workspace(D.Dims(w, h, 2400.0, wrap))
    monkeypatch.delenv("DT_MG_FUSED")
    return fused, apart


@pytest.mark.parametrize("w,h,wrap", RASTERS)
@pytest.mark.parametrize("cycle", [L.CYCLE_JACOBI, L.CYCLE_RBGS])
def test_the_tiled_cycle_is_bit_for_bit_the_separate_launches(w, h, wrap, cycle, monkeypatch):
    rng = np.random.default_rng(w * 7 + h)
    kd = 10.0 ** rng.uniform(-2.0, 1.0, (h, w))
    r = rng.random((h, w)) - 0.5
    fused, apart = pair(monkeypatch, w, h, wrap)
    for _ in range(2):
        zf, lf = fused.vcycle(kd, 2.0e6, r, cycle)
        za, la = apart.vcycle(kd, 2.0e6, r, cycle)
        assert lf == la and np.array_equal(zf, za), float(np.abs(zf - za).max())


@pytest.mark.parametrize("w,h,wrap", [(2048, 656, True), (257, 129, True), (301, 77, False)])
def test_the_reference_split_takes_the_same_steps(w, h, wrap, monkeypatch):
    rng = np.random.default_rng(w + h)
    kd = 10.0 ** rng.uniform(-2.0, 1.0, (h, w))
    z0 = 500.0 * rng.standard_normal((h, w))
    fused, apart = pair(monkeypatch, w, h, wrap)
    xf, rf = fused.solve_with(z0, kd, 2.0e6, D.params(tol=1e-6))
    xa, ra = apart.solve_with(z0, kd, 2.0e6, D.params(tol=1e-6))
    assert rf.iterations == ra.iterations and np.array_equal(xf, xa)
