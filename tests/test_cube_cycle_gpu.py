"""The cube's V-cycle at the sizes where its joined passes and its one-block part change form: one
level only (n = 3, 54 cells), sides that halve unevenly, the block's largest level (16) and one just
above it, all levels in the block refused for its shared memory. Against the oracle's cycle (FP32,
1e-6 relative, as test_cube_gpu) and bit for bit against every level launching its own kernels."""
import numpy as np
import pytest

from oracle import oracle as O
from deeptime_gpu import cube as C
from tests.fixtures import cube_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,fuse", [(3, None), (5, None), (16, None), (17, None), (33, "6144"), (40, "100000"), (51, None)])
def test_the_cycle_at_its_edges(n, fuse, monkeypatch):
    slots = O.cube_topology(n)
    lap, areas, kd, _ = cube_case(n, n + 400, slots)
    r = np.random.default_rng(n).standard_normal(6 * n * n)
    if fuse:
        monkeypatch.setenv("DT_CUBE_FUSE_CELLS", fuse)
    one = C.CubeDiffusion(n, slots, lap, areas)
    monkeypatch.setenv("DT_CUBE_FUSE_CELLS", "0")
    apart = C.CubeDiffusion(n, slots, lap, areas)
    got = one.vcycle(kd, 7.0, r)
    want = O.cube_vcycle(n, slots, lap, areas, kd, 7.0, r)
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
    assert np.array_equal(got, apart.vcycle(kd, 7.0, r))
