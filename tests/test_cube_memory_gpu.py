"""The cube handle's device memory: the rows stored both by row and entry by entry took it from 527 to 562 bytes a
cell at 6 x 512^2, so the first guess's line systems share the CG's vectors; and that sharing shows nowhere, whichever
of the first guess and the solve came last."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from deeptime_gpu import cube as C  # noqa: E402
from deeptime_gpu import inputs as I  # noqa: E402

pytestmark = pytest.mark.gpu


def test_a_handle_takes_no_more_memory_for_the_rows_by_entry():
    n = 512
    slots = C.topology(n)
    lap, areas = np.where(slots != C.NO_CELL, 1.0, 0.0), np.ones(6 * n * n)
    C.CubeDiffusion(4, C.topology(4), np.where(C.topology(4) != C.NO_CELL, 1.0, 0.0), np.ones(96)).close()  # the context
    before = torch.cuda.mem_get_info()[0]
    cb = C.CubeDiffusion(n, slots, lap, areas)
    used = before - torch.cuda.mem_get_info()[0]
    cb.close()
    assert used < 545 * 6 * n * n, used / (6 * n * n)


@pytest.mark.parametrize("host", ["0", "1"])
def test_first_guesses_and_solves_leave_each_other_alone(host, monkeypatch):
    monkeypatch.setenv("DT_CUBE_HOST_LOOP", host)
    n, dt = 24, 7.0
    slots = C.topology(n)
    lap, areas, kd, h = I.cube_problem(n, 5, slots)
    fresh = C.CubeDiffusion(n, slots, lap, areas)
    guess, (x, rep) = fresh.lod(kd, dt, h), C.CubeDiffusion(n, slots, lap, areas).solve(h, kd, dt, 1e-6)
    for _ in range(3):
        y, again = fresh.solve(h, kd, dt, 1e-6)
        assert again.iterations == rep.iterations and np.array_equal(y, x)
        assert np.array_equal(fresh.lod(kd, dt, h), guess)
