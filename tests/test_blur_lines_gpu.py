"""The box blur's line blocks at their edges: line counts around a block's 8, 16 and 32 lines and past
the counts that choose among them (1184 lines, 7104 columns), lengths around a tile of 32 positions,
radii up to the ring's, against the oracle bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from deeptime_gpu import grid as Gr  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(15, 17), (16, 16), (17, 15), (31, 64), (33, 33), (64, 100), (700, 49), (49, 700), (7, 9), (1184, 40), (1185, 40), (40, 1185), (7104, 33), (7105, 33)])
@pytest.mark.parametrize("r", [1, 5, 31, 32, 63])
@pytest.mark.parametrize("wrap", [False, True])
def test_box_blur_at_block_edges(w, h, r, wrap):
    v = np.random.default_rng(w * h + r).standard_normal((h, w))
    got = Gr.box_blur(torch.from_numpy(v).cuda(), r, 2, wrap_x=wrap)
    want = O.box_blur(v, r, 2, wrap=wrap)
    assert np.array_equal(got.cpu().numpy(), want)
