"""The box blur's last block of lines, which takes the last 8, 16 or 32 lines whole and so some of the block
before's again, against the oracle bit for bit: line counts a line more and a line less than whole blocks in
each form, and fewer lines than a block."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from deeptime_gpu import grid as Gr  # noqa: E402
from oracle import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(70, 9), (70, 7), (70, 1193), (70, 1191), (70, 2369), (70, 2399), (9, 70), (1193, 70), (7111, 40),
                                 (7137, 40), (3, 5)])
@pytest.mark.parametrize("wrap", [False, True])
def test_box_blur_with_lines_left_over(w, h, wrap):
    r = min(2, w - 1, h - 1)
    v = np.random.default_rng(h).standard_normal((h, w))
    got = Gr.box_blur(torch.from_numpy(v).cuda(), r, 2, wrap_x=wrap)
    assert np.array_equal(got.cpu().numpy(), O.box_blur(v, r, 2, wrap=wrap))
