"""The convolutions' two kernels take their products in the same order (by tap, then channel, 16 at a time), so
which one a layer gets, by the number of its tiles, does not show: an image alone, whose coarser layers have few
tiles, gives the bits it gives in a batch of sixteen."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from deeptime_gpu import unet as U  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(16, 64, 512), (16, 256, 512), (5, 24, 1024)])
def test_an_image_alone_gives_the_bits_of_the_batch(B, H, W):
    model = U.UNet(seed=11)
    x = torch.from_numpy(np.random.default_rng(H).standard_normal((B, H, W, 2)).astype(np.float32)).cuda()
    batch, alone = (torch.empty((B, H, W), dtype=torch.float32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    model.predict_dev(x.data_ptr(), batch.data_ptr(), B, H, W)
    for k in range(B):
        model.predict_dev(x[k].data_ptr(), alone[k].data_ptr(), 1, H, W)
    torch.cuda.synchronize()
    assert torch.equal(batch, alone)


def test_small_predictions_keep_their_speed():
    # on the resident-region kernel alone a 64 x 512 image took 475 us of 674 for eight times the pixels, on
    # the line kernel 285 of 622: 0.70 and 0.46, the line between them
    model = U.UNet(seed=11)
    t = {}
    for H in (64, 512):
        x, y = torch.zeros((1, H, 512, 2), device="cuda"), torch.empty((1, H, 512), device="cuda")
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        best = []
        for _ in range(12):
            torch.cuda.synchronize()
            a.record()
            model.predict_dev(x.data_ptr(), y.data_ptr(), 1, H, 512)
            torch.cuda.synchronize()
            b.record()
            b.synchronize()
            best.append(a.elapsed_time(b))
        t[H] = min(best)
    assert t[64] < 0.57 * t[512], t
