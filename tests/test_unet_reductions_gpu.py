"""The U-Net's bias and head gradients (pixel sums taken eight channels at a time over many blocks)
and the pooled and upsampled gradients, at the smallest batch and at pixel counts that leave a
block's rows partly empty, against torch autograd on the CPU. Bounds as test_unet_gpu's: the
device keeps its gradients in BF16 between layers, the reference does not."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from deeptime_gpu import unet as U  # noqa: E402

from .test_unet_gpu import reference, unpack  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 8, 512), (3, 24, 512), (1, 8, 1024)])
def test_bias_and_head_gradients_match_torch(B, H, W):
    rng = np.random.default_rng(B * H + W)
    model = U.UNet(seed=77)
    x = rng.standard_normal((B, H, W, 2)).astype(np.float32)
    t = rng.standard_normal((B, H, W)).astype(np.float32) * 0.1
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    model.loss_and_grad_dev(xd.data_ptr(), td.data_ptr(), B, H, W)
    got, ghw, ghb = unpack(model.gradients().astype(np.float64))
    convs, hw, hb = unpack(model.params().astype(np.float64))
    prm = ([(torch.tensor(w, requires_grad=True), torch.tensor(b, requires_grad=True)) for w, b in convs],
           torch.tensor(hw, requires_grad=True), torch.tensor(hb, requires_grad=True))
    reference(prm, torch.from_numpy(x).double(), torch.from_numpy(t).double()).backward()
    for (_, gb), (_, tb) in zip(got, prm[0]):
        want = tb.grad.numpy()
        assert np.linalg.norm(gb - want) <= 0.08 * np.linalg.norm(want) + 1e-12
    for g, p in ((ghw, prm[1]), (ghb, prm[2])):
        want = p.grad.numpy()
        assert np.linalg.norm(g - want) <= 0.02 * np.linalg.norm(want)
