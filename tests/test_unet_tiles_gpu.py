"""The U-Net's convolutions and weight gradients at heights that leave a block's rows partly outside
the image (1, 2, 4 and 3, 6, 12 rows at the coarser levels) and at an odd batch, against torch autograd
on the CPU. Bounds as test_unet_gpu's (the device keeps its gradients in BF16 between layers, the
reference does not)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from deeptime_gpu import unet as U  # noqa: E402

from .test_unet_gpu import reference, unpack  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W", [(1, 8, 512), (3, 24, 512), (1, 40, 1024)])
def test_loss_and_weight_gradients_at_partial_rows(B, H, W):
    rng = np.random.default_rng(H + W)
    model = U.UNet(seed=31)
    x = rng.standard_normal((B, H, W, 2)).astype(np.float32)
    t = rng.standard_normal((B, H, W)).astype(np.float32) * 0.1
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    loss = model.loss_and_grad_dev(xd.data_ptr(), td.data_ptr(), B, H, W)
    got = unpack(model.gradients().astype(np.float64))[0]
    convs, hw, hb = unpack(model.params().astype(np.float64))
    prm = ([(torch.tensor(w, requires_grad=True), torch.tensor(b, requires_grad=True)) for w, b in convs],
           torch.tensor(hw, requires_grad=True), torch.tensor(hb, requires_grad=True))
    ref = reference(prm, torch.from_numpy(x).double(), torch.from_numpy(t).double())
    ref.backward()
    assert abs(loss - ref.item()) <= 2e-3 * abs(ref.item())
    for k, ((gw, _), (tw, _)) in enumerate(zip(got, prm[0])):
        want = tw.grad.numpy()
        if k == 0:  # the input's padding channels carry no gradient
            gw, want = gw[:, :2], want[:, :2]
        assert np.linalg.norm(gw - want) <= 0.08 * np.linalg.norm(want) + 1e-12, k
