"""Block reductions whose last block sums every block's partial: v.Av over a raster of thousands of tiles, call
after call on two inputs in turn, so that a partial of the call before would show. Each call gives its
input's first bits again, and the sum of the products to 1e-12 (both sums of 5e5 terms in FP64)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from deeptime_gpu import _lib as L  # noqa: E402
from deeptime_gpu import diffusion as D  # noqa: E402
from deeptime_gpu import inputs as I  # noqa: E402

pytestmark = pytest.mark.gpu


def test_the_dot_of_many_blocks_is_never_a_call_late():
    w, h, dx = 1024, 512, 10_000.0
    lib, dev, stream = L.lib(), torch.device("cuda"), torch.cuda.current_stream().cuda_stream
    d, c, _ = I.flexure_problem(w, h, 8.0, 3)
    td, tc = torch.from_numpy(d).to(dev), torch.from_numpy(c).to(dev)
    rng = np.random.default_rng(3)
    vs = [torch.from_numpy(s * rng.standard_normal((h, w))).to(dev) for s in (1.0, 1000.0)]
    ys = [torch.empty_like(td) for _ in vs]
    out = torch.empty((200, 2), dtype=torch.float64, device=dev)
    for k in range(200):
        for q in range(2):
            st = lib.dt_flex_operator_dot_noalloc(w, h, ctypes.c_double(dx), *(ctypes.c_void_p(t.data_ptr()) for t in (
                td, tc, vs[q], ys[q], out[k, q])), ctypes.c_void_p(stream))
            assert st == L.DT_OK, L.last_error()
    got = out.cpu().numpy()
    assert np.array_equal(got, np.broadcast_to(got[0], got.shape))
    for q in range(2):
        assert abs(got[0, q] - torch.sum(vs[q] * ys[q]).item()) <= 1e-12 * abs(got[0, q])


def test_a_solve_repeats_its_bits():
    w, h = 1000, 600
    rng = np.random.default_rng(5)
    z = 500.0 * rng.standard_normal((h, w))
    kd = 10.0 ** rng.uniform(-2.0, 1.0, (h, w))
    ws = D.Workspace(D.Dims(w, h, 2400.0, True))
    p = D.params(cycle=L.CYCLE_RBGS, precision=L.DIFF_MIXED_RELIABLE, stop=L.STOP_REL_RESIDUAL, tol=1e-10)
    first, rep = ws.solve_with(z, kd, 2.0e6, p)
    for _ in range(20):
        x, again = ws.solve_with(z, kd, 2.0e6, p)
        assert again.iterations == rep.iterations and np.array_equal(x, first)
