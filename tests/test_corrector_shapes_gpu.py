"""Edges of the corrector convolutions' work items (4 image rows x 128
pixels, 2 rows for the weight gradients): images of one row, odd heights, widths one below, at and one above
128 and 256, the narrowest images, and more items than CTAs, against the CPU
restatement oracle/cnn.py with the tolerances of test_corrector_gpu.py (the
same operand roundings; FP32 accumulation in another order may move an
activation across a bfloat16 tie or a ReLU's zero)."""
import numpy as np
import pytest

from ouc_b200.corrector import Net
from oracle import cnn

pytestmark = pytest.mark.gpu

TOL_OUT = 2e-3
TOL_GRAD = 2e-2


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("n,H,W", [(1, 1, 1), (1, 1, 127), (2, 2, 128), (1, 3, 129), (3, 5, 17), (1, 7, 256), (2, 9, 257),
                                   (1, 299, 130), (5, 64, 33)])
def test_convolutions_at_item_edges(n, H, W):
    import torch
    rng = np.random.default_rng(n * 100 + H + W)
    p = cnn.init_params(seed=3)
    x = rng.normal(size=(n, H, W, cnn.DIMS[0][0])).astype(np.float32)
    gout = rng.normal(size=(n, H, W, 8)).astype(np.float32)
    ref = cnn.Net(p)
    y_ref = ref.forward(x)
    g_ref = ref.backward(gout)
    dx, dg = torch.from_numpy(x).cuda(), torch.from_numpy(gout).cuda()
    dy = torch.empty((n, H, W, 8), device="cuda")
    with Net(0, p) as net:
        net.forward_dev(n, H, W, dx.data_ptr(), dy.data_ptr())
        net.zero_grad()
        net.backward_dev(dg.data_ptr())
        torch.cuda.synchronize()
        g = net.grads()
        assert net.error() == 0
    assert _rel(dy.cpu().numpy(), y_ref) <= TOL_OUT
    k = 0
    for ci, co in cnn.DIMS:
        nw = co * ci * cnn.TAPS
        assert _rel(g[k:k + nw], g_ref[k:k + nw]) <= TOL_GRAD
        assert _rel(g[k + nw:k + nw + co], g_ref[k + nw:k + nw + co]) <= TOL_GRAD
        k += nw + co
