"""The corrector's convolutions and weight gradients with enough work items that
every CTA comes back to each of its two pipeline stages more than once (600
and 630 items of a convolution on 148 CTAs, twice that of a weight gradient),
against the CPU restatement oracle/cnn.py with the tolerances of
test_corrector_gpu.py."""
import numpy as np
import pytest

from ouc_b200.corrector import Net
from oracle import cnn

pytestmark = pytest.mark.gpu

TOL_OUT = 2e-3
TOL_GRAD = 2e-2


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("n,H,W", [(4, 300, 130), (3, 417, 201)])
def test_stages_in_turn(n, H, W):
    import torch
    rng = np.random.default_rng(H)
    p = cnn.init_params(seed=5)
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
    y = dy.cpu().numpy()
    assert _rel(y, y_ref) <= TOL_OUT
    # and row by row: a stage taken too early would spoil single items
    for k in range(n):
        for h in range(H):
            assert _rel(y[k, h], y_ref[k, h]) <= 10 * TOL_OUT, (k, h)
    k = 0
    for ci, co in cnn.DIMS:
        nw = co * ci * cnn.TAPS
        assert _rel(g[k:k + nw], g_ref[k:k + nw]) <= TOL_GRAD
        assert _rel(g[k + nw:k + nw + co], g_ref[k + nw:k + nw + co]) <= TOL_GRAD
        k += nw + co
