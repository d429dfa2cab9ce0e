"""The first-order step's bounded copy wait, as test_copy_wait_gpu.py has it for
the second order: with the test hook on, the tiles' waits run out, the call
returns OUC_ETIMEOUT, and the context then reproduces a fresh one's results.
The grids take small tiles (one and two per SM) and 16 x 64 tiles."""
import numpy as np
import pytest

import ouc_b200 as o
from ouc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(48, 40), (310, 230), (700, 300)])
def test_copy_wait_times_out_and_context_recovers(nx, nz):
    vp = np.random.default_rng(nx).uniform(2500.0, 2700.0, (nx, nz)).astype(np.float32)
    vs = (vp / 1.8).astype(np.float32)
    cfg = o.Config(nx=nx, nz=nz, npml=12, dx=10.0, dz=10.0, dt=1e-3, nt=6, half_order=5)
    w = np.array([1.0, -0.5, 0.25, 0, 0, 0], np.float32)
    shot = o.Shot(sx=20, sz=4, rz=4)
    with o.Context(cfg, vp, vs) as ref:
        gx0, gz0, f0 = ref.forward_first_order(shot, w, fields=True)
        b0 = ref.backward_first_order(shot, gx0, gz0)
    assert np.abs(gz0).max() > 0 and np.abs(b0).max() > 0
    with o.Context(cfg, vp, vs) as ctx:
        for call in (lambda: ctx.forward_first_order(shot, w, fields=True), lambda: ctx.backward_first_order(shot, gx0, gz0)):
            ctx.debug_copy_stall(True)
            with pytest.raises(o.OucError) as e:
                call()
            assert e.value.code == _lib.OUC_ETIMEOUT
            ctx.debug_copy_stall(False)
        gx, gz, f = ctx.forward_first_order(shot, w, fields=True)
        b = ctx.backward_first_order(shot, gx0, gz0)
    for got, ref in ((gx, gx0), (gz, gz0), (f, f0), (b, b0)):
        np.testing.assert_array_equal(got, ref)
