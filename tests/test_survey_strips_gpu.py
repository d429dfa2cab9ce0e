"""Surveys whose windows are narrower than their model, at every precision of
the boundary strips: the RTM images of a batch of uneven windows equal, bit
for bit, single-shot runs of contexts created on the windows (16-bit strips
carry an exponent per field and step, so the last step's strip must be
converted by the window's own ring, not the model's)."""
import numpy as np
import pytest

import ouc_b200 as o

pytestmark = pytest.mark.gpu


# one narrow window of a wide model, and a batch of uneven ones
@pytest.mark.parametrize("nx,nz,L,N,apertures", [
    (700, 60, 12, 5, [(330, 380)]),
    (310, 84, 14, 6, [(0, 41), (100, 170), (269, 310)]),
    (200, 50, 10, 2, [(0, 200), (20, 61)]),
])
@pytest.mark.parametrize("precision", [o.api.PREC_FP32, o.api.PREC_FP16, o.api.PREC_BF16])
def test_narrow_windows_equal_window_runs(nx, nz, L, N, apertures, precision):
    nt = 240
    rng = np.random.default_rng(nx)
    vp = np.pad(rng.uniform(2200.0, 3800.0, (nx, nz)).astype(np.float32), L, mode="edge")
    vs = (vp / 1.8).astype(np.float32)
    w, t0 = o.ricker(35.0, 8e-4, nt)

    def cfg(width, batch):
        return o.Config(nx=width, nz=nz, npml=L, dx=8.0, dz=8.0, dt=8e-4, nt=nt, half_order=N, max_batch=batch,
                        model_layout=o.MODEL_PADDED, strip_precision=precision)

    shots = [o.Shot((a + b) // 2, 3, 2, t0=t0) for a, b in apertures]
    with o.Context(cfg(nx, len(apertures)), vp, vs) as ctx:
        got = ctx.survey_rtm(shots, apertures, w)
    for s, (x0, x1), images in zip(shots, apertures, got):
        with o.Context(cfg(x1 - x0, 1), np.ascontiguousarray(vp[x0:x1 + 2 * L]),
                       np.ascontiguousarray(vs[x0:x1 + 2 * L])) as win:
            ref = win.rtm_shot(o.Shot(s.sx - x0, s.sz, s.rz, t0=t0), w)
        for a, b in zip(images, ref):
            assert np.isfinite(b).all() and np.abs(b).max() > 0
            np.testing.assert_array_equal(a, b)
