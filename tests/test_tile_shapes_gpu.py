"""Every tile shape of the step kernels on one and the same grid (the library
would choose one by the number of tiles; ouc_debug_tile_shape forces each):
the first-order step forward and backward, RTM batches, the FWI gradient (one
launch per back-step on small tiles, two streams on the others) and surveys of
uneven windows give the same bits on all of them.  The first-order results
also stay as close to the FP64 oracle as the oracle's own FP32 run: within
twice its error plus 1e-7, the bound of test_first_order_gpu.py."""
import numpy as np
import pytest

import ouc_b200 as o
from ouc_b200 import _lib
from helpers import rel_l2
from oracle.oracle import Shot

pytestmark = pytest.mark.gpu

SHAPES = (0, 1, 2, 3, 4, 5)   # by the rule; 32 x 64, 16 x 64, 24 x 32, 16 x 32 two per SM, 16 x 32


def _model(nx, nz, L):
    rng = np.random.default_rng(100 * nx + nz)
    vp = rng.uniform(1900.0, 3900.0, (nx, nz)).astype(np.float32)
    return vp, (vp / 1.8).astype(np.float32)


def _set_shape(ctx, shape):
    """False where the context's fields do not hold tiles of this shape."""
    try:
        ctx.debug_tile_shape(shape)
    except o.OucError as e:
        assert shape == 3 and e.code == _lib.OUC_EINVAL
        return False
    return True


def _same_on_all(ctx, run):
    """run(ctx) on every shape; returns the rule's result."""
    ref, ran = None, 0
    for shape in SHAPES:
        if not _set_shape(ctx, shape):
            continue
        out = run(ctx)
        ran += 1
        if ref is None:
            ref = out
            assert all(np.abs(a[np.isfinite(a)]).max() > 0 for a in ref)
        for k, (a, b) in enumerate(zip(out, ref)):
            np.testing.assert_array_equal(a, b, err_msg=f"shape {shape}, output {k}")
    assert ran >= 5
    return ref


@pytest.mark.parametrize("nx,nz,L,N", [(61, 47, 10, 5), (131, 88, 13, 6), (95, 201, 16, 2), (150, 60, 21, 5)])
def test_first_order(oracle, nx, nz, L, N):
    nt, dx, dt = 90, 8.0, 6e-4
    vp, vs = _model(nx, nz, L)
    w, _ = o.ricker(35.0, dt, nt)
    sx, sz, rz = nx - 1, 4, 2   # on the last interior column
    cfg = o.Config(nx=nx, nz=nz, npml=L, dx=dx, dz=dx, dt=dt, nt=nt, half_order=N)

    def run(ctx):
        gx, gz, f = ctx.forward_first_order(o.Shot(sx, sz, rz), w, fields=True)
        return gx, gz, f, ctx.backward_first_order(o.Shot(sx, sz, rz), gx, gz)

    with o.Context(cfg, vp, vs) as ctx:
        gx, gz, f, b = _same_on_all(ctx, run)
    vpp, vsp = (oracle.pad(np.pad(a, L), L) for a in (vp, vs))
    ax, az = oracle.profile(vpp, L)
    sh = Shot(X=nx + 2 * L, Z=nz + 2 * L, L=L, N=N, nt=nt, sx=sx + L, sz=sz + L, rz=rz + L, dx=dx, dz=dx, dt=dt)
    exact = oracle.forward_fo(sh, vpp, vsp, ax, az, w, fp64=True)
    single = oracle.forward_fo(sh, vpp, vsp, ax, az, w)
    bexact = oracle.backward_fo(sh, vpp, vsp, ax, az, gx, gz, fp64=True)
    bsingle = oracle.backward_fo(sh, vpp, vsp, ax, az, gx, gz)
    pairs = [("gx", gx, exact[0], single[0]), ("gz", gz, exact[1], single[1])]
    pairs += [(f"field {k}", f[k], exact[2][k], single[2][k]) for k in range(16)]
    pairs += [(f"backward field {k}", b[k], bexact[k], bsingle[k]) for k in range(16)]
    for name, got, e64, e32 in pairs:
        assert rel_l2(got, e64) <= 2 * rel_l2(e32, e64) + 1e-7, (name, rel_l2(got, e64), rel_l2(e32, e64))


@pytest.mark.parametrize("nx,nz,L,N,kw", [
    (61, 47, 10, 5, {}),
    (131, 88, 13, 6, dict(strip_precision=1)),
    (95, 201, 16, 2, dict(compensated_image=1, strip_level=1)),
    (150, 60, 21, 5, dict(snapshot_every=2)),
    (77, 90, 12, 6, dict(density=1)),
    (90, 77, 12, 6, dict(gradient=1)),
    (120, 104, 14, 5, dict(gradient=1, image_align=1)),
    (88, 61, 9, 2, dict(gradient=1)),
])
def test_rtm_and_gradient(nx, nz, L, N, kw):
    n, nt, dt = 3, 150, 6e-4
    vp, vs = _model(nx, nz, L)
    rho = (2000.0 + 0.1 * vp).astype(np.float32) if kw.get("density") or kw.get("gradient") else None
    w, t0 = o.ricker(35.0, dt, nt)
    cfg = o.Config(nx=nx, nz=nz, npml=L, dx=8.0, dz=8.0, dt=dt, nt=nt, half_order=N, max_batch=n, **kw)
    shots = [o.Shot(min(nx - 1, 3 + 31 * k), 2 + k, 2, t0=t0) for k in range(n)]

    def run(ctx):
        out = [a for im in ctx.rtm_batch(shots, w) for a in im] + list(ctx.stack(reset=True))
        return out + list(ctx.gradient(reset=True)) if kw.get("gradient") else out

    with o.Context(cfg, vp, vs, rho) as ctx:
        _same_on_all(ctx, run)


@pytest.mark.parametrize("nx,nz,L,N,apertures,precision", [
    (260, 57, 10, 5, [(0, 41), (37, 121), (90, 260)], 0),
    (401, 84, 14, 6, [(180, 221)], 1),
    (150, 120, 12, 2, [(0, 150), (60, 101), (109, 150), (5, 70)], 2),
])
def test_survey_windows(nx, nz, L, N, apertures, precision):
    nt, dt = 160, 6e-4
    vp, vs = _model(nx, nz, L)
    w, t0 = o.ricker(35.0, dt, nt)
    cfg = o.Config(nx=nx, nz=nz, npml=L, dx=8.0, dz=8.0, dt=dt, nt=nt, half_order=N, max_batch=len(apertures),
                   strip_precision=precision)
    shots = [o.Shot((a + b) // 2, 3, 2, t0=t0) for a, b in apertures]

    def run(ctx):
        recs = ctx.survey_forward(shots, apertures, w)
        images = ctx.survey_rtm(shots, apertures, w, recs)
        return [a for pair in recs + images for a in pair] + list(ctx.stack(reset=True))

    with o.Context(cfg, vp, vs) as ctx:
        _same_on_all(ctx, run)


def test_shapes_out_of_range_are_refused():
    vp, vs = _model(40, 40, 10)
    with o.Context(o.Config(nx=40, nz=40, npml=10, dx=8.0, dz=8.0, dt=6e-4, nt=10), vp, vs) as ctx:
        for shape in (-1, 6):
            with pytest.raises(o.OucError) as e:
                ctx.debug_tile_shape(shape)
            assert e.value.code == _lib.OUC_EINVAL
