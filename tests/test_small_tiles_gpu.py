"""Tile shapes of the step kernels.  The library picks 32 x 64, 16 x 64 or
small tiles by the number of tiles of a launch; every shape must give the
x-marching kernel's results (an independent geometry) bit for bit.  Each grid
below lands in another shape on 148 SMs, at the edges of its tiles: one cell
more or less than whole tiles, remainders in both directions, the narrowest
interior (4N), and batches whose reconstruction and receiver launches share a
launch or run beside each other."""
import numpy as np
import pytest

import ouc_b200 as o

pytestmark = pytest.mark.gpu


def _run(seg, nx, nz, L, N, n, nt, **kw):
    rng = np.random.default_rng(nx * 1000 + nz)
    vp = rng.uniform(1800.0, 4200.0, (nx, nz)).astype(np.float32)
    cfg = o.Config(nx=nx, nz=nz, npml=L, dx=10.0, dz=8.0, dt=8e-4, nt=nt, half_order=N, max_batch=n, **kw)
    w, t0 = o.ricker(40.0, 8e-4, nt)
    # sources near the corners and edges of tiles, one on the boundary ring
    shots = [o.Shot(min(nx - 1, 1 + k * (nx // n)), (7 * k) % nz, 2, k % 2 if n == 1 else 0, 5, k & 1) for k in range(n)]
    rho = (2000.0 + 0.1 * vp).astype(np.float32) if kw.get("density") else None
    with o.Context(cfg, vp, (vp / 1.8).astype(np.float32), rho) as ctx:
        ctx.set_step_kernel(seg)
        out = list(ctx.forward(shots[0], w, fields=True))
        for im in ctx.rtm_batch(shots, w):
            out += im
        return out + list(ctx.stack(reset=True))


@pytest.mark.parametrize("nx,nz,L,N,n,kw", [
    (20, 20, 6, 5, 1, {}),                                    # narrowest interior; 16-row tiles, one wave
    (103, 87, 12, 6, 1, dict(density=1)),                     # 127 x 111: one short of whole tiles
    (97, 65, 16, 2, 1, dict(strip_precision=1)),              # 129 x 97: one over; f16 strips
    (201, 223, 20, 5, 1, dict(compensated_image=1)),          # 24-row tiles (forward), two per SM (back-steps)
    (256, 233, 20, 6, 1, dict(image_align=1, strip_level=1)),  # 24-row tiles
    (301, 215, 21, 5, 1, {}),                                 # two 16-row CTAs per SM
    (90, 70, 10, 5, 5, dict(strip_precision=2)),              # the same from a batch
    (333, 190, 22, 2, 3, {}),                                 # 16 x 64 tiles
    (180, 131, 18, 6, 6, dict(snapshot_every=3)),
    (600, 261, 30, 5, 4, {}),                                 # forward 16 x 64, back-steps 32 x 64
])
def test_tile_shapes_match_the_marching_kernel(nx, nz, L, N, n, kw):
    nt = 60
    a = _run(0, nx, nz, L, N, n, nt, **kw)
    b = _run(64, nx, nz, L, N, n, nt, **kw)
    assert np.abs(a[0]).max() > 0
    for k, (x, y) in enumerate(zip(a, b)):
        np.testing.assert_array_equal(x, y, err_msg=f"output {k}")
