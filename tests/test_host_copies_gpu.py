"""Copies of large results to the host: below 4 MiB direct, from 4 MiB with the
pages touched first, from 32 MiB through the pinned ring (whole and partial
1 MiB chunks, more chunks than slots).  A pinned destination always takes the
direct copy, so both must hold the same bytes."""
import ctypes as C

import numpy as np
import pytest

import ouc_b200 as o
from ouc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(60, 50), (480, 400), (1500, 1100), (2003, 1501)])
def test_pageable_equals_pinned(nx, nz):
    import torch
    L, nt = 10, 6
    vp = np.random.default_rng(nx).uniform(1800.0, 4200.0, (nx, nz)).astype(np.float32)
    w = np.ones(nt, np.float32)
    with o.Context(o.Config(nx=nx, nz=nz, npml=L, dx=10.0, dz=10.0, dt=1e-3, nt=nt), vp, (vp / 1.8).astype(np.float32)) as ctx:
        shot = o.Shot(nx // 2, nz // 2, 2)
        _, _, f = ctx.forward(shot, w, fields=True)
        pin = torch.full((6, ctx.X, ctx.Z), float("nan"), pin_memory=True).numpy()
        fp, sc = C.POINTER(C.c_float), shot.c()
        _lib.check(_lib.lib().ouc_forward(ctx.handle, C.byref(sc), w.ctypes.data_as(fp), None, None, pin.ctypes.data_as(fp)), ctx.handle)
    assert np.abs(f).max() > 0
    np.testing.assert_array_equal(f, pin)
    np.testing.assert_array_equal(f[0], f[2] + f[4])   # U = P + S
    np.testing.assert_array_equal(f[1], f[3] + f[5])
