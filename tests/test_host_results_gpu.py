"""Forward results into host arrays of either kind: gathers and fields that are
pageable, pinned or left out, large enough that the pages of the pageable ones
are touched ahead of the copies, hold the same bytes in every combination."""
import ctypes as C
import itertools

import numpy as np
import pytest

import ouc_b200 as o
from ouc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,nt", [(40, 30, 12), (500, 60, 2100), (700, 1300, 8)])
def test_every_combination_of_arrays(nx, nz, nt):
    import torch
    vp = np.random.default_rng(nx).uniform(1800.0, 4200.0, (nx, nz)).astype(np.float32)
    w = np.ones(nt, np.float32)
    fp = C.POINTER(C.c_float)
    cfg = o.Config(nx=nx, nz=nz, npml=10, dx=10.0, dz=10.0, dt=1e-3, nt=nt, gather_layout=o.GATHER_TX)

    def array(kind, shape):
        if kind == "none":
            return None
        return torch.full(shape, float("nan"), pin_memory=kind == "pinned").numpy()

    with o.Context(cfg, vp, (vp / 1.8).astype(np.float32)) as ctx:
        shot = o.Shot(nx // 2, 3, 2)
        ref = ctx.forward(shot, w, fields=True)
        assert all(np.abs(r).max() > 0 for r in ref)
        sc = shot.c()
        for kinds in itertools.product(("none", "pageable", "pinned"), repeat=3):
            out = [array(k, r.shape) for k, r in zip(kinds, ref)]
            _lib.check(_lib.lib().ouc_forward(ctx.handle, C.byref(sc), w.ctypes.data_as(fp),
                                              *(None if a is None else a.ctypes.data_as(fp) for a in out)), ctx.handle)
            for a, r in zip(out, ref):
                if a is not None:
                    np.testing.assert_array_equal(a, r, err_msg=str(kinds))
