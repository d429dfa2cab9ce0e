"""Order of ouc_forward_noalloc's launches.  A step kernel reads its shot
descriptor and model before it waits for the launch ahead, so it may be
launched programmatically (overlapping that launch) only behind another step
kernel, never behind the kernels that write the descriptor and the model.
The first test captures the call into a graph, which runs nothing, and looks
at its edges; the second queues runs of different geometry without a
synchronisation between them and compares each with ouc_forward."""
import ctypes as C

import numpy as np
import pytest

import ouc_b200 as o
from helpers import rel_l2

pytestmark = pytest.mark.gpu

TOL_GATHER = 1e-5   # the parity tests' gather tolerance
KERNEL, PROGRAMMATIC = 0, 1   # CU_GRAPH_NODE_TYPE_KERNEL, CU_GRAPH_DEPENDENCY_TYPE_PROGRAMMATIC


class EdgeData(C.Structure):
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


class KernelParams(C.Structure):   # CUDA_KERNEL_NODE_PARAMS_v2
    _fields_ = [("func", C.c_void_p), ("dims", C.c_uint * 7), ("params", C.c_void_p), ("extra", C.c_void_p),
                ("kern", C.c_void_p), ("ctx", C.c_void_p)]


def _case(seed, nx, nz, L, N, nt, sx, sz):
    import torch
    rng = np.random.default_rng(seed)
    X, Z = nx + 2 * L, nz + 2 * L
    vp = rng.uniform(1800.0, 4200.0, (X, Z)).astype(np.float32)
    vs = (vp / 1.8).astype(np.float32)
    w, _ = o.ricker(40.0, 8e-4, nt)
    cfg = o.Config(nx=nx, nz=nz, npml=L, dx=10.0, dz=10.0, dt=8e-4, nt=nt, half_order=N, model_layout=o.MODEL_PADDED)
    shot = o.Shot(sx, sz, 2)
    with o.Context(cfg, vp, vs) as ctx:
        ref = ctx.forward(shot, w)[:2]
    dev = [torch.from_numpy(a).cuda() for a in (vp, vs, w)]
    out = [torch.full(ref[0].shape, float("nan"), device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    return cfg, shot, dev, out, ref


def _call(case, stream):
    cfg, shot, dev, out, _ = case
    c, s = cfg.c(), shot.c()
    c.stream = stream
    rc = o.lib().ouc_forward_noalloc(C.byref(c), C.byref(s), *(t.data_ptr() for t in dev + out))
    assert rc == 0, rc


def _check(case):
    for got, ref in zip(case[3], case[4]):
        assert np.abs(ref).max() > 0
        assert rel_l2(got.cpu().numpy(), ref) <= TOL_GATHER


# 16-row, 24-row, two small tiles per SM, 16 x 64 tiles
@pytest.mark.parametrize("nx,nz,N", [(60, 50, 5), (230, 233, 6), (301, 215, 5), (700, 300, 2)])
def test_programmatic_edges_join_step_kernels_only(nx, nz, N):
    import torch
    nt = 5
    case = _case(nx, nx, nz, 14, N, nt, nx // 2, 3)
    st = torch.cuda.Stream()
    _call(case, st.cuda_stream)   # set-up of the device, outside any capture
    torch.cuda.synchronize()
    _check(case)

    cu = C.CDLL("libcuda.so.1")
    stream, graph = C.c_void_p(st.cuda_stream), C.c_void_p()
    assert cu.cuStreamBeginCapture_v2(stream, 1) == 0   # thread-local mode
    try:
        _call(case, st.cuda_stream)
    finally:
        assert cu.cuStreamEndCapture(stream, C.byref(graph)) == 0
    n = C.c_size_t()
    assert cu.cuGraphGetEdges_v2(graph, None, None, None, C.byref(n)) == 0
    a, b, e = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (EdgeData * n.value)()
    assert cu.cuGraphGetEdges_v2(graph, a, b, e, C.byref(n)) == 0

    def kernel(node):
        kind, p = C.c_int(-1), KernelParams()
        assert cu.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        assert kind.value == KERNEL
        assert cu.cuGraphKernelNodeGetParams_v2(C.c_void_p(node), C.byref(p)) == 0
        return p.func, p.kern

    early = [(kernel(a[i]), kernel(b[i])) for i in range(n.value) if e[i].type == PROGRAMMATIC]
    assert cu.cuGraphDestroy(graph) == 0
    assert len(early) == nt - 1                       # step 0 waits for the set-up as a whole
    assert all(x == y and any(x) for x, y in early)   # one step kernel behind another


def test_runs_of_other_geometry_back_to_back():
    import torch
    cases = [_case(1, 60, 50, 14, 5, 40, 30, 3), _case(2, 150, 41, 10, 2, 30, 9, 20), _case(3, 41, 233, 20, 6, 25, 40, 12)]
    st = torch.cuda.Stream()
    _call(cases[0], st.cuda_stream)
    torch.cuda.synchronize()
    for _ in range(3):
        for case in cases:
            for t in case[3]:
                t.fill_(float("nan"))
        torch.cuda.synchronize()
        for case in cases:
            _call(case, st.cuda_stream)
        torch.cuda.synchronize()
        for case in cases:
            _check(case)
