"""Images of a batch that the caller sends to one shared array (it only wants
the stack, say): the copies are made in the order of the shots, so the array
holds the last shot's image, also when together they are large enough for the
ring of hostcopy.h, whose threads would write them in any order."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

import ouc_b200 as o
from ouc_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "hostcopy.h"
using namespace ouc::host;
int main() {
    int bad = 0, checked = 0;
    static char mem[64];
    std::srand(3);
    for (int round = 0; round < 20000; ++round) {
        std::vector<HostCopy> c;
        int used[64] = {};
        bool shared = false;
        for (int n = std::rand() % 5; n > 0; --n) {
            const int at = std::rand() % 60, bytes = std::rand() % (64 - at < 12 ? 64 - at : 12);
            c.push_back({mem + at, nullptr, (size_t)bytes});
            for (int k = at; k < at + bytes; ++k) shared = ++used[k] > 1 || shared;
        }
        bad += overlapping(c) != shared;
        ++checked;
    }
    std::printf("%d %d\n", checked, bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_overlap_of_destinations(tmp_path):
    src = tmp_path / "o.cpp"
    src.write_text(SRC)
    exe = tmp_path / "o"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "ouc_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    checked, bad = map(int, r.stdout.split())
    assert checked > 1000 and bad == 0 and r.returncode == 0, r.stdout


@pytest.mark.gpu
def test_shared_array_holds_the_last_image():
    nx, nz, nt, n = 600, 500, 40, 16   # 32 images, 38 MB
    vp = np.random.default_rng(1).uniform(1800.0, 4200.0, (nx, nz)).astype(np.float32)
    w, _ = o.ricker(40.0, 1e-3, nt)
    cfg = o.Config(nx=nx, nz=nz, npml=10, dx=10.0, dz=10.0, dt=1e-3, nt=nt, max_batch=n)
    shots = [o.Shot(15 + 37 * k, 2, 2) for k in range(n)]
    FP = C.POINTER(C.c_float)
    with o.Context(cfg, vp, (vp / 1.8).astype(np.float32)) as ctx:
        ref = ctx.rtm_batch(shots, w)[-1]
        sh = (_lib.ouc_shot * n)(*[s.c() for s in shots])
        for _ in range(5):
            out = [np.full((nx, nz), np.nan, np.float32) for _ in range(2)]
            ptr = [(FP * n)(*[a.ctypes.data_as(FP)] * n) for a in out]
            _lib.check(_lib.lib().ouc_rtm_batch(ctx.handle, n, sh, w.ctypes.data_as(FP), None, None, *ptr), ctx.handle)
            for a, r in zip(out, ref):
                np.testing.assert_array_equal(a, r)
