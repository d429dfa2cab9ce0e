"""Host logic of the corrector kernels' two-stage pipeline
(ouc_b200/csrc/pipeline.h), compiled and run on the CPU with barriers that
complete a phase only when somebody waits for it: for every number of items,
and with the operands or a completion wait of every item running out,
* items are issued in order, each after its operands;
* when the issuing side returns, every commit that it made has been waited
  for, so that what the multiplications write can be released;
* it reports failure exactly when a wait ran out."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include "pipeline.h"
int main() {
    int bad = 0, checked = 0;
    for (int count = 0; count <= 9; ++count)
        for (int no_operands = -1; no_operands < count; ++no_operands)       // item whose operands never land
            for (int lost = -1; lost < 2; ++lost) {                          // stage whose completion waits run out
                int issued = 0, committed[2] = {0, 0}, waited[2] = {0, 0};   // commits per stage, and those waited for
                const bool ok = ouc::run_items(
                    count,
                    [&](int k) { bad += k != issued; return k != no_operands; },
                    [&](int k) { bad += k != issued; ++issued; ++committed[k & 1]; },
                    [&](int s, unsigned parity) {
                        // a bounded wait for the phase of this parity: the last commit's, which
                        // completes the earlier ones of the stage too
                        bad += committed[s] == 0 || parity != ((unsigned)(committed[s] - 1) & 1u);
                        waited[s] = committed[s];
                        return s != lost;
                    });
                bad += issued != (no_operands < 0 ? count : no_operands);
                for (int s = 0; s < 2; ++s) bad += waited[s] != committed[s];
                bad += ok != (no_operands < 0 && (lost < 0 || committed[lost] == 0));
                ++checked;
            }
    std::printf("%d %d\n", checked, bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_commit_is_waited_for(tmp_path):
    src = tmp_path / "p.cpp"
    src.write_text(SRC)
    exe = tmp_path / "p"
    cuda_inc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "ouc_b200", "csrc"), "-I", cuda_inc,
                    str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    checked, bad = map(int, r.stdout.split())
    assert checked > 100 and bad == 0 and r.returncode == 0, r.stdout
