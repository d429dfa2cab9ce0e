"""The team of threads behind large copies to the host
(ouc_b200/csrc/hostcopy.h), compiled and run on the CPU with a thread in the
stream's place: every byte arrives for sizes around a chunk, several arrays
and more chunks than slots, and an error of a copy or of a wait, which a
worker thread meets, comes back as it is with the team ended."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <condition_variable>
#include <deque>
#include <functional>
#include <mutex>
#include "hostcopy.h"
using namespace ouc::host;

// copies run later, in order, on one thread; an event per slot
struct Stream {
    std::mutex m;
    std::condition_variable cv;
    std::deque<std::function<void()>> work;
    std::vector<int> recorded, reached;
    bool end = false;
    std::thread t;
    explicit Stream(int slots) : recorded(slots, 0), reached(slots, 0), t([this] { run(); }) {}
    ~Stream() {
        { std::lock_guard<std::mutex> g(m); end = true; }
        cv.notify_all();
        t.join();
    }
    void run() {
        std::unique_lock<std::mutex> g(m);
        for (;;) {
            cv.wait(g, [&] { return end || !work.empty(); });
            if (work.empty()) return;
            auto w = work.front();
            work.pop_front();
            g.unlock(); w(); g.lock();
            cv.notify_all();
        }
    }
    void push(int s, std::function<void()> f) {
        std::lock_guard<std::mutex> g(m);
        const int id = ++recorded[s];
        work.push_back([this, s, id, f] { f(); std::lock_guard<std::mutex> h(m); reached[s] = id; });
        cv.notify_all();
    }
    void wait(int s) {
        std::unique_lock<std::mutex> g(m);
        const int id = recorded[s];
        cv.wait(g, [&] { return reached[s] >= id; });
    }
};

int main() {
    int bad = 0, checked = 0;
    const size_t chunk = 1000;
    for (int slots : {1, 2, 8})
        for (int threads : {1, 2, 6})
            for (int shape = 0; shape < 6; ++shape) {
                const std::vector<std::vector<size_t>> shapes = {{}, {1}, {1000}, {999, 0, 1001}, {12345}, {8000, 3, 20001, 1000}};
                std::vector<std::vector<char>> dev, out;
                int total = 0;
                for (size_t n : shapes[shape]) {
                    dev.emplace_back(n);
                    out.emplace_back(n, (char)-1);
                    for (size_t k = 0; k < n; ++k) dev.back()[k] = (char)(k * 7 + n + k / 251);
                    total += (int)((n + chunk - 1) / chunk);
                }
                // no error; copy `f` refused with 7; the f-th wait fails with 9
                for (int f = -1; f < (total < 12 ? total : 12); ++f)
                    for (int kind = 0; kind < (f < 0 ? 1 : 2); ++kind) {
                        std::vector<HostCopy> copies;
                        for (size_t k = 0; k < dev.size(); ++k) copies.push_back({out[k].data(), dev[k].data(), dev[k].size()});
                        std::vector<char> ring(slots * chunk);
                        std::atomic<int> waits{0};
                        int copied = 0;
                        Stream st(slots);
                        const int e = ring_copy(
                            copies, ring.data(), chunk, slots, threads,
                            [&](int s, void* d, size_t n) {
                                if (kind == 0 && copied++ == f) return 7;
                                char* to = ring.data() + s * chunk;
                                st.push(s, [=] { memcpy(to, d, n); });
                                return 0;
                            },
                            [&](int s) {
                                if (kind == 1 && waits++ == f) return 9;
                                st.wait(s);
                                return 0;
                            });
                        bad += e != (f < 0 ? 0 : kind == 0 ? 7 : 9);
                        if (e == 0) bad += out != dev;
                        ++checked;
                    }
            }
    std::printf("%d %d\n", checked, bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_bytes_and_errors(tmp_path):
    src = tmp_path / "r.cpp"
    src.write_text(SRC)
    exe = tmp_path / "r"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "ouc_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    checked, bad = map(int, r.stdout.split())
    assert checked > 100 and bad == 0 and r.returncode == 0, r.stdout
