"""The list of launch shapes (csrc/launch_fits.h) on the CPU: it stays bounded
however many shapes pass through it, never answers with another shape's
figure, and keeps the latest ones, from several threads too."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cstdio>
#include <thread>
#include "launch_fits.h"
static int figure(size_t shape) { return 1 + (int)(shape % 7); }
int main() {
    mgv::LaunchFits fits;
    const char kernels[3] = {};
    auto pass = [&](size_t from, size_t to) {
        for (size_t s = from; s < to; ++s) {
            int n = -1;
            const void* k = kernels + s % 3;
            if (fits.find(k, 512, s, &n) && n != figure(s)) return 1;
            fits.add(k, 512, s, figure(s));
        }
        return 0;
    };
    if (pass(0, 100000) || fits.size() > mgv::LaunchFits::kMost) return 1;
    for (size_t s = 100000 - mgv::LaunchFits::kMost; s < 100000; ++s) {
        int n = -1;
        if (!fits.find(kernels + s % 3, 512, s, &n) || n != figure(s)) return 2;
        if (fits.find(kernels + s % 3, 256, s, &n) || fits.find(kernels + (s + 1) % 3, 512, s, &n)) return 3;
    }
    int bad[4] = {};
    std::vector<std::thread> ts;
    for (int t = 0; t < 4; ++t) ts.emplace_back([&, t] { bad[t] = pass(20 * t, 20 * t + 5000); });
    for (auto& t : ts) t.join();
    if (bad[0] | bad[1] | bad[2] | bad[3] || fits.size() > mgv::LaunchFits::kMost) return 4;
    std::puts("ok");
    return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_launch_fits(tmp_path):
    src, exe = tmp_path / "fits.cpp", tmp_path / "fits"
    src.write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(REPO, "multigpu-vector_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out
