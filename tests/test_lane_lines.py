"""Which line of the warp-exchanged passes a lane works on (anyfft.cuh): every
line has its lanes once, and lanes without a line keep to a line of their own
warp.  A lane that read another warp's line would race with its in-place
transform.  Runs the header's own index functions on the host."""

import os
import subprocess

import pytest
from conftest import ROOT

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
CSRC = os.path.join(ROOT, "surfacelets.jl_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "anyfft.cuh"
using namespace sfl;
template <int N>
bool check() {
    using L = AnyLine<N>;
    for (int warps : {1, 4, 7, 16, 32})
        for (int n : {1, 2, 3, 5, 17, 49, 55, 64, 109, 130})
            for (int pairs = 0; pairs < 2; ++pairs) {
                std::vector<int> lanes(n, 0);
                for (int w = 0; w < warps; ++w)
                    for (int l0 = w * L::LPW; l0 < n; l0 += warps * L::LPW)
                        for (int lane = 0; lane < 32; ++lane) {
                            const int s = lane / L::N2;
                            const LaneLine a = pairs ? any_lane_pair<N>(l0, s, n) : any_lane_line<N>(l0, s, n);
                            if (a.l < l0 || a.l >= l0 + L::LPW || a.l >= n) return false;
                            if (a.valid) ++lanes[a.l];
                        }
                for (int c : lanes)
                    if (c != L::N2) return false;
            }
    return true;
}
int main() {
    int bad = 0;
#define SFL_ANY_CASE(N_) if (!check<N_>()) { std::printf("length %d\n", N_); ++bad; }
    SFL_ANY_LENGTHS(SFL_ANY_CASE)
    return bad != 0;
}
"""


@pytest.mark.skipif(not os.path.exists(NVCC), reason="needs nvcc")
def test_lanes_keep_to_their_warps_lines(tmp_path):
    src, exe = tmp_path / "lanes.cu", tmp_path / "lanes"
    src.write_text(PROGRAM)
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-I",
                    CSRC, "-I", os.path.join(ROOT, "include"), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
