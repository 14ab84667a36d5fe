"""The range of a Similarity sample's offsets (csrc/geometry.cuh), compiled here: what the dispatches ask before they keep an offset in
32 bits must hold for every tap and every patch corner of the shape."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include "geometry.cuh"

using simnets::SimGeo;
static SimGeo shape(int C, int H, int W, int bh, int bw, int sh, int sw, int ph, int pw) {
    SimGeo g = {};
    g.B = g.M = 1; g.C = C; g.H = H; g.W = W; g.bh = bh; g.bw = bw; g.sh = sh; g.sw = sw; g.ph = ph; g.pw = pw;
    g.oh = (H + 2 * ph - bh) / sh + 1; g.ow = (W + 2 * pw - bw) / sw + 1;
    return g;
}
#define EXPECT(what) do { if (!(what)) { std::printf("line %d: %s\n", __LINE__, #what); return 1; } } while (0)
int main() {
    std::srand(1);
    for (int i = 0; i < 20000; ++i) {
        const int bh = 1 + std::rand() % 6, bw = 1 + std::rand() % 6, ph = std::rand() % 6, pw = std::rand() % 6;
        const SimGeo g = shape(1 + std::rand() % 4, std::max(1, bh - 2 * ph) + std::rand() % 6, std::max(1, bw - 2 * pw) + std::rand() % 9, bh, bw, 1 + std::rand() % 3,
                               1 + std::rand() % 3, ph, pw);
        long long tap = 0;
        for (int c = 0; c < g.C; ++c)
            for (int kh = 0; kh < g.bh; ++kh)
                for (int kw = 0; kw < g.bw; ++kw) tap = std::max(tap, (long long)(c * g.H + kh) * g.W + kw);
        EXPECT(!simnets::sim_offsets_below(g, tap) && simnets::sim_offsets_below(g, tap + 1));
    }
    // the line between 31 and 32 bits of a byte offset, and of an element's
    EXPECT(simnets::sim_offsets_below(shape(1, 1 << 14, (1 << 15) - 3, 1, 1, 1, 1, 0, 0), 1LL << 29));
    EXPECT(!simnets::sim_offsets_below(shape(3, 1 << 14, 1 << 14, 1, 1, 56, 56, 0, 0), 1LL << 29));
    EXPECT(!simnets::sim_offsets_below(shape(1, 17, 1 << 25, 17, 1, 1, 512, 0, 0), 1LL << 29));
    EXPECT(!simnets::sim_offsets_below(shape(1, 1, 1 << 25, 18, 1, 1, 512, 17, 0), 1LL << 29));          // rows of the block beyond the image
    EXPECT(simnets::sim_offsets_below(shape(3, 1 << 14, 1 << 14, 1, 1, 56, 56, 0, 0), 1LL << 31));
    EXPECT(!simnets::sim_offsets_below(shape(33, 8200, 8200, 1, 1, 64, 64, 0, 0), 1LL << 31));
    EXPECT(!simnets::sim_offsets_below(shape(1, 46342, 46342, 1, 1, 1, 1, 0, 0), 1LL << 31));          // corners beyond 32 bits, on either side
    EXPECT(simnets::sim_offsets_below(shape(1, 46342, 46338, 3, 1, 1, 1, 0, 0), 1LL << 31));
    EXPECT(!simnets::sim_offsets_below(shape(1, 1, 1 << 27, 16, 1, 1, 512, 16, 0), 1LL << 31));
    // nothing that lies in a sample of fewer than 2^29 values, blocks inside the image, is refused
    EXPECT(simnets::sim_offsets_below(shape(1, 16384, 32767, 1, 1, 1, 1, 0, 0), 1LL << 29));
    EXPECT(simnets::sim_offsets_below(shape(8, 64, (1 << 20) - 1, 64, 5, 1, 1, 63, 4), 1LL << 29));
    return 0;
}
"""


def test_no_offset_of_a_shape_is_beyond_what_its_range_says(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "range.cpp", tmp_path / "range"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", str(src), "-o", str(exe), "-isystem", include, "-I", os.path.join(ROOT, "simnets_tf_b200", "csrc")])
    got = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert got.returncode == 0, got.stdout
