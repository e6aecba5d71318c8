"""coarse_near, the integer test of the near filter, on the CPU: never false for two positions within
the cut, over the whole range of 16-bit coordinates, and without an overflow of signed arithmetic (the
kernels' function is compiled for the host with the compiler's own check of that)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")

SOURCE = r"""
#include <cstdio>
#include <cstdint>
#include <cmath>
#include <random>
#include <initializer_list>
#include "pbd_device.cuh"
using namespace pbd;
int main() {
    std::mt19937_64 rng(5);
    // positions in [0, 128), their coarse coordinates as coarse_axis rounds them
    auto coarse = [](const double* p) {
        uint32_t q[3];
        for (int a = 0; a < 3; ++a) q[a] = (uint32_t)std::fmin(std::nearbyint(p[a] * 512.0), 65535.0);
        return make_uint2(q[0] | (q[1] << 16), q[2]);
    };
    std::uniform_real_distribution<double> u(0.0, 128.0), s(-1.0, 1.0);
    long lost = 0, far = 0;
    for (double cut : {0.3, 1.0, 2.4, 20.0, 49.0}) {
        const double steps = 512.0 * std::sqrt(cut * cut * 1.0001) + 3.0;
        const uint32_t limit = (uint32_t)std::fmin(steps * steps + 1.0, 4294967295.0);
        for (int k = 0; k < 400000; ++k) {
            double a[3], b[3], r2 = 0.0;
            for (int c = 0; c < 3; ++c) a[c] = u(rng);
            double d[3], n = 0.0;
            for (int c = 0; c < 3; ++c) { d[c] = s(rng); n += d[c] * d[c]; }
            const double len = (k & 1) ? cut * (1.0 - 1e-6) : 128.0 * (s(rng) + 1.0);   // at the cut; anywhere
            for (int c = 0; c < 3; ++c) {
                b[c] = std::fmin(std::fmax(a[c] + d[c] / std::sqrt(n) * len, 0.0), 127.999);
                r2 += (b[c] - a[c]) * (b[c] - a[c]);
            }
            if (k % 16 == 0)
                for (int c = 0; c < 3; ++c) { a[c] = (k >> (4 + c)) & 1 ? 127.999 : 0.0; b[c] = (k >> (7 + c)) & 1 ? 127.999 : 0.0; }
            if (k % 16 == 0) { r2 = 0.0; for (int c = 0; c < 3; ++c) r2 += (b[c] - a[c]) * (b[c] - a[c]); }
            const bool near = coarse_near(coarse(a), coarse(b), limit), in = r2 < cut * cut;
            if (in && !near) ++lost;
            if (!in && near && r2 > (cut + 0.02) * (cut + 0.02) && r2 < 63.0 * 63.0) ++far;
            if (coarse_near(coarse(a), coarse(b), 0u)) ++lost;
        }
    }
    std::printf("%ld lost, %ld far\n", lost, far);
    return lost || far ? 1 : 0;
}
"""


@pytest.mark.skipif(not (os.path.exists(NVCC) or shutil.which(NVCC)), reason="no nvcc")
def test_coarse_near_on_the_host(tmp_path):
    src, exe = tmp_path / "coarse.cu", tmp_path / "coarse"
    src.write_text(SOURCE)
    subprocess.run([NVCC, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O1", "-I", os.path.join(PKG, "csrc"),
                    "-Xcompiler", "-fsanitize=signed-integer-overflow,-fno-sanitize-recover=all", "-o", str(exe), str(src)],
                   check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
