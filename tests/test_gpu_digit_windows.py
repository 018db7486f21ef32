"""The norms that the length of an exact accumulation is chosen from (csrc/digits.cuh,
dg_windows): over any blocks that follow one another, since a split of the contraction may
start at any block.  A small program compares them with the definition."""
import os
import subprocess

import pytest

from tdscha_gb300 import build

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "digits.cuh"
using namespace tdscha;
void tdscha::set_error(const char *, ...) {}
int main() {
    std::mt19937 gen(1);
    const int sizes[][3] = {{1, 64, 1}, {2, 64, 2}, {1, 128, 3}, {3, 64, 8}, {2, 128, 31}, {1, 64, 33},
                            {2, 64, 64}, {1, 64, 71}, {2, 64, 200}};
    for (auto &z : sizes) {
        const int tiles = z[0], rows = z[1], nkb = z[2];
        std::vector<float> nrm((size_t)tiles * nkb * kRes * rows);
        for (float &v : nrm) v = (float)(gen() % 1000);
        // large blocks on both sides of multiples of 5 and 6
        for (int t = 0; t < tiles; ++t)
            for (int kb = 0; kb < nkb; ++kb)
                if (kb % 5 == 4 || kb % 5 == 0 || kb % 6 == 5)
                    for (int d = 0; d < kRes; ++d)
                        nrm[(((size_t)t * nkb + kb) * kRes + d) * rows + (kb + d) % rows] = 1048576.f;
        std::vector<float> ref(kFlushes * kRes, 0.f), got(ref.size());
        for (int L = kFlushMin; L <= kFlushMax; ++L)
            for (int t = 0; t < tiles; ++t)
                for (int r = 0; r < rows; ++r)
                    for (int d = 0; d < kRes; ++d)
                        for (int s = 0; s < nkb; ++s) {
                            float v = 0;
                            for (int k = s; k < std::min(nkb, s + L); ++k)
                                v += nrm[(((size_t)t * nkb + k) * kRes + d) * rows + r];
                            float &m = ref[(L - kFlushMin) * kRes + d];
                            m = std::max(m, v);
                        }
        float *a, *b;
        cudaMalloc(&a, nrm.size() * 4);
        cudaMalloc(&b, got.size() * 4);
        cudaMemcpy(a, nrm.data(), nrm.size() * 4, cudaMemcpyHostToDevice);
        cudaMemset(b, 0, got.size() * 4);
        if (dg_windows(a, tiles, rows, nkb, b, 0) != cudaSuccess) return 2;
        if (cudaMemcpy(got.data(), b, got.size() * 4, cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
        cudaFree(a);
        cudaFree(b);
        if (got != ref) {
            printf("%d tiles of %d rows, %d blocks\n", tiles, rows, nkb);
            return 1;
        }
    }
    return 0;
}
"""


def test_windows(tmp_path):
    src, exe = tmp_path / "windows.cu", tmp_path / "windows"
    src.write_text(PROGRAM)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC,
                    "-I", os.path.join(os.path.dirname(build.HERE), "include"), str(src), "-o", str(exe)],
                   check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout
