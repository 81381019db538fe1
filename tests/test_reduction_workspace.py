"""The reductions of the row passes stay inside an instance's partials.

A reducing store writes its values once per CTA, so the launch with the most
CTAs (one row per CTA on the largest grid) sets the size of the workspace.
The row counts and the stride come from the kernels' own headers, compiled as
a host program: every transform length, precision and launch variant.
"""

import os
import subprocess

import pytest

from aspher_b200 import build as B

PROGRAM = r"""
#include <cstdio>
#include "pk_device.cuh"
#include "fft_launch.cuh"
using namespace asb;
template <typename T, typename F>
int check(int values, const char* what) {
    int bad = 0;
    const int lengths[] = {8, 16, 32, 64, 128, 256, 512, 768, 1024, 1536, 2048, 3072, 4096, 8192,
                           16384};
    for (int LR : lengths)
        for (int v = 0; v < kVariants; ++v)
            for (int pad = 0; pad < 2; ++pad) {
                const long rows = pad ? LR : 2 * LR;  // free space: Ns = LR, periodic: 2 LR
                if (rows > kMaxNs || row_smem_v<T>(LR, v) > kSmemPerSM) continue;
                const int rb = row_rb_v<T>(LR, v);
                const long need = (rows + rb - 1) / rb * values;
                if (need > kPartStride) {
                    std::printf("%s: %ld rows (LR %d, variant %d) need %ld of %ld doubles\n",
                                what, rows, LR, v, need, (long)kPartStride);
                    ++bad;
                }
            }
    return bad;
}
template <class S> constexpr int values() { return sizeof(S::acc) / sizeof(double); }
int main() {
    int bad = 0;
    bad += check<float, float>(values<StoreEval<float, float>>(), "evaluate() FP32");
    bad += check<float, double>(values<StoreEval<double, float>>(), "evaluate() defect-corrected");
    bad += check<double, double>(values<StoreEval<double, double>>(), "evaluate() FP64");
    bad += check<float, float>(values<StoreLineSums<float, float>>(), "line sums FP32");
    bad += check<float, double>(values<StoreLineSums<double, float>>(), "line sums defect-corrected");
    bad += check<double, double>(values<StoreLineSums<double, double>>(), "line sums FP64");
    // the widest vector pass: six values per CTA
    if (kMaxBlocks * 6 > (long)kPartStride) { std::printf("vector passes\n"); ++bad; }
    std::printf("checked %d\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(not os.path.exists(B.NVCC), reason="needs nvcc")
def test_row_reductions_fit_the_partials(tmp_path):
    src, exe = tmp_path / "fit.cu", tmp_path / "fit"
    src.write_text(PROGRAM)
    p = subprocess.run([B.NVCC, "-std=c++17", "--expt-relaxed-constexpr", *B.ARCH, "-I", B.CSRC,
                        "-o", str(exe), str(src)], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and "checked 0" in r.stdout, r.stdout
