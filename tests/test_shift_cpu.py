"""The translation of cell expansions (csrc/ddx_shift.cuh) on the host under the compiler's bounds checks: the
coefficient rows and the sums are of exactly the size that the kernel gives them, so a row or a sum past their
end ends the program, and every sum is the same chain of fused multiply-adds as here."""
import subprocess
from pathlib import Path

import pytest

from diskdyn_gb300 import build

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "ddx_shift.cuh"
constexpr int kNodes = NODES, kReal = 130, kEntries = 300;
int main() {
    // a block of its own for each, so that the next byte is out of bounds
    auto* par = (float (*)[kNodes])aligned_alloc(16, sizeof(float) * kReal * kNodes);
    auto* val = (float*)malloc(sizeof(float) * kEntries);
    auto* idx = (unsigned char*)malloc(kEntries);
    unsigned r = 12345u;
    auto next = [&]() { r = r * 1664525u + 1013904223u; return r >> 8; };
    for (int i = 0; i < kReal; ++i)
        for (int j = 0; j < kNodes; ++j) par[i][j] = (float)next() / 8388608.f - 1.f;
    for (int e = 0; e < kEntries; ++e) {
        val[e] = (float)next() / 8388608.f - 1.f;
        idx[e] = (unsigned char)(e % 7 == 0 ? kReal - 1 : next() % kReal);      // the last row often
    }
    int bad = 0;
    for (int e0 = 0; e0 < 5; ++e0)
        for (int e1 = kEntries - 5; e1 <= kEntries; ++e1) {
            float acc[kNodes] = {};
            ddx::shift_sums(par, val, idx, e0, e1, acc);
            for (int j = 0; j < kNodes; ++j) {
                float want = 0.f;
                for (int e = e0; e < e1; ++e) want = fmaf(val[e], par[idx[e]][j], want);
                bad += acc[j] != want;
            }
        }
    std::printf("%d wrong sums\n", bad);
    free(par); free(val); free(idx);
    return bad != 0;
}
"""


@pytest.mark.parametrize("nodes", [4, 8])
def test_translation_stays_within_its_rows_and_sums(tmp_path, nodes):
    src, exe = tmp_path / "shift.cpp", tmp_path / "shift"
    src.write_text(MAIN)
    cuda = Path(build.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-Wno-unknown-pragmas", "-fsanitize=address,undefined",
                    "-fno-sanitize-recover=all", f"-DNODES={nodes}", "-I", str(build.CSRC), "-I", str(cuda),
                    str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
