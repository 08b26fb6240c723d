// One coefficient of the translation of expansions (cells_shift_kernel), for N nodes at once.  Plain
// code, so that a host program can run it under a bounds checker.
#pragma once
#include <math.h>
#include <vector_types.h>

namespace ddx {

// acc[j] += sum of val[e] par[idx[e]][j] over the entries e0 <= e < e1.  A row of par, one
// coefficient of the N nodes' parents, is read in 16-byte parts.
template <int N>
__host__ __device__ __forceinline__ void shift_sums(const float (*par)[N], const float* val, const unsigned char* idx,
                                                    int e0, int e1, float (&acc)[N]) {
    static_assert(N % 4 == 0, "a row of par is read four floats at a time");
#pragma unroll 4
    for (int e = e0; e < e1; ++e) {
        const float c = val[e];
        const float4* const p = reinterpret_cast<const float4*>(par[idx[e]]);
#pragma unroll
        for (int q = 0; q < N / 4; ++q) {
            const float4 f = p[q];
            acc[4 * q] = fmaf(c, f.x, acc[4 * q]);
            acc[4 * q + 1] = fmaf(c, f.y, acc[4 * q + 1]);
            acc[4 * q + 2] = fmaf(c, f.z, acc[4 * q + 2]);
            acc[4 * q + 3] = fmaf(c, f.w, acc[4 * q + 3]);
        }
    }
}

}  // namespace ddx
