// column_sum.cuh -- one output of the product, entry by entry, for the kernels that multiply W's bit tiles as a dense matrix of
// 0 / +-2.
//
// Those kernels turn 0 * Inf into NaN in columns that do not use the row, an Inf cut into three bf16 values into NaN everywhere, and
// finite activations of 2^127 and above into Inf.  Every one of these shows in the sum: it is not finite.  The kernels look
// at each sum once as they store it, and where it is not finite they take this one instead: W as +-1, only the rows that the column
// uses, like the kernels on index lists.  A finite sum is never affected, and finite activations pay one comparison per result.
#pragma once
#include "bittile_format.h"
#include "kernels.cuh"

namespace tllm {

__device__ __forceinline__ bool finite_sum(float v) { return fabsf(v) <= 3.402823466e38f; }

// sum of x(k) * W[k][n]; dense: entries that are zero take part as 0 * x(k).  One lane's work; fp64, so that the order does not matter.
template <typename F>
__device__ __forceinline__ float column_sum(const uint32_t* bits, int n, int K, int KB, bool dense, F x) {
    double s = 0.0;
    for (int k0 = 0; k0 < K && s == s; k0 += 16) {
        const uint32_t w = __ldcg(bits + mm_word_index(n, k0 >> 6, (k0 >> 4) & 3, KB));
        if (w == 0u && !dense) continue;
        for (int j = 0; j < 16 && k0 + j < K; ++j) {
            const uint32_t c = (w >> mm_code_bit(j)) & 3u;
            if (c == 0u && !dense) continue;
            const float v = x(k0 + j);
            s += (double)(c == 0u ? v * 0.f : c == 1u ? v : -v);
        }
    }
    return (float)s;
}

}  // namespace tllm
