// lists_kernel.cuh -- the reference's merged tiled CSC arrays (16-bit tile-local row ids, four 32-bit words per column and
// tile) -> two-bit tiles (bittile_format.h), on the device, for the product on arrays that nobody repacked beforehand.
//
// One block per group of sixteen columns: its part of the image (KB * 256 bytes) is built in shared memory with atomic ORs,
// eight lanes per list, and leaves as one contiguous stream.  Bound by the latency of a list -- its offsets, then its ids --
// hence many short lists in flight: 64 per block, up to four blocks per SM.  The bytes are 2 per non-zero plus 16 per list in and
// a quarter per entry out: 6.7 + 1 + 4 MB at 2048 x 8192, 80 % zeros.
//
// Two bits cannot hold an entry that is named twice.  A pair that names one row twice is skipped (it adds nothing); everything else
// is counted, and where the count is not the number of entries in the image the block's flag is raised.
#pragma once
#include "bittile_format.h"
#include "kernels.cuh"

namespace tllm {

#define LB_THREADS 512
#define LB_SLICES 128                 // slices of 64 rows that a block builds at a time: 32 KiB (even, so that pairs stay together)

static __global__ void __launch_bounds__(LB_THREADS) lists_to_bits_kernel(const int16_t* __restrict__ idx, const int32_t* __restrict__ off, uint32_t* __restrict__ bits,
                                                                          unsigned int* __restrict__ counters, int ncounters, int* __restrict__ flags, int N, int K,
                                                                          int T, int KB) {
    __shared__ __align__(16) uint32_t image[LB_SLICES * 64];
    const int tid = threadIdx.x, sub = tid >> 3, l8 = tid & 7, group = blockIdx.x;
    const int tiles = (K + T - 1) / T, cols = min(16, N - group * 16);      // may be <= 0: padding columns
    for (int i = group * LB_THREADS + tid; i < ncounters; i += gridDim.x * LB_THREADS) counters[i] = 0;
    if (group == 0 && tid == 0) flags[gridDim.x] = 0;                       // the product's status word
    uint32_t* out = bits + (size_t)group * KB * 64;
    int surplus = 0;                                                        // entries put in, minus entries found in the image
    bool odd_sign = false;                                                  // a list's factor is neither +1 nor -1
    for (int s0 = 0; s0 < KB; s0 += LB_SLICES) {
        const int ns = min(LB_SLICES, KB - s0), k0 = s0 * 64, k1 = min(K, k0 + ns * 64);
        for (int i = tid; i < ns * 16; i += LB_THREADS) ((uint4*)image)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        const int t0 = k0 / T, nt = (k1 - 1) / T - t0 + 1;
        for (int item = sub; item < cols * nt; item += LB_THREADS / 8) {
            const int c = item / nt, t = t0 + item - c * nt, base = t * T;
            const int4 o = __ldg((const int4*)off + (size_t)(group * 16 + c) * tiles + t);
            auto put = [&](int id, uint32_t code) {
                const int k = base + id;
                if (k < k0 || k >= k1) return;
                const int word = (int)mm_word_index(c, k >> 6, (k >> 4) & 3, KB) - s0 * 64;
                atomicOr(image + word, code << mm_code_bit(k & 15));
                ++surplus;
            };
#pragma unroll 4
            for (int i = o.x + 2 * l8; i + 1 < o.y; i += 16) {
                const int a = idx[i], b = idx[i + 1];
                if (a != b) {
                    put(a, 1u);
                    put(b, 3u);
                }
            }
            const uint32_t code = o.w > 0 ? 1u : 3u;
#pragma unroll 2
            for (int i = o.y + l8; i < o.z; i += 8) put(idx[i], code);
            odd_sign |= o.w != 1 && o.w != -1 && o.y < o.z;
        }
        __syncthreads();
        for (int i = tid; i < ns * 16; i += LB_THREADS) {
            const uint4 v = ((const uint4*)image)[i];
            ((uint4*)(out + (size_t)s0 * 64))[i] = v;
            surplus -= __popc(v.x & 0x55555555u) + __popc(v.y & 0x55555555u) + __popc(v.z & 0x55555555u) + __popc(v.w & 0x55555555u);
        }
        __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) surplus += __shfl_xor_sync(0xffffffffu, surplus, o);
    __shared__ int total;
    if (tid == 0) total = 0;
    __syncthreads();
    if ((tid & 31) == 0) atomicAdd(&total, surplus);
    const int any = __syncthreads_or(odd_sign);
    if (tid == 0) flags[group] = any || total != 0;
}

}  // namespace tllm
