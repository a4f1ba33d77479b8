// lists_kernel.cuh -- the reference's merged tiled CSC arrays (16-bit tile-local row ids, four 32-bit words per column and
// tile) -> two-bit tiles (bittile_format.h), on the device, for the product on arrays that nobody repacked beforehand.
//
// One block per group of sixteen columns: 2048 rows of it at a time are built in shared memory, a byte per entry, which any thread may
// store to, then packed and written once as a contiguous stream.  (Two-bit codes ORed in by atomics waited for one another, since neighbours
// in a list share a word.  A call of 256 rows of fp32 on 2048 x 8192, 80 % zeros, took 57 us with them, 19 of it here; 39 with bytes, the
// activations' planes made beside this kernel and the launches chained.)  Bound by the latency of a list -- its offsets, then its ids --
// hence all lists of a part at once, as many lanes per list as there are threads for them, up to four blocks per SM.  The bytes are 2 per
// non-zero plus 16 per list in and a quarter per entry out: 6.7 + 1 + 4 MB there.
//
// Two bits cannot hold an entry that is named twice.  A pair that names one row twice is skipped (it adds nothing); everything else
// is counted, and where the count is not the number of entries in the image the block's flag is raised.
#pragma once
#include "bittile_format.h"
#include "kernels.cuh"

namespace tllm {

#define LB_THREADS 512
#define LB_SLICES 32                  // slices of 64 rows that a block builds at a time: 32 KiB (even, so that pairs stay together)

// sixteen codes, a byte each -> a word of them (mm_code_bit)
__device__ __forceinline__ uint32_t lb_pack(const uint4& v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t x = ((w[i] << 2) | (w[i] >> 16)) & 0x0F0Fu;          // rows 4i, 4i + 2 in one nibble, 4i + 1, 4i + 3 in the other
        o |= (x & 0xFu) << (12 - 4 * i) | (x & 0xF00u) << (20 - 4 * i);
    }
    return o;
}

static __global__ void __launch_bounds__(LB_THREADS) lists_to_bits_kernel(const int16_t* __restrict__ idx, const int32_t* __restrict__ off, uint32_t* __restrict__ bits,
                                                                          unsigned int* __restrict__ counters, int ncounters, int* __restrict__ flags, int N, int K,
                                                                          int T, int KB) {
    constexpr int ROWS = LB_SLICES * 64;
    __shared__ __align__(16) unsigned char image[16 * ROWS];                // [column][row]: 0, 1 (+1) or 3 (-1)
    const int tid = threadIdx.x, group = blockIdx.x;
    const int tiles = (K + T - 1) / T, cols = min(16, N - group * 16);      // may be <= 0: padding columns
    pdl_wait();                                                             // bits, counters and flags may still be read by an earlier call's kernels
    pdl_launch_dependents();                                                // behind the wait: what starts now need not wait for what came before this
    for (int i = group * LB_THREADS + tid; i < ncounters; i += gridDim.x * LB_THREADS) counters[i] = 0;
    if (group == 0 && tid == 0) flags[gridDim.x] = 0;                       // the product's status word
    uint32_t* out = bits + (size_t)group * KB * 64;
    int surplus = 0;                                                        // entries put in, minus entries found in the image
    bool odd_sign = false;                                                  // a list's factor is neither +1 nor -1
    for (int s0 = 0; s0 < KB; s0 += LB_SLICES) {
        const int ns = min(LB_SLICES, KB - s0), k0 = s0 * 64, k1 = min(K, k0 + ns * 64);
        for (int i = tid; i < ROWS; i += LB_THREADS) ((uint4*)image)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        const int t0 = k0 / T, nt = (k1 - 1) / T - t0 + 1, items = cols * nt;
        int log = 5;                                                        // lanes per list: 4 to 32
        while (log > 2 && items << log > LB_THREADS) --log;
        const int lanes = 1 << log, l = tid & (lanes - 1);
        for (int item = tid >> log; item < items; item += LB_THREADS >> log) {
            const int c = item / nt, t = t0 + item - c * nt, base = t * T - k0;
            const int4 o = __ldg((const int4*)off + (size_t)(group * 16 + c) * tiles + t);
            auto put = [&](int id, unsigned char code) {
                const int k = base + id;
                if (k < 0 || k >= k1 - k0) return;
                image[c * ROWS + k] = code;
                ++surplus;
            };
#pragma unroll 8
            for (int i = o.x + 2 * l; i + 1 < o.y; i += 2 * lanes) {
                const int a = idx[i], b = idx[i + 1];
                if (a != b) {
                    put(a, 1);
                    put(b, 3);
                }
            }
            const unsigned char code = o.w > 0 ? 1 : 3;
#pragma unroll 2
            for (int i = o.y + l; i < o.z; i += lanes) put(idx[i], code);
            odd_sign |= o.w != 1 && o.w != -1 && o.y < o.z;
        }
        __syncthreads();
        for (int i = tid; i < ns * 64; i += LB_THREADS) {                   // word i of the part (mm_word_index)
            int kb, g, t, hi;
            if ((s0 + ((i >> 7) << 1) | 1) < KB) {
                const int chunk = (i >> 2) & 31;
                g = chunk >> 2, t = (chunk & 3) ^ ((g >> 1) & 3), kb = ((i >> 7) << 1) + ((i >> 1) & 1), hi = i & 1;
            } else {                                                        // an odd last slice
                const int at = i & 63;
                g = at >> 3, t = (at >> 1) & 3, kb = i >> 6, hi = at & 1;
            }
            const uint32_t w = lb_pack(*(const uint4*)(image + (g + 8 * hi) * ROWS + kb * 64 + t * 16));
            out[(size_t)s0 * 64 + i] = w;
            surplus -= __popc(w & 0x55555555u);
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
