// attn_kernel.cuh -- attention straight from the fused q | k | v product: prompts (causal; 16-bit and fp32) and a 16-bit decode
// step over a cache.  Stock code in the reference (ternaryLLM_GPU/TernaryLLM/TernaryAttn.py:96-112), where it is several launches:
// transpositions, copies of the repeated heads and of the new key and value, and in fp32 with grouped heads two batched products, a
// mask and a softmax as well.  Here it is one, reading and writing the projections' own layouts.
//
// Scores and probabilities x values are mma.sync m16n8k16 with fp32 sums; a warp owns sixteen queries and keeps their scores,
// probabilities and results in registers (the accumulators of the first product are, rounded, the A operand of the second).  Softmax
// runs along with the tiles of keys, in fp32 and in powers of two.  Keys and values come by cp.async into rows whose 16-byte
// chunks are xor-ed with the row number, which makes every ldmatrix free of bank conflicts.
//
// The kernels differ in who shares a tile of keys: in a prompt four warps hold 64 queries and go through the same tiles, and a second group of four takes
// every other tile: the prompts served here fill an SM with one block, and one warp per scheduler spends two thirds
// of its time waiting.  In a decode step there is one query a head, the query heads of one key head are the rows of the one operand, and
// every warp goes through keys of its own.
#pragma once
#include <type_traits>

#include "kernels.cuh"

namespace tllm {

#define AM_THREADS 128
#define AM_KEYS 64                    // keys per tile of the 16-bit prompt kernel, and queries per block
#define AM_SHARES 2                   // groups of four warps that share the tiles of a block of queries
#define AM_P_THREADS (AM_THREADS * AM_SHARES)
#define AM_RING 3                     // tiles per warp on the way in the decode kernel
#define AM_MAX_GROUP 16               // query heads per key head of the decode kernel: the rows of one operand

__device__ __forceinline__ void am_cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void am_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void am_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void am_ldm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void am_ldm_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <typename T>
__device__ __forceinline__ void am_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if constexpr (std::is_same<T, __half>::value)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <typename T>
__device__ __forceinline__ uint32_t am_pack(float lo, float hi) {
    if constexpr (std::is_same<T, __half>::value) {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *(const uint32_t*)&h;
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *(const uint32_t*)&h;
    }
}
// What the exponents are taken from: the maximum, or 0 as long as every score was -Inf (and their weights 0, not Inf - Inf)
__device__ __forceinline__ float am_base(float m) { return m == -INFINITY ? 0.f : m; }
// 16-byte chunk c of row r of a tile whose rows hold HD values
template <int HD>
__device__ __forceinline__ uint32_t am_chunk(int r, int c) { return (uint32_t)(r * (HD * 2) + ((c ^ (r & 7)) << 4)); }

// sixteen queries of a warp and what they have seen so far; a lane holds rows lane / 4 and lane / 4 + 8
template <typename T, int HD>
struct AmQueries {
    uint32_t q[HD / 16][4];
    float o[HD / 8][4];
    float mx[2], sum[2];                                   // running maximum (in units of log2) and this lane's share of the sum

    // row pointers of the lane's two rows (null: zeros)
    __device__ __forceinline__ void load(const T* r0, const T* r1, int lane) {
        const int t = lane & 3;
#pragma unroll
        for (int s = 0; s < HD / 16; ++s) {
            q[s][0] = r0 ? *(const uint32_t*)(r0 + 16 * s + 2 * t) : 0u;
            q[s][1] = r1 ? *(const uint32_t*)(r1 + 16 * s + 2 * t) : 0u;
            q[s][2] = r0 ? *(const uint32_t*)(r0 + 16 * s + 2 * t + 8) : 0u;
            q[s][3] = r1 ? *(const uint32_t*)(r1 + 16 * s + 2 * t + 8) : 0u;
        }
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
        mx[0] = mx[1] = -INFINITY, sum[0] = sum[1] = 0.f;
    }
    // a tile of KT keys at shared addresses ks, vs; the lane's two rows see the keys up to last0 and last1 of the tile.  scale: of the
    // scores, times log2(e).  The first tile that a row goes through has a key that it sees.
    template <int KT>
    __device__ __forceinline__ void tile(uint32_t ks, uint32_t vs, int last0, int last1, float scale, int lane) {
        const int t = lane & 3;
        float s[KT / 8][4];
#pragma unroll
        for (int j = 0; j < KT / 8; ++j) {
            s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
        }
        // JB sums side by side: one after the other, each MMA would wait for the one before
        constexpr int JB = KT / 8 < 4 ? KT / 8 : 4;
#pragma unroll
        for (int j0 = 0; j0 < KT / 8; j0 += JB)
#pragma unroll
            for (int c = 0; c < HD / 32; ++c) {
                uint32_t b[JB][4];
#pragma unroll
                for (int j = 0; j < JB; ++j) am_ldm(b[j], ks + am_chunk<HD>(8 * (j0 + j) + (lane & 7), 4 * c + (lane >> 3)));
#pragma unroll
                for (int j = 0; j < JB; ++j) am_mma<T>(s[j0 + j], q[2 * c], b[j][0], b[j][1]);
#pragma unroll
                for (int j = 0; j < JB; ++j) am_mma<T>(s[j0 + j], q[2 * c + 1], b[j][2], b[j][3]);
            }
        float m0 = mx[0], m1 = mx[1];
#pragma unroll
        for (int j = 0; j < KT / 8; ++j) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int key = 8 * j + 2 * t + i;
                s[j][i] = key <= last0 ? s[j][i] * scale : -INFINITY;
                s[j][2 + i] = key <= last1 ? s[j][2 + i] * scale : -INFINITY;
                m0 = fmaxf(m0, s[j][i]), m1 = fmaxf(m1, s[j][2 + i]);
            }
        }
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) {
            m0 = fmaxf(m0, __shfl_xor_sync(0xffffffffu, m0, x));
            m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, x));
        }
        const float b0 = am_base(m0), b1 = am_base(m1), f0 = exp2f(mx[0] - b0), f1 = exp2f(mx[1] - b1);
        mx[0] = m0, mx[1] = m1;
        sum[0] *= f0, sum[1] *= f1;
#pragma unroll
        for (int j = 0; j < HD / 8; ++j) o[j][0] *= f0, o[j][1] *= f0, o[j][2] *= f1, o[j][3] *= f1;
#pragma unroll
        for (int j = 0; j < KT / 8; ++j) {
            s[j][0] = exp2f(s[j][0] - b0), s[j][1] = exp2f(s[j][1] - b0), s[j][2] = exp2f(s[j][2] - b1), s[j][3] = exp2f(s[j][3] - b1);
            sum[0] += s[j][0] + s[j][1], sum[1] += s[j][2] + s[j][3];
        }
#pragma unroll
        for (int k = 0; k < KT / 16; ++k) {
            const uint32_t a[4] = {am_pack<T>(s[2 * k][0], s[2 * k][1]), am_pack<T>(s[2 * k][2], s[2 * k][3]), am_pack<T>(s[2 * k + 1][0], s[2 * k + 1][1]),
                                   am_pack<T>(s[2 * k + 1][2], s[2 * k + 1][3])};
#pragma unroll
            for (int c = 0; c < HD / 16; ++c) {
                uint32_t b[4];
                am_ldm_t(b, vs + am_chunk<HD>(16 * k + (lane & 15), 2 * c + (lane >> 4)));
                am_mma<T>(o[2 * c], a, b[0], b[1]);
                am_mma<T>(o[2 * c + 1], a, b[2], b[3]);
            }
        }
    }
    __device__ __forceinline__ void finish() {              // the four lanes of a row add up their shares
#pragma unroll
        for (int x = 1; x < 4; x <<= 1) {
            sum[0] += __shfl_xor_sync(0xffffffffu, sum[0], x);
            sum[1] += __shfl_xor_sync(0xffffffffu, sum[1], x);
        }
    }
};

// one group's barrier
__device__ __forceinline__ void am_group_sync(int group) { asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory"); }
// The second group's results join the first's.  buf: [4 warps][N * 4 + 4][32 lanes]; called by the whole block.
template <int N>
__device__ __forceinline__ void am_join(float (&o)[N][4], float (&mx)[2], float (&sum)[2], float* buf, int warp, int lane) {
    __syncthreads();
    float* at = buf + (warp & 3) * (N * 4 + 4) * 32 + lane;
    if (warp >= 4) {
#pragma unroll
        for (int j = 0; j < N * 4; ++j) at[32 * j] = o[j >> 2][j & 3];
        at[32 * N * 4] = mx[0], at[32 * (N * 4 + 1)] = mx[1], at[32 * (N * 4 + 2)] = sum[0], at[32 * (N * 4 + 3)] = sum[1];
    }
    __syncthreads();
    if (warp < 4) {
        float f[2], g[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float m1 = at[32 * (N * 4 + r)], m = am_base(fmaxf(mx[r], m1));
            f[r] = exp2f(mx[r] - m), g[r] = exp2f(m1 - m);
            sum[r] = sum[r] * f[r] + at[32 * (N * 4 + 2 + r)] * g[r];
        }
#pragma unroll
        for (int j = 0; j < N * 4; ++j) o[j >> 2][j & 3] = o[j >> 2][j & 3] * f[(j >> 1) & 1] + at[32 * j] * g[(j >> 1) & 1];
    }
}

// ---- a prompt: out[b, m, h] from the fused product qkv [batch * M][ld] (query heads, key heads, value heads), queries see the keys up
// to their own position.  grid (query tiles, H, batch), longest first; two tiles of keys per group in shared memory.
template <int HD>
constexpr size_t am_prompt_smem() { return (size_t)AM_SHARES * 2 * 2 * AM_KEYS * HD * 2; }

template <typename T, int HD>
__global__ void __launch_bounds__(AM_P_THREADS) prompt_attention_kernel(const T* __restrict__ qkv, T* __restrict__ out, int M, int H, int HKV, int ld, float scale) {
    extern __shared__ __align__(128) unsigned char am_smem[];
    constexpr uint32_t TILE = AM_KEYS * HD * 2;
    const int tid = threadIdx.x & (AM_THREADS - 1), lane = tid & 31, warp = threadIdx.x >> 5, group = warp >> 2;
    const int qt = gridDim.x - 1 - blockIdx.x, h = blockIdx.y, hk = h / (H / HKV);
    const T* base = qkv + (size_t)blockIdx.z * M * ld;
    const T *k = base + (size_t)(H + hk) * HD, *v = k + (size_t)HKV * HD;
    const uint32_t s0 = smem_u32(am_smem) + (uint32_t)group * 4 * TILE;
    pdl_launch_dependents();
    pdl_wait();
    auto fetch = [&](int t) {                               // rows past the end repeat the last one; no query looks at them
        const uint32_t dst = s0 + (uint32_t)(t >> 1 & 1) * 2 * TILE;
#pragma unroll
        for (int i = 0; i < AM_KEYS * HD / 8 / AM_THREADS; ++i) {
            const int e = tid + i * AM_THREADS, r = e / (HD / 8), c = e % (HD / 8);
            const size_t at = (size_t)min(t * AM_KEYS + r, M - 1) * ld + c * 8;
            am_cp16(dst + am_chunk<HD>(r, c), k + at);
            am_cp16(dst + TILE + am_chunk<HD>(r, c), v + at);
        }
        am_commit();
    };
    if (group <= qt) fetch(group);
    const int r0 = qt * AM_KEYS + (warp & 3) * 16 + (lane >> 2), r1 = r0 + 8;
    AmQueries<T, HD> w;
    w.load(base + (size_t)min(r0, M - 1) * ld + (size_t)h * HD, base + (size_t)min(r1, M - 1) * ld + (size_t)h * HD, lane);
#pragma unroll 1
    for (int t = group; t <= qt; t += AM_SHARES) {
        if (t + AM_SHARES <= qt) {
            fetch(t + AM_SHARES);
            am_wait<1>();
        } else am_wait<0>();
        am_group_sync(group);
        const uint32_t ks = s0 + (uint32_t)(t >> 1 & 1) * 2 * TILE;
        w.template tile<AM_KEYS>(ks, ks + TILE, r0 - t * AM_KEYS, r1 - t * AM_KEYS, scale, lane);
        am_group_sync(group);                               // the tile has been read before the next but one overwrites it
    }
    am_join(w.o, w.mx, w.sum, (float*)am_smem, warp, lane);
    if (group) return;
    w.finish();
    const float i0 = 1.f / w.sum[0], i1 = 1.f / w.sum[1];
    T* y = out + ((size_t)blockIdx.z * M) * ((size_t)H * HD) + (size_t)h * HD + 2 * (lane & 3);
#pragma unroll
    for (int j = 0; j < HD / 8; ++j) {
        if (r0 < M) *(uint32_t*)(y + (size_t)r0 * H * HD + 8 * j) = am_pack<T>(w.o[j][0] * i0, w.o[j][1] * i0);
        if (r1 < M) *(uint32_t*)(y + (size_t)r1 * H * HD + 8 * j) = am_pack<T>(w.o[j][2] * i1, w.o[j][3] * i1);
    }
}

// ---- an fp32 prompt: every value as the three bf16 numbers that add up to it (rounded to nearest: what is left after the third is below
// 2^-27 of it), every product as the six of theirs that count, the products of a kind summed in accumulators of their own
// because the tensor core cuts small terms off beside large ones.  Six MMAs take 48 clocks where 64 of FMA would be needed, and
// read shared memory a fifth as often: the CUDA-core version of this kernel was bound by those reads.
// Measured, 256 positions of 32 / 8 heads of 64: 37 -> 15 us (23 with one group of warps).
#define AM_F32_KEYS 32
__device__ __forceinline__ void am_split(float a, float b, uint32_t (&w)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        w[i] = am_pack<__nv_bfloat16>(a, b);
        a -= __uint_as_float(w[i] << 16), b -= __uint_as_float(w[i] & 0xFFFF0000u);
    }
}
// d[kind] += a * b for one pair of operand tiles
__device__ __forceinline__ void am_mma6(float (&d)[3][4], const uint32_t (&a0)[4], const uint32_t (&a1)[4], const uint32_t (&a2)[4], const uint32_t* b0, const uint32_t* b1,
                                        const uint32_t* b2) {
    using B = __nv_bfloat16;
    am_mma<B>(d[2], a0, b2[0], b2[1]);
    am_mma<B>(d[1], a0, b1[0], b1[1]);
    am_mma<B>(d[0], a0, b0[0], b0[1]);
    am_mma<B>(d[2], a1, b1[0], b1[1]);
    am_mma<B>(d[1], a1, b0[0], b0[1]);
    am_mma<B>(d[2], a2, b0[0], b0[1]);
}
// two tiles of keys and values as they are, one as pieces
template <int HD>
constexpr size_t am_f32_smem() { return (size_t)AM_SHARES * AM_F32_KEYS * HD * (2 * 2 * 4 + 2 * 3 * 2); }

template <int HD>
__global__ void __launch_bounds__(AM_P_THREADS) prompt_attention_f32_kernel(const float* __restrict__ qkv, float* __restrict__ out, int M, int H, int HKV, int ld, float scale) {
    extern __shared__ __align__(128) unsigned char am_smem[];
    constexpr int KT = AM_F32_KEYS, NC = KT * HD / 8 / AM_THREADS;          // chunks of eight values per thread
    constexpr uint32_t RAW = KT * HD * 4, PL = KT * HD * 2;
    const int tid = threadIdx.x & (AM_THREADS - 1), lane = tid & 31, warp = threadIdx.x >> 5, group = warp >> 2, t4 = lane & 3;
    const int qt = gridDim.x - 1 - blockIdx.x, q0 = qt * AM_KEYS, h = blockIdx.y, hk = h / (H / HKV);
    const float* base = qkv + (size_t)blockIdx.z * M * ld;
    const float *k = base + (size_t)(H + hk) * HD, *v = k + (size_t)HKV * HD;
    unsigned char* mem = am_smem + group * (4 * RAW + 6 * PL);
    const uint32_t s0 = smem_u32(mem), ps = s0 + 4 * RAW;
    pdl_launch_dependents();
    pdl_wait();
    // a thread turns the chunks that it has fetched itself
    auto fetch = [&](int t) {
        const uint32_t dst = s0 + (uint32_t)(t >> 1 & 1) * 2 * RAW;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int e = tid + i * AM_THREADS;
            const size_t at = (size_t)min(t * KT + e / (HD / 8), M - 1) * ld + e % (HD / 8) * 8;
            am_cp16(dst + e * 32, k + at), am_cp16(dst + e * 32 + 16, k + at + 4);
            am_cp16(dst + RAW + e * 32, v + at), am_cp16(dst + RAW + e * 32 + 16, v + at + 4);
        }
        am_commit();
    };
    const int n = min(q0 + AM_KEYS - 1, M - 1) / KT + 1;
    if (group < n) fetch(group);
    const int r0 = q0 + (warp & 3) * 16 + (lane >> 2), r1 = r0 + 8;
    uint32_t q[3][HD / 16][4];
    {
        const float *a = base + (size_t)min(r0, M - 1) * ld + (size_t)h * HD + 2 * t4, *b = base + (size_t)min(r1, M - 1) * ld + (size_t)h * HD + 2 * t4;
#pragma unroll
        for (int s = 0; s < HD / 16; ++s)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 x = *(const float2*)((i & 1 ? b : a) + 16 * s + 8 * (i >> 1));
                uint32_t w[3];
                am_split(x.x, x.y, w);
                q[0][s][i] = w[0], q[1][s][i] = w[1], q[2][s][i] = w[2];
            }
    }
    float o[HD / 8][4], mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};          // mx: in units of log2
#pragma unroll
    for (int j = 0; j < HD / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
#pragma unroll 1
    for (int t = group; t < n; t += AM_SHARES) {
        if (t + AM_SHARES < n) {
            fetch(t + AM_SHARES);
            am_wait<1>();
        } else am_wait<0>();
        const unsigned char* raw = mem + (t >> 1 & 1) * 2 * RAW;
#pragma unroll
        for (int i = 0; i < 2 * NC; ++i) {
            const int e = tid + (i >> 1) * AM_THREADS;
            const float4 lo = *(const float4*)(raw + (i & 1) * RAW + e * 32), hi = *(const float4*)(raw + (i & 1) * RAW + e * 32 + 16);
            uint32_t w[4][3];
            am_split(lo.x, lo.y, w[0]), am_split(lo.z, lo.w, w[1]), am_split(hi.x, hi.y, w[2]), am_split(hi.z, hi.w, w[3]);
#pragma unroll
            for (int pl = 0; pl < 3; ++pl)
                *(uint4*)(mem + 4 * RAW + (3 * (i & 1) + pl) * PL + am_chunk<HD>(e / (HD / 8), e % (HD / 8))) = make_uint4(w[0][pl], w[1][pl], w[2][pl], w[3][pl]);
        }
        am_group_sync(group);
        if (t * KT <= q0 + (warp & 3) * 16 + 15) {                   // else no query of this warp sees any of the tile
            float s[KT / 8][4];
#pragma unroll
            for (int j = 0; j < KT / 8; j += 2) {              // two sums of each kind side by side
                float acc[2][3][4] = {};
#pragma unroll
                for (int c = 0; c < HD / 32; ++c) {
                    uint32_t b[2][3][4];
#pragma unroll
                    for (int x = 0; x < 2; ++x)
#pragma unroll
                        for (int pl = 0; pl < 3; ++pl) am_ldm(b[x][pl], ps + pl * PL + am_chunk<HD>(8 * (j + x) + (lane & 7), 4 * c + (lane >> 3)));
#pragma unroll
                    for (int y = 0; y < 2; ++y)
#pragma unroll
                        for (int x = 0; x < 2; ++x) am_mma6(acc[x], q[0][2 * c + y], q[1][2 * c + y], q[2][2 * c + y], b[x][0] + 2 * y, b[x][1] + 2 * y, b[x][2] + 2 * y);
                }
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool seen = t * KT + 8 * (j + x) + 2 * t4 + (i & 1) <= (i < 2 ? r0 : r1);
                        s[j + x][i] = seen ? acc[x][0][i] + (acc[x][1][i] + acc[x][2][i]) : -INFINITY;
                    }
            }
            float f[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float m = -INFINITY;
#pragma unroll
                for (int j = 0; j < KT / 8; ++j) m = fmaxf(m, fmaxf(s[j][2 * r], s[j][2 * r + 1]));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
                m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
                m = fmaxf(mx[r], m * scale);
                const float base = am_base(m);
                f[r] = exp2f(mx[r] - base);
                mx[r] = m;
                sum[r] *= f[r];
#pragma unroll
                for (int j = 0; j < KT / 8; ++j)
#pragma unroll
                    for (int i = 2 * r; i < 2 * r + 2; ++i) sum[r] += s[j][i] = exp2f(fmaf(s[j][i], scale, -base));
            }
            uint32_t p[3][KT / 16][4];
#pragma unroll
            for (int kk = 0; kk < KT / 16; ++kk)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t w[3];
                    am_split(s[2 * kk + (i >> 1)][2 * (i & 1)], s[2 * kk + (i >> 1)][2 * (i & 1) + 1], w);
                    p[0][kk][i] = w[0], p[1][kk][i] = w[1], p[2][kk][i] = w[2];
                }
#pragma unroll
            for (int c = 0; c < HD / 16; ++c) {
                float acc[2][3][4] = {};
#pragma unroll
                for (int kk = 0; kk < KT / 16; ++kk) {
                    uint32_t b[3][4];
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl) am_ldm_t(b[pl], ps + (3 + pl) * PL + am_chunk<HD>(16 * kk + (lane & 15), 2 * c + (lane >> 4)));
#pragma unroll
                    for (int x = 0; x < 2; ++x) am_mma6(acc[x], p[0][kk], p[1][kk], p[2][kk], b[0] + 2 * x, b[1] + 2 * x, b[2] + 2 * x);
                }
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int i = 0; i < 4; ++i) o[2 * c + x][i] = fmaf(o[2 * c + x][i], f[i >> 1], acc[x][0][i] + (acc[x][1][i] + acc[x][2][i]));
            }
        }
        am_group_sync(group);
    }
    am_join(o, mx, sum, (float*)am_smem, warp, lane);
    if (group) return;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
        sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
        const float inv = 1.f / sum[r];
        const int row = r ? r1 : r0;
        float* y = out + ((size_t)blockIdx.z * M + row) * ((size_t)H * HD) + (size_t)h * HD + 2 * t4;
        if (row < M)
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) *(float2*)(y + 8 * j) = make_float2(o[j][2 * r] * inv, o[j][2 * r + 1] * inv);
    }
}

// ---- a decode step: one new token a sequence.  Its key and value go from the fused product into position `len` of the caches
// ([sequence][key head][position][HD]), and its query heads attend to positions 0 .. len.  grid (parts, key heads, sequences), a cluster
// of `parts` blocks for the keys of one head of one sequence; each warp goes through tiles of 8 KB of keys and values, two of
// them on the way.  Bound by reading the caches: 5.2 TB/s at 60 sequences of 8 heads (126 MB).  The warps' results are put together in shared memory, the blocks' through the cluster's.
template <int HD>
constexpr size_t am_decode_smem() { return (size_t)(AM_THREADS / 32) * AM_RING * 8192; }

__device__ __forceinline__ float am_peer_f32(uint32_t addr, uint32_t rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void am_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float am_weight(float m, float top) { return m == -INFINITY ? 0.f : exp2f(m - top); }

template <typename T, int HD>
__global__ void __launch_bounds__(AM_THREADS) decode_attention_kernel(const T* __restrict__ qkv, T* __restrict__ kc, T* __restrict__ vc, T* __restrict__ out, int H,
                                                                      int HKV, int len, long long seq_step, long long head_step, float scale) {
    extern __shared__ __align__(128) unsigned char am_smem[];
    constexpr int KT = 2048 / HD, WARPS = AM_THREADS / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int parts = gridDim.x, part = blockIdx.x, hk = blockIdx.y, G = H / HKV;
    const T* row = qkv + (size_t)blockIdx.z * (size_t)(H + 2 * HKV) * HD;
    const T *knew = row + (size_t)(H + hk) * HD, *vnew = knew + (size_t)HKV * HD;
    const size_t at0 = (size_t)blockIdx.z * seq_step + (size_t)hk * head_step;
    const T *k = kc + at0, *v = vc + at0;
    const int tiles = (len + KT) / KT, per = (tiles + parts - 1) / parts, t1 = min(tiles, (part + 1) * per);     // len + 1 keys
    const uint32_t ring = smem_u32(am_smem) + (uint32_t)warp * (AM_RING * 8192);
    pdl_launch_dependents();
    pdl_wait();
    auto fetch = [&](int t, int slot) {                     // keys past the new one repeat it; no query looks at them
        if (t < t1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int e = lane + i * 32, r = e / (HD / 8), c = e % (HD / 8), key = t * KT + r;
                const bool old = key < len;
                const uint32_t dst = ring + (uint32_t)slot * 8192u + am_chunk<HD>(r, c);
                am_cp16(dst, (old ? k + (size_t)key * HD : knew) + c * 8);
                am_cp16(dst + 4096u, (old ? v + (size_t)key * HD : vnew) + c * 8);
            }
        }
        am_commit();
    };
    int t = part * per + warp;
#pragma unroll
    for (int i = 0; i < AM_RING - 1; ++i) fetch(t + i * WARPS, i);
    // the part that holds position len appends to the caches (nobody reads it there in this launch)
    if (len / KT >= part * per && len / KT < t1 && tid < HD / 4) {
        const int c = tid % (HD / 8);
        *(uint4*)((tid < HD / 8 ? kc : vc) + at0 + (size_t)len * HD + c * 8) = *(const uint4*)((tid < HD / 8 ? knew : vnew) + c * 8);
    }
    const int g0 = lane >> 2, g1 = g0 + 8;
    const T* q = row + (size_t)hk * G * HD;
    AmQueries<T, HD> w;
    w.load(g0 < G ? q + (size_t)g0 * HD : nullptr, g1 < G ? q + (size_t)g1 * HD : nullptr, lane);
    int slot = 0;
#pragma unroll 1
    for (; t < t1; t += WARPS) {
        fetch(t + (AM_RING - 1) * WARPS, slot ? slot - 1 : AM_RING - 1);
        am_wait<AM_RING - 1>();
        __syncwarp();
        const uint32_t ks = ring + (uint32_t)slot * 8192u;
        w.template tile<KT>(ks, ks + 4096u, len - t * KT, len - t * KT, scale, lane);
        __syncwarp();
        slot = slot + 1 == AM_RING ? 0 : slot + 1;
    }
    am_wait<0>();
    w.finish();
    __syncthreads();
    // [warp][row][HD] results, [warp][row] maxima and sums, then the block's
    float* po = (float*)am_smem;
    float *pm = po + WARPS * G * HD, *pl = pm + WARPS * G, *bo = pl + WARPS * G, *bm = bo + G * HD, *bl = bm + G;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int g = g0 + 8 * r;
        if (g < G) {
            float* y = po + ((size_t)warp * G + g) * HD + 2 * (lane & 3);
#pragma unroll
            for (int j = 0; j < HD / 8; ++j) *(float2*)(y + 8 * j) = make_float2(w.o[j][2 * r], w.o[j][2 * r + 1]);
            if ((lane & 3) == 0) pm[warp * G + g] = w.mx[r], pl[warp * G + g] = w.sum[r];
        }
    }
    __syncthreads();
    for (int e = tid; e < G * HD; e += AM_THREADS) {
        const int g = e / HD;
        float top = -INFINITY, o = 0.f, l = 0.f;
#pragma unroll
        for (int i = 0; i < WARPS; ++i) top = fmaxf(top, pm[i * G + g]);
#pragma unroll
        for (int i = 0; i < WARPS; ++i) {
            const float f = am_weight(pm[i * G + g], top);
            o += f * po[(size_t)i * G * HD + e], l += f * pl[i * G + g];
        }
        bo[e] = o;
        if (e % HD == 0) bm[g] = top, bl[g] = l;
    }
    am_cluster_sync();
    T* y = out + ((size_t)blockIdx.z * H + (size_t)hk * G) * HD;
    for (int e = part * AM_THREADS + tid; e < G * HD; e += parts * AM_THREADS) {
        const int g = e / HD;
        float top = -INFINITY, o = 0.f, l = 0.f;
        for (int i = 0; i < parts; ++i) top = fmaxf(top, am_peer_f32(smem_u32(bm + g), i));
        for (int i = 0; i < parts; ++i) {
            const float f = am_weight(am_peer_f32(smem_u32(bm + g), i), top);
            o += f * am_peer_f32(smem_u32(bo + e), i), l += f * am_peer_f32(smem_u32(bl + g), i);
        }
        if constexpr (std::is_same<T, __half>::value) y[e] = __float2half_rn(o / l);
        else y[e] = __float2bfloat16_rn(o / l);
    }
    am_cluster_sync();                                      // nobody leaves while its shared memory is read
}

}  // namespace tllm
