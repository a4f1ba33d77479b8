// attn_kernel.cuh -- causal attention of one prompt straight from the fused q | k | v product, in fp32 arithmetic.
//
// The reference's attention core is stock code (ternaryLLM_GPU/TernaryLLM/TernaryAttn.py:96-112).  In fp32, and with fewer key
// heads than query heads, the stock path is a chain of a dozen launches (two batched products, mask, softmax, copies of the
// repeated heads: 75 us of GPU time and more on the host for 256 positions of 32 heads of 64); here it is one, and it reads
// and writes the projections' own layouts, so that no transposition is left either.
//
// One block of 128 threads per 32 queries of a head; keys in tiles of 32.  A thread holds 2 x 4 scores and 2 rows of HD / 32
// vectors of the output; scores and output take as many clocks of FMA issue as of shared-memory loads.  The next tile's keys and
// values are on the way in registers while the present one is worked on.  Softmax runs along with the tiles (running
// maximum and sum).  Longest rows first: a tail of short blocks fills the SMs.
#pragma once
#include "kernels.cuh"

namespace tllm {

#define AT_ROWS 32
#define AT_THREADS 128

// four consecutive values as floats; 8-byte (16-bit types) or 16-byte loads
template <typename T>
__device__ __forceinline__ float4 at_load4(const T* p);
template <>
__device__ __forceinline__ float4 at_load4<float>(const float* p) { return __ldcg((const float4*)p); }
template <>
__device__ __forceinline__ float4 at_load4<__half>(const __half* p) {
    const uint2 a = __ldcg((const uint2*)p);
    const float2 lo = __half22float2(*(const __half2*)&a.x), hi = __half22float2(*(const __half2*)&a.y);
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
template <>
__device__ __forceinline__ float4 at_load4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 a = __ldcg((const uint2*)p);
    const float2 lo = __bfloat1622float2(*(const __nv_bfloat162*)&a.x), hi = __bfloat1622float2(*(const __nv_bfloat162*)&a.y);
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
__device__ __forceinline__ void at_store4(float* p, float4 v) { *(float4*)p = v; }
__device__ __forceinline__ void at_store4(__half* p, float4 v) {
    const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    *(uint2*)p = make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b);
}
__device__ __forceinline__ void at_store4(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *(uint2*)p = make_uint2(*(const uint32_t*)&a, *(const uint32_t*)&b);
}

template <int HD>
constexpr size_t at_smem_bytes() { return (size_t)AT_ROWS * ((HD + 4) * 2 + HD + 36) * sizeof(float); }

// qkv: [batch * M][ld], query heads, then key heads, then value heads of HD each; out: [batch * M][H * HD].
// grid (query tiles, H, batch); queries see the keys up to their own position.
template <typename T, int HD>
__global__ void __launch_bounds__(AT_THREADS) causal_attention_kernel(const T* __restrict__ qkv, T* __restrict__ out, int M, int H, int HKV, int ld, float scale) {
    extern __shared__ __align__(16) float at_smem[];
    constexpr int P = HD + 4, V4 = HD / 4, NL = AT_ROWS * V4 / AT_THREADS, NO = HD / 32;    // pitch, vectors per row, loads per thread and tile, output vectors
    float *Qs = at_smem, *Ks = Qs + AT_ROWS * P, *Vs = Ks + AT_ROWS * P, *Ps = Vs + AT_ROWS * HD;   // Ps: [32][36]
    const int tid = threadIdx.x, tx = tid & 7, r0 = (tid >> 3) * 2;
    const int qt = gridDim.x - 1 - blockIdx.x, q0 = qt * AT_ROWS, h = blockIdx.y, hk = h / (H / HKV);
    const T* base = qkv + (size_t)blockIdx.z * M * ld;
    const T *q = base + (size_t)h * HD, *k = base + (size_t)(H + hk) * HD, *v = base + (size_t)(H + HKV + hk) * HD;
    pdl_launch_dependents();
    pdl_wait();
    float4 kn[NL], vn[NL];
    auto fetch = [&](int t) {
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            const int e = tid + i * AT_THREADS, row = min(t * AT_ROWS + e / V4, M - 1), c = e % V4 * 4;
            kn[i] = at_load4<T>(k + (size_t)row * ld + c);
            vn[i] = at_load4<T>(v + (size_t)row * ld + c);
        }
    };
    fetch(0);
#pragma unroll
    for (int i = 0; i < NL; ++i) {
        const int e = tid + i * AT_THREADS, row = min(q0 + e / V4, M - 1), c = e % V4 * 4;
        float4 a = at_load4<T>(q + (size_t)row * ld + c);
        a.x *= scale, a.y *= scale, a.z *= scale, a.w *= scale;
        *(float4*)(Qs + (e / V4) * P + c) = a;
    }
    float4 o[2][NO];
    float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int j = 0; j < NO; ++j) o[r][j] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int t = 0; t <= qt; ++t) {
        __syncthreads();                                   // the previous tile has been read
#pragma unroll
        for (int i = 0; i < NL; ++i) {
            const int e = tid + i * AT_THREADS;
            *(float4*)(Ks + (e / V4) * P + e % V4 * 4) = kn[i];
            *(float4*)(Vs + (e / V4) * HD + e % V4 * 4) = vn[i];
        }
        __syncthreads();
        if (t < qt) fetch(t + 1);
        float s[2][4] = {};
#pragma unroll 8
        for (int d = 0; d < V4; ++d) {
            float4 a[2], b[4];
#pragma unroll
            for (int r = 0; r < 2; ++r) a[r] = *(const float4*)(Qs + (r0 + r) * P + 4 * d);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *(const float4*)(Ks + (tx + 8 * j) * P + 4 * d);
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[r][j] += a[r].x * b[j].x + a[r].y * b[j].y + a[r].z * b[j].z + a[r].w * b[j].w;
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float m = mx[r];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (t == qt && tx + 8 * j > r0 + r) s[r][j] = -INFINITY;      // keys after the query (past the end of the prompt among them)
                m = fmaxf(m, s[r][j]);
            }
#pragma unroll
            for (int x = 1; x < 8; x <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
            const float shrink = expf(mx[r] - m);          // first tile: exp(-inf) = 0
            mx[r] = m;
            sum[r] *= shrink;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float e = expf(s[r][j] - m);
                sum[r] += e;
                Ps[(r0 + r) * 36 + tx + 8 * j] = e;
            }
#pragma unroll
            for (int j = 0; j < NO; ++j) o[r][j].x *= shrink, o[r][j].y *= shrink, o[r][j].z *= shrink, o[r][j].w *= shrink;
        }
        __syncwarp();                                      // a row's scores come from eight lanes of this warp
#pragma unroll 2
        for (int c = 0; c < AT_ROWS; c += 4) {
            const float4 p0 = *(const float4*)(Ps + r0 * 36 + c), p1 = *(const float4*)(Ps + (r0 + 1) * 36 + c);
            const float w0[4] = {p0.x, p0.y, p0.z, p0.w}, w1[4] = {p1.x, p1.y, p1.z, p1.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < NO; ++j) {
                    const float4 b = *(const float4*)(Vs + (c + i) * HD + tx * 4 + 32 * j);
                    o[0][j].x += w0[i] * b.x, o[0][j].y += w0[i] * b.y, o[0][j].z += w0[i] * b.z, o[0][j].w += w0[i] * b.w;
                    o[1][j].x += w1[i] * b.x, o[1][j].y += w1[i] * b.y, o[1][j].z += w1[i] * b.z, o[1][j].w += w1[i] * b.w;
                }
        }
        __syncwarp();
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
#pragma unroll
        for (int x = 1; x < 8; x <<= 1) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], x);
        const int row = q0 + r0 + r;
        if (row < M) {
            const float inv = 1.f / sum[r];
            T* y = out + ((size_t)blockIdx.z * M + row) * ((size_t)H * HD) + (size_t)h * HD;
#pragma unroll
            for (int j = 0; j < NO; ++j) at_store4(y + tx * 4 + 32 * j, make_float4(o[r][j].x * inv, o[r][j].y * inv, o[r][j].z * inv, o[r][j].w * inv));
        }
    }
}

}  // namespace tllm
