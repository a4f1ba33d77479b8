// bits_kernel.cuh -- the product on few activation rows: two-bit tiles of W streamed from HBM, decoded in registers and
// multiplied with mma.sync.
//
//   D[n, m] = sum_k Wt[n, k] * X[m, k]      A = sixteen columns of W (decoded in registers), B = eight activation rows
//
// What bounds it.  At 0.25 bytes per entry the stream is the smallest form of W this library has (a 4096 x 11008 matrix is
// 11.3 MB, 1.7 us at the measured copy bandwidth), so on all but the largest matrices the time of a launch is its chain
// of latencies: launch, first bytes of W, activations once the preceding kernel has left, sum over the warps, store.
// Hence:
//   * no tensor memory, no operand tiles in shared memory, no role hand-over: a lane decodes what it loaded (a shift and
//     an AND per two entries, bittile_format.h) straight into the A fragment of mma.sync.m16n8k16.  tcgen05 would need the
//     decoded tile written to shared memory or tensor memory first, and its rate is not what limits eight rows;
//   * a block owns whole columns (groups of sixteen, dealt out evenly) over all of K; its sixteen warps cut K, and the
//     columns two or four ways where it owns many: no scratch, no counters, no second pass over global memory.  The warps'
//     partial sums meet in shared memory and are added in warp order, so results do not depend on scheduling;
//   * W travels by cp.async, several pairs of slices ahead, into slots that belong to one warp: no block barrier in
//     the main loop, and W is in flight before the preceding kernel has finished (griddepcontrol.wait);
//   * X travels the same way, each warp its own pairs of slices; or, where several warps would fetch the same ones (the columns cut two or four ways, several
//     passes) or a warp's loads would lie apart (most calls by columns or on odd addresses), whole, once, for all warps of the block (SHARED; bits_share has the
//     rule and its figures): as much of it as of W went through L2 four times over (16 rows of fp16 on 2048 x 16384: 64 KB of X a block, fetched four
//     times, for 57 KB of W);
//   * sixteen warps (four per scheduler hide the latency of shared-memory load -> decode -> MMA; with two per scheduler the
//     loop issued 0.49 instructions per clock), one block to an SM (bits_launch);
//   * the shifts of the decode are multiplications by a value in a register: they run on the FMA pipe beside the ANDs on the
//     ALU pipe, both of which take two clocks per warp instruction.
//
// Measured, fp16, CUDA-graph chain of distinct weights from HBM (us; before = the fastest of the other kernels):
//   2048 x 2048    1 row  2.1 (gather 3.9)      8 rows  2.3 (batched 11.5)
//   4096 x 11008   1 row  5.6 (gather 8.2, 75 % zeros; four-bit planes 10.5)   8 rows  6.0 (17.2)   16 rows  9.2 (19.5)
//   8192 x 10240   1 row  8.8 (four-bit planes 15.4)     8 rows 10.2 (22.7)
// fp32: three MMAs per eight rows, whose values a lane cuts into all three pieces at once (BY_PIECE; each block of columns of B by itself 4.5, 8.0 and 11.5):
//   2048 x 2048    8 rows  3.7      4096 x 4096    8 rows  6.6       8192 x 2048    8 rows  8.8
// int8: seven instructions instead of fifteen decode sixteen entries, and two MMAs (m16n8k32) replace four:
//   2048 x 8192    1 row  2.7 (as fp16 3.5)      32 rows 5.4 in one launch (9.3 in two)
//   8192 x 10240   1 row  6.6 (12.0)             16 rows 11.8 (22)
// Of the 8.8 us of 8192 x 10240, 5.4 are there without decode and MMAs; masks and MMAs, which hardly overlap, take 65 to 70 clocks of a scheduler per
// 1024 entries (53 with the same instructions and nothing to wait for).
//
// Precision.  fp16 / bf16 activations are multiplied as they are; int8 as int8 with int32 sums of +-64 * x
// (exact below BT_MAX_INT8_K inners); an fp32 value is cut into
// three bf16 values of eight significant bits each (truncation, so the three add up to it exactly), three columns of B
// whose sums are added at the end.  W is 0 / +-2 (the factor two is taken back with the scale), products are exact, sums
// are fp32; integer activations give exact sums below 2^24.  A sum that is not finite is taken again entry by entry
// (column_sum.cuh).  fp32 values below 2^-110 lose the bits under 2^-133, the last place of a bf16 value.
#pragma once
#include <type_traits>

#include "bittile_format.h"
#include "column_sum.cuh"
#include "kernels.cuh"

namespace tllm {

#define BT_WARPS 16
#define BT_SMEM_ALONE (116u * 1024u)    // two blocks of this size do not share an SM
#define BT_MAX_ROWS 16                  // rows of one launch (NB = 2 blocks of eight columns of B; fp32: 8 rows, three blocks; int8: 32, four)
#define BT_MASK 0xC000C000u             // the two codes at the top of a word's halves: 16-bit floats 0 / +-2
#define BT_MASK8 0xC0C0C0C0u            // the four at the top of its bytes: 0 / +-64
#define BT_SMEM_ALL (226u * 1024u)
#define BT_BAR_BYTES 32u                // two barriers, and whether a wait ran out
#define BT_ERR_WAIT 3                   // status word: a bounded wait ran out
#define BT_MAX_INT8_K (1 << 18)         // int8: 64 * 128 * K has to stay below 2^31

struct BitsParams {
    const uint4* bits;
    const void* X;
    void* Y;
    int* status;
    int x_dtype, x_layout, x_ld;   // row-major X: elements between rows; column-major X: elements between k
    int y_dtype, epilogue;         // epilogue 1: columns are (gate, up) pairs, Y[c / 2] = silu(g * scale) * (u * scale2)
    long long y_step_n, y_step_m;  // elements from column to column and from row to row of Y
    bool y_wide;                   // four neighbouring columns are one store
    int M, K, N, KB;               // KB = ceil(K / 64) slices
    int own, own_more;             // groups of sixteen columns per block; the first own_more blocks have one more
    int per_pass;                  // groups per pass (<= split * GR)
    int split_log;                 // the warps cut the block's columns 1 << split_log ways (1, 2 or 4); 16 >> split_log warps cut K
    int slots, depth;              // pairs of slices of W a warp has room for, pairs in flight (1, 2, 4 or 8; < slots unless no slot is used twice)
    uint32_t slot_bytes;           // shared memory of one pair of slices: GR * 512, and of X, unless it is shared, M * 128 * E
    int x_pairs, x_chunks;         // X shared by the warps: pairs of slices of a chunk (a multiple of sixteen), one chunk or two
    uint32_t x_pitch, x_chunk;     // shared memory of a row, and of the first chunk of it
    uint32_t ring_at, red_at, bar_at;      // where W, the partial sums and the barriers lie
    uint32_t m_inv;                // ceil(2^32 / M): idx / M = umulhi(idx, m_inv) for M > 1
    uint32_t mul4, mul16;          // 4 and 16
    bool pdl;                      // host: launch beside the preceding kernel
    float scale, scale2;
};

template <int XT>
struct BitsAct;   // E: bytes of an activation; P: columns of B (16-bit values) it becomes
template <>
struct BitsAct<TLLM_F32> { static constexpr int E = 4, P = 3; };
template <>
struct BitsAct<TLLM_F16> { static constexpr int E = 2, P = 1; };
template <>
struct BitsAct<TLLM_BF16> { static constexpr int E = 2, P = 1; };
template <>
struct BitsAct<TLLM_I8> { static constexpr int E = 1, P = 1; };

template <bool BF16>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_16832(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
// `bytes` (a multiple of 16) of a row by the TMA unit
__device__ __forceinline__ void bt_load_row(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits until at most `left` of the newest groups are in flight (7, 3, 1 or 0)
__device__ __forceinline__ void cp_wait(int left) {
    if (left >= 7) asm volatile("cp.async.wait_group 7;" ::: "memory");
    else if (left >= 3) asm volatile("cp.async.wait_group 3;" ::: "memory");
    else if (left >= 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ uint4 bt_lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint2 bt_lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void bt_sts128(uint32_t addr, const uint4& v) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Sixteen bytes of a row that starts on any address: the one or two aligned vectors that hold them, shifted; bytes past the
// row's end are zero.  Only vectors that hold at least one byte of the row are read.
__device__ __forceinline__ uint4 bt_load_unaligned(const char* row, int off, int row_bytes) {
    const int left = row_bytes - off;
    if (left <= 0) return make_uint4(0u, 0u, 0u, 0u);
    const char* p = row + off;
    const uint32_t sh = (uint32_t)((uintptr_t)p & 15u);
    const uint4* v = (const uint4*)(p - sh);
    const uint4 a = __ldcg(v), b = sh && left > (int)(16u - sh) ? __ldcg(v + 1) : make_uint4(0u, 0u, 0u, 0u);
    uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    if (sh & 8u) {
#pragma unroll
        for (int i = 0; i < 6; ++i) w[i] = w[i + 2];
    }
    if (sh & 4u) {
#pragma unroll
        for (int i = 0; i < 5; ++i) w[i] = w[i + 1];
    }
    const uint32_t bs = (sh & 3u) * 8u;
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        o[i] = __funnelshift_r(w[i], w[i + 1], bs);
        const int keep = left - 4 * i;                    // bytes of this word inside the row
        if (keep < 4) o[i] = keep <= 0 ? 0u : o[i] & (0xFFFFFFFFu >> (8 * (4 - keep)));
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
// The same sixteen bytes of a column-major X (elements of one row are x_ld apart).  All loads are issued, past the end of K that of the last element again: with a
// condition each, sixteen of them wait for one another's predicates (two rows of int8, 2048 x 2048: 4.5 us, 4.0 so; 2048 x 8192 5.3 and 4.3).
template <int E>
__device__ __forceinline__ uint4 bt_load_strided(const void* X, int m, int k, int K, size_t ld) {
    constexpr int COUNT = 16 / E;
    uint32_t x[COUNT], o[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < COUNT; ++i) {
        const size_t at = (size_t)min(k + i, K - 1) * ld + m;
        x[i] = E == 4 ? __ldcg((const unsigned int*)X + at) : E == 2 ? (uint32_t)__ldcg((const unsigned short*)X + at) : (uint32_t)__ldcg((const unsigned char*)X + at);
    }
#pragma unroll
    for (int i = 0; i < COUNT; ++i) o[i * E / 4] |= (k + i < K ? x[i] : 0u) << (8 * E * i % 32);
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// Where the 16-byte chunk `ch` of a pair of slices of row m lies in the row's 128 * E bytes: the four lanes that multiply one
// row and the rows of two neighbouring groups of four then read eight different bank groups.  (The copy writes whole rows
// in order but for this: chunks scattered by lane instead made cp.async four times slower, 57 against 15 us for sixteen rows
// of a 4096 x 11008 matrix.)
template <int XT>
__device__ __forceinline__ uint32_t bt_chunk(uint32_t ch, uint32_t m) {
    if (XT == TLLM_F32) return ch ^ (((ch >> 3) & 1u) | ((m & 1u) << 1));
    if (XT == TLLM_I8) return ch ^ ((m & 1u) << 2);
    return ch ^ (m & 1u);
}
// Offset of the lane's first chunk of slice 0 in row m; the other chunks are an addition (slice) and an exclusive or (chunk) away.
template <int XT>
__device__ __forceinline__ uint32_t bt_lane_chunk(uint32_t t, uint32_t m) { return bt_chunk<XT>(t * BitsAct<XT>::E, m) * 16u; }
// The lane's sixteen activations of slice h (rows 16t .. 16t+15) -> the eight words of a B fragment (word p = rows 2p, 2p+1);
// `at` is the address of the lane's first chunk of slice 0.  fp32: the `piece`-th of the three bf16 values that add up to
// each of them.  int8: four words, word s = rows 8+2s, 2s, 9+2s, 2s+1, which is where the codes stand that a shift by 2s brings to the
// top of a word's bytes.  IN_ORDER: the chunks follow one another; else they lie where bt_chunk says.
template <int XT, bool IN_ORDER>
__device__ __forceinline__ uint4 bt_load_chunk(uint32_t at, uint32_t h, uint32_t c) {
    constexpr uint32_t CS = BitsAct<XT>::E;
    if (IN_ORDER) return bt_lds128(at + h * (CS * 64u) + c * 16u);
    return bt_lds128((XT == TLLM_I8 ? at ^ (h * 64u) : at + h * (CS * 64u)) ^ (c * 16u));
}
template <int XT, bool IN_ORDER>
__device__ __forceinline__ void bt_fragment(uint32_t at, uint32_t h, int piece, uint32_t (&b)[XT == TLLM_I8 ? 4 : 8]) {
    constexpr uint32_t CS = BitsAct<XT>::E;
    uint32_t w[4 * CS];
#pragma unroll
    for (uint32_t c = 0; c < CS; ++c) {
        const uint4 v = bt_load_chunk<XT, IN_ORDER>(at, h, c);
        w[4 * c] = v.x, w[4 * c + 1] = v.y, w[4 * c + 2] = v.z, w[4 * c + 3] = v.w;
    }
    if constexpr (XT == TLLM_F32) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
#pragma unroll
            for (int p = 0; p < 2; ++p) {       // what the upper half (eight significant bits) leaves, exactly
                const float rest = __uint_as_float(w[i]) - __uint_as_float(w[i] & 0xFFFF0000u);
                if (p < piece) w[i] = __float_as_uint(rest);
            }
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i] = __byte_perm(w[2 * i], w[2 * i + 1], 0x7632);
    } else if constexpr (XT == TLLM_I8) {
#pragma unroll
        for (int i = 0; i < 4; ++i) b[i] = __byte_perm(w[i >> 1], w[2 + (i >> 1)], i & 1 ? 0x3726 : 0x1504);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i] = w[i];
    }
}
// fp32: all three pieces, as fragments of three blocks of columns of B; the values are read and cut once
template <bool IN_ORDER>
__device__ __forceinline__ void bt_pieces(uint32_t at, uint32_t h, uint32_t (&b)[3][8]) {
#pragma unroll
    for (uint32_t c = 0; c < 4; ++c) {
        const uint4 v = bt_load_chunk<TLLM_F32, IN_ORDER>(at, h, c);
        uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            b[p][2 * c] = __byte_perm(w[0], w[1], 0x7632), b[p][2 * c + 1] = __byte_perm(w[2], w[3], 0x7632);
            if (p < 2) {
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = __float_as_uint(__uint_as_float(w[i]) - __uint_as_float(w[i] & 0xFFFF0000u));
            }
        }
    }
}

// elements at .. at + 3, which lie on a multiple of their size
__device__ __forceinline__ void store_four(void* Y, int dtype, size_t at, const float (&v)[4]) {
    if (dtype == TLLM_F32) {
        *(float4*)((float*)Y + at) = make_float4(v[0], v[1], v[2], v[3]);
        return;
    }
    uint32_t w[2];
    if (dtype == TLLM_F16) {
        const __half2 a = __floats2half2_rn(v[0], v[1]), b = __floats2half2_rn(v[2], v[3]);
        w[0] = *reinterpret_cast<const uint32_t*>(&a), w[1] = *reinterpret_cast<const uint32_t*>(&b);
    } else {
        const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
        w[0] = *reinterpret_cast<const uint32_t*>(&a), w[1] = *reinterpret_cast<const uint32_t*>(&b);
    }
    *(uint2*)((unsigned short*)Y + at) = make_uint2(w[0], w[1]);
}
// column n of row m, entry by entry, for a sum that is not finite
template <int XT>
__device__ __noinline__ float bt_column_sum(const BitsParams& p, int n, int m) {
    return column_sum((const uint32_t*)p.bits, n, p.K, p.KB, false, [&](int k) {
        return load_act_f32_cg(p.X, XT, p.x_layout == TLLM_ROW_MAJOR ? (size_t)m * p.x_ld + k : (size_t)k * p.x_ld + m);
    });
}
// Those of columns n .. n + 3 of row m again, entry by entry, whose sums (v0 .. v3) are not finite: behind the stores of all four, so that next to no register
// has to live through the call.  A finite sum keeps its bits.
template <int XT>
__device__ __noinline__ void bt_store_again(const BitsParams& p, int n, int m, float v0, float v1, float v2, float v3) {
    const auto result = [&](int k, float v, float sc) {              // (a call of bt_column_sum from here cost the callers registers)
        if (finite_sum(v)) return v * sc;
        return column_sum((const uint32_t*)p.bits, n + k, p.K, p.KB, false, [&](int i) {
                   return load_act_f32_cg(p.X, XT, p.x_layout == TLLM_ROW_MAJOR ? (size_t)m * p.x_ld + i : (size_t)i * p.x_ld + m);
               }) * (2.f * sc);
    };
#pragma unroll 1
    for (int k = 0; k < 4 && n + k < p.N; k += 2, v0 = v2, v1 = v3) {
        size_t at = (size_t)m * p.y_step_m;
        if (p.epilogue == 0) {
            at += (size_t)(n + k) * p.y_step_n;
            if (!finite_sum(v0)) store_out(p.Y, p.y_dtype, at, result(k, v0, p.scale));
            if (n + k + 1 < p.N && !finite_sum(v1)) store_out(p.Y, p.y_dtype, at + p.y_step_n, result(k + 1, v1, p.scale));
        } else if (n + k + 1 < p.N && !(finite_sum(v0) && finite_sum(v1)))
            store_out(p.Y, p.y_dtype, at + ((n + k) >> 1), silu_mul(result(k, v0, p.scale), result(k + 1, v1, p.scale2)));
    }
}

// A warp multiplies up to GR groups of sixteen columns by NB blocks of eight columns of B (activation rows; fp32: pieces of
// rows).  A block with more than split * GR groups makes several passes.
// ASYNC: the rows of X start on 16 bytes and are a multiple of 16 bytes long; otherwise they pass through registers.
// SHARED: X lies in shared memory once for all warps, else each has its own pairs of slices.
//
// The code is kept short (rolled loops, no divisions): a warp of a small product runs the loop body once or twice, and then
// fetching instructions costs more than executing them.
template <int XT, int NB, int GR, bool ASYNC, bool SHARED>
__global__ void __launch_bounds__(BT_WARPS * 32, 1) bits_spmm_kernel(const __grid_constant__ BitsParams p) {
    extern __shared__ __align__(128) unsigned char bt_smem[];
    using Act = BitsAct<XT>;
    constexpr bool BF16 = XT == TLLM_BF16 || XT == TLLM_F32, I8 = XT == TLLM_I8;
    using Sum = typename std::conditional<I8, int, float>::type;
    // The tensor core cuts bits off its running sum at every MMA: fp32 sums leave it after the eight of a pair of slices (gate and up of a
    // 2560 / 6912 MLP, 8 rows, h = silu(gate) * up: off by 1.4e-7 with a warp's 40 MMAs in one sum, 1.1e-7 now).
    constexpr bool PARTS = XT == TLLM_F32;
    // Columns of B: piece of row m is column 3 m + piece; with three blocks of them block `piece` has column m, so that a lane cuts the values of one
    // row and has all of its columns.
    constexpr bool BY_PIECE = XT == TLLM_F32 && NB == 3;
    constexpr uint32_t PAIR = 128u * Act::E;                               // bytes of a row in a pair of slices
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int b = blockIdx.x, c0 = b * p.own + min(b, p.own_more), own = p.own + (b < p.own_more);
    const int KB = p.KB, KP = (KB + 1) >> 1, D = p.depth, S = p.slots, M = p.M, SL = p.split_log;
    // Which share of the columns: the shares may differ by a group, and every scheduler (warp modulo 4) gets some of each, so that none has
    // all of the larger ones (8192 x 10240, one row of bf16: 10.2 us, 11.5 with share = warp modulo shares; 4096 x 11008, fp16 6.0 and 6.5).  One
    // expression for two and for four shares: with a choice between two every call got slower (2048 x 8192, eight rows of fp32 8.03 us, 7.85 now).
    const int kw = warp >> SL, klog = 4 - SL, kstep = 1 << klog, cw = (warp + (warp >> 2)) & ((1 << SL) - 1);
    const int np = kw < KP ? (KP - kw + kstep - 1) >> klog : 0;      // pairs of this warp: kw, kw + kstep, ...
    const uint32_t smem = smem_u32(bt_smem), ring = smem + p.ring_at + (uint32_t)warp * (uint32_t)S * p.slot_bytes;
    Sum* red = (Sum*)(bt_smem + p.red_at);                           // [warp][group][column of B][20] partial sums
    const uint32_t bars = smem + p.bar_at;
    volatile int* abort_flag = (volatile int*)(bt_smem + p.bar_at + 16);
    const uint32_t group_bytes = (uint32_t)KB * 256u;
#define BT_FULL(i) (bars + 8u * (uint32_t)(i))           // X's chunks, 0 and 1
    pdl_launch_dependents();
    // There is a block for every SM even where there are fewer groups; the spare ones hold their place until the preceding kernel is through.  (Without them 96 MLPs
    // of 512 to 2560 / 1024 to 8192, 1 to 16 rows, in graphs took 1.003 of the time, 512 / 1408 up to 1.05; 1765 products after themselves 0.999, 0.92 to 1.07.)
    if (own == 0) {
        pdl_wait();
        return;
    }

    // A pass covers groups [q0, q0 + n) of the block; this warp's share is [n * cw / split, n * (cw + 1) / split) of them.
    // ---- copies of W: the warp's step s (its pairs in order, pass after pass) goes to slot s % S ----------------------
    const char* wsrc;                                                // first group of the pass being fetched, this warp's next pair
    uint32_t last;                                                   // offset of the last group from it
    int fpass = 0, fi = 0, fs = 0;                                   // next copy: first group of the pass, pair, slot
    auto open_pass = [&]() {
        const int n = min(p.per_pass, own - fpass), a = (n * cw) >> SL, e = (n * (cw + 1)) >> SL;
        wsrc = (const char*)p.bits + (size_t)(c0 + fpass + a) * group_bytes + (size_t)kw * 512u;
        last = (uint32_t)max(e - a - 1, 0) * group_bytes;
    };
    const uint32_t wchunk = (uint32_t)mm_chunk(g, t) * 16u;          // where this lane's chunk of a pair lies
    auto copy_w = [&](uint32_t slot) {
        uint32_t dst = slot + (uint32_t)lane * 16u;
        if (2 * (kw + (fi << klog)) + 2 <= KB) {
#pragma unroll
            for (int j = 0; j < GR; ++j) cp_async16(dst + (uint32_t)j * 512u, wsrc + min((uint32_t)j * group_bytes, last) + lane * 16);
        } else {                                                     // an odd last slice
            dst = slot + wchunk;
#pragma unroll
            for (int j = 0; j < GR; ++j) {
                cp_async8(dst + (uint32_t)j * 512u, wsrc + min((uint32_t)j * group_bytes, last) + lane * 8);
                asm volatile("st.shared.v2.b32 [%0], {%1, %1};" ::"r"(dst + (uint32_t)j * 512u + 8u), "r"(0u) : "memory");
            }
        }
    };
    auto advance = [&]() {
        wsrc += (uint32_t)kstep * 512u;
        if (++fi == np) {
            fi = 0, fpass += p.per_pass;
            open_pass();
        }
        if (++fs == S) fs = 0;
    };
    open_pass();
#pragma unroll 1
    for (int s = 0; s < D; ++s) {                                    // W does not depend on the preceding kernel
        if (fpass < own && np) {
            copy_w(ring + (uint32_t)fs * p.slot_bytes);
            advance();
            if (SHARED) cp_commit();
        } else if (SHARED) cp_commit();
    }
    const int pre_pass = fpass, pre_i = fi;
    if (SHARED) {
        if (tid == 0) {
            mbar_init(BT_FULL(0), ASYNC ? M : BT_WARPS * 32);
            mbar_init(BT_FULL(1), ASYNC ? M : BT_WARPS * 32);
            *abort_flag = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncthreads();
    }

    // ---- X, of one warp's pair: the lanes copy whole rows, 16 bytes each
    constexpr int CPR = 8 * Act::E, RPI = 32 / CPR, KPC = 16 / Act::E;     // chunks per row (and pair of slices), rows per warp copy, values per chunk
    const uint32_t xm = (uint32_t)lane / CPR, xch = (uint32_t)lane % CPR;
    auto copy_x = [&](int i, uint32_t slot) {
        const int k = (kw + (i << klog)) * 128 + (int)xch * KPC;
        const char* src = (const char*)p.X + ((size_t)xm * p.x_ld + k) * Act::E;
        const uint32_t xb = slot + GR * 512u;
#pragma unroll 1
        for (uint32_t m = xm; m < (uint32_t)M; m += RPI, src += (size_t)RPI * p.x_ld * Act::E) {
            const uint32_t dst = xb + (m * CPR + bt_chunk<XT>(xch, m)) * 16u;
            if (ASYNC) {
                if (k < p.K) cp_async16(dst, src);
                else bt_sts128(dst, make_uint4(0u, 0u, 0u, 0u));
            } else if (p.x_layout == TLLM_ROW_MAJOR) {
                bt_sts128(dst, bt_load_unaligned((const char*)p.X + (size_t)m * p.x_ld * Act::E, k * Act::E, p.K * Act::E));
            } else {
                bt_sts128(dst, bt_load_strided<Act::E>(p.X, (int)m, k, p.K, (size_t)p.x_ld));
            }
        }
    };
    // ---- X, of all warps: whole, in one chunk of x_pairs pairs of slices or in two that arrive one after the other.  (Rows are x_pitch bytes apart,
    // 16 (fp32: 32, int8: 64) more than a multiple of 128, so that the lanes of a fragment read different banks.)
    auto load_x = [&](int chunk) {
        const int k0 = chunk * p.x_pairs * 128, k1 = min(k0 + p.x_pairs * 128, KP * 128);      // zero past the end of K
        const uint32_t to = smem + (uint32_t)chunk * p.x_chunk;
        if (ASYNC) {
            if (warp == BT_WARPS - 1 && lane < M) {                  // a lane per row
                const uint32_t row = to + (uint32_t)lane * p.x_pitch, bytes = (uint32_t)(min(k1, p.K) - k0) * Act::E;
                for (uint32_t z = bytes; z < (uint32_t)(k1 - k0) * Act::E; z += 16u) bt_sts128(row + z, make_uint4(0u, 0u, 0u, 0u));
                mbar_expect_tx(BT_FULL(chunk), bytes);
                bt_load_row(row, (const char*)p.X + ((size_t)lane * p.x_ld + k0) * Act::E, bytes, BT_FULL(chunk));
            }
        } else {
            const bool rows = p.x_layout == TLLM_ROW_MAJOR;
            const uint32_t per_row = (uint32_t)(k1 - k0) * Act::E / 16u, inner = rows ? per_row : (uint32_t)M;
#pragma unroll 1
            for (uint32_t i = (uint32_t)tid; i < per_row * (uint32_t)M; i += BT_WARPS * 32) {
                const uint32_t hi = i / inner, lo = i - hi * inner, m = rows ? hi : lo, c = rows ? lo : hi;
                const int k = k0 + (int)c * (16 / Act::E);
                bt_sts128(to + m * p.x_pitch + c * 16u, rows ? bt_load_unaligned((const char*)p.X + (size_t)m * p.x_ld * Act::E, k * Act::E, p.K * Act::E)
                                                             : bt_load_strided<Act::E>(p.X, (int)m, k, p.K, (size_t)p.x_ld));
            }
            mbar_arrive_n(BT_FULL(chunk), 1u);
        }
    };
    pdl_wait();
    if (SHARED) {
        load_x(0);
        if (p.x_chunks > 1) load_x(1);
    } else {
        int i = 0, pass = 0;
#pragma unroll 1
        for (int s = 0; s < D; ++s) {
            if (np && (pass < pre_pass || i < pre_i)) {
                copy_x(i, ring + (uint32_t)s * p.slot_bytes);
                if (++i == np) i = 0, pass += p.per_pass;
            }
            cp_commit();
        }
    }

    // This lane's column of B in block nb: a row of X (any row, past the last column: those sums are not used) and its piece.
    uint32_t bat[NB];
    int bpiece[NB];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
        const uint32_t c = (uint32_t)(nb * 8 + g), m = min(BY_PIECE ? (uint32_t)g : c / Act::P, (uint32_t)M - 1u);
        bpiece[nb] = (int)(c % Act::P);
        bat[nb] = SHARED ? smem + (uint32_t)kw * PAIR + m * p.x_pitch + (uint32_t)t * (16u * Act::E) : GR * 512u + m * PAIR + bt_lane_chunk<XT>((uint32_t)t, m);
    }
    // Multipliers in registers: a shift by an immediate would run on the ALU pipe, which the ANDs already fill.
    uint32_t m4, m16;
    asm volatile("mov.b32 %0, %2;\n\tmov.b32 %1, %3;" : "=r"(m4), "=r"(m16) : "r"(p.mul4), "r"(p.mul16));
    int cs = 0;                                                      // slot being consumed
    bool ok = true;
#pragma unroll 1
    for (int q0 = 0; q0 < own; q0 += p.per_pass) {
        const int ng = min(p.per_pass, own - q0), w0 = (ng * cw) >> SL, mine = ((ng * (cw + 1)) >> SL) - w0;    // this warp's groups of the pass
        Sum acc[GR][NB][4];
#pragma unroll
        for (int j = 0; j < GR; ++j)
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[j][nb][i] = 0;
        int left = np;                                               // pairs of the pass
#pragma unroll 1
        for (int chunk = 0; chunk < (SHARED ? p.x_chunks : 1); ++chunk) {
            if (SHARED) ok = ok && bounded_wait(BT_FULL(chunk), 0u, abort_flag);
            uint32_t xat = (uint32_t)chunk * p.x_chunk;
            int here = SHARED ? min(left, p.x_pairs >> klog) : np;
            left -= here;
#pragma unroll 1
            for (; here > 0; --here, xat += (uint32_t)kstep * PAIR) {
                cp_wait(D - 1);
                __syncwarp();                                        // other lanes' chunks of W are here, and they have read the slot before
                const uint32_t slot = ring + (uint32_t)cs * p.slot_bytes;
                if (fpass < own) {                                   // into the slot that was consumed one step ago
                    const uint32_t dst = ring + (uint32_t)fs * p.slot_bytes;
                    copy_w(dst);
                    if (!SHARED) copy_x(fi, dst);
                    advance();
                }
                cp_commit();
                if (!SHARED) xat = slot;
                float part[GR][NB][4];                               // fp32: the sums of this pair of slices
                if constexpr (PARTS) {
#pragma unroll
                    for (int j = 0; j < GR; ++j)
#pragma unroll
                        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                            for (int k = 0; k < 4; ++k) part[j][nb][k] = 0.f;
                }
#pragma unroll 1
                for (uint32_t h = 0; h < 2; ++h) {
                    uint32_t bf[NB][I8 ? 4 : 8];
                    if constexpr (BY_PIECE) bt_pieces<SHARED>(bat[0] + xat, h, bf);
                    else {
#pragma unroll
                        for (int nb = 0; nb < NB; ++nb) bt_fragment<XT, SHARED>(bat[nb] + xat, h, bpiece[nb], bf[nb]);
                    }
                    auto half = [&](auto first, auto end) {          // groups [lo, hi) of the warp
                        constexpr int lo = decltype(first)::value, hi = decltype(end)::value;
                        uint2 a[GR];
#pragma unroll
                        for (int j = lo; j < hi; ++j) a[j] = bt_lds64(slot + (uint32_t)j * 512u + wchunk + h * 8u);
                        // consecutive MMAs go to different accumulators: a chain of dependent ones costs their full latency each
                        constexpr int MMAS = I8 ? 2 : 4;
                        constexpr uint32_t MASK = I8 ? BT_MASK8 : BT_MASK;
#pragma unroll
                        for (int s = 0; s < MMAS; ++s)
#pragma unroll
                            for (int j = lo; j < hi; ++j) {
                                const uint32_t a0 = a[j].x & MASK, a1 = a[j].y & MASK, a2 = (a[j].x * m4) & MASK, a3 = (a[j].y * m4) & MASK;
                                if (s < MMAS - 1) a[j].x *= m16, a[j].y *= m16;
#pragma unroll
                                for (int nb = 0; nb < NB; ++nb) {
                                    if constexpr (I8) mma_16832(acc[j][nb], a0, a1, a2, a3, bf[nb][2 * s], bf[nb][2 * s + 1]);
                                    else mma_16816<BF16>(PARTS ? part[j][nb] : acc[j][nb], a0, a1, a2, a3, bf[nb][2 * s], bf[nb][2 * s + 1]);
                                }
                            }
                    };
                    // a warp's share of a pass is GR groups or one less (or none: GR = 1)
                    if constexpr (GR > 1) half(std::integral_constant<int, 0>{}, std::integral_constant<int, GR - 1>{});
                    if (mine == GR) half(std::integral_constant<int, GR - 1>{}, std::integral_constant<int, GR>{});
                }
                if constexpr (PARTS) {
#pragma unroll
                    for (int j = 0; j < GR; ++j)
#pragma unroll
                        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                            for (int k = 0; k < 4; ++k) acc[j][nb][k] += part[j][nb][k];
                }
                if (++cs == S) cs = 0;
            }
        }
        // ---- sum over the warps that share columns: lane (g, t) holds columns g, g + 8 of W for columns 2t, 2t + 1 of B (20
        // floats apart: no bank conflicts)
        const int MC = M * Act::P;
        const int kw_step = p.per_pass * MC * 20;
        if (q0 > 0) __syncthreads();                                 // the previous pass has been read
#pragma unroll
        for (int j = 0; j < GR; ++j)
            if (j < mine) {
                Sum* r = red + (size_t)kw * kw_step + (w0 + j) * MC * 20 + g;
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    const int m = BY_PIECE ? 6 * t + nb : nb * 8 + 2 * t, m1 = m + (BY_PIECE ? 3 : 1);
                    if (m < MC) r[m * 20] = acc[j][nb][0], r[m * 20 + 8] = acc[j][nb][2];
                    if (m1 < MC) r[m1 * 20] = acc[j][nb][1], r[m1 * 20 + 8] = acc[j][nb][3];
                }
            }
        __syncthreads();
        // Sums of the warps' sums; idx = group * M + row.  Up to thirty-two of them: half a warp each, a column per thread.
        if (ng * M <= BT_WARPS * 2) {
            const int c = lane & 15;
#pragma unroll 1
            for (int i0 = warp * 2; i0 < ng * M; i0 += BT_WARPS * 2) {
                const int idx = i0 + (lane >> 4), j = M > 1 ? (int)__umulhi((uint32_t)idx, p.m_inv) : idx, m = idx - j * M;
                const bool valid = idx < ng * M;
                Sum v = 0;
                if (valid) {
                    const Sum* r = red + (j * MC + m * Act::P) * 20 + c;
#pragma unroll
                    for (int pc = Act::P - 1; pc >= 0; --pc)        // fp32: the small pieces first
#pragma unroll 4
                        for (int w = 0; w < kstep; ++w) v += r[w * kw_step + pc * 20];
                }
                const int n = (c0 + q0 + j) * 16 + c;
                if constexpr (I8) {                                  // an exact multiple of 64
                    if (valid && n < p.N) ((int*)p.Y)[(size_t)m * p.y_step_m + (size_t)n * p.y_step_n] = v >> 6;
                    continue;
                }
                const float sc = p.epilogue && (c & 1) ? p.scale2 : p.scale;
                float y = v * sc;
                if (__builtin_expect(!finite_sum(v), 0)) y = bt_column_sum<XT>(p, min(n, p.N - 1), m) * (2.f * sc);
                if (p.epilogue == 0) {
                    // (the address is computed here: before the sum it made ptxas allot other registers, 2048 x 2048, eight rows of fp16 3.15 us instead of 2.61)
                    if (valid && n < p.N) store_out(p.Y, p.y_dtype, (size_t)m * p.y_step_m + (size_t)n * p.y_step_n, y);
                } else {
                    const float u = __shfl_xor_sync(0xffffffffu, y, 1);
                    if (valid && !(c & 1) && n + 1 < p.N) store_out(p.Y, p.y_dtype, (size_t)m * p.y_step_m + (n >> 1), silu_mul(y, u));
                }
            }
            continue;
        }
        // More: four columns per thread.  (With a column per thread the loop went round four times as often, each time a chain of some 600 clocks: 16 rows of
        // fp16 on 2048 x 16384 7.2 us, 6.5 so; 32 of int8 9.7 and 8.7.)
#pragma unroll 1
        for (int i = tid; i < ng * M * 4; i += BT_WARPS * 32) {
            const int idx = i >> 2, c = (i & 3) * 4, j = M > 1 ? (int)__umulhi((uint32_t)idx, p.m_inv) : idx, m = idx - j * M;
            Sum v[4] = {};
            const Sum* r = red + (j * MC + m * Act::P) * 20 + c;
#pragma unroll
            for (int pc = Act::P - 1; pc >= 0; --pc)
#pragma unroll 4
                for (int w = 0; w < kstep; ++w) {
                    Sum x[4];
                    *(uint4*)x = *(const uint4*)(r + w * kw_step + pc * 20);
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[k] += x[k];
                }
            const int n = (c0 + q0 + j) * 16 + c;
            size_t at = (size_t)m * p.y_step_m + (size_t)n * p.y_step_n;
            if constexpr (I8) {                                      // exact multiples of 64
                if (p.y_wide && n < p.N) *(int4*)((int*)p.Y + at) = make_int4(v[0] >> 6, v[1] >> 6, v[2] >> 6, v[3] >> 6);
                else
#pragma unroll
                    for (int k = 0; k < 4; ++k, at += p.y_step_n)
                        if (n + k < p.N) ((int*)p.Y)[at] = v[k] >> 6;
                continue;
            }
            float z = 0.f;                                           // 0, or NaN from the first Inf or NaN on
#pragma unroll
            for (int k = 0; k < 4; ++k) z = fmaf((float)v[k], 0.f, z);
            if (p.epilogue == 0) {
                float y[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) y[k] = v[k] * p.scale;
                if (p.y_wide && n < p.N) store_four(p.Y, p.y_dtype, at, y);
                else
#pragma unroll
                    for (int k = 0; k < 4; ++k, at += p.y_step_n)
                        if (n + k < p.N) store_out(p.Y, p.y_dtype, at, y[k]);
            } else {
                at = (size_t)m * p.y_step_m + (n >> 1);
                if (n + 1 < p.N) store_out(p.Y, p.y_dtype, at, silu_mul(v[0] * p.scale, v[1] * p.scale2));
                if (n + 3 < p.N) store_out(p.Y, p.y_dtype, at + 1, silu_mul(v[2] * p.scale, v[3] * p.scale2));
            }
            if (__builtin_expect(z != 0.f, 0)) bt_store_again<XT>(p, n, m, v[0], v[1], v[2], v[3]);
        }
    }
    if (!ok) atomicExch(p.status, BT_ERR_WAIT);
#undef BT_FULL
}

// one launch of up to BT_MAX_ROWS rows (half of it fp32, twice int8); fills in y_wide and everything from `own` to `mul16` (bits.cu)
int bits_launch(BitsParams& p, int sms, int device, void* stream);
// how this thread's last launch was cut (tllm_bits_last_plan)
extern thread_local int bits_last_plan[6];
// How it reads X: rows on 16 bytes (cp.async), rows that start anywhere, or a column-major X
enum BitsAccess { BITS_ROWS16, BITS_ROWS, BITS_COLUMNS };
inline BitsAccess bits_access(const void* X, int x_dtype, int x_layout, int x_ld) {
    const int e = x_dtype == TLLM_F32 ? 4 : x_dtype == TLLM_I8 ? 1 : 2;
    if (x_layout != TLLM_ROW_MAJOR) return BITS_COLUMNS;
    return (uintptr_t)X % 16 == 0 && (size_t)x_ld * e % 16 == 0 ? BITS_ROWS16 : BITS_ROWS;
}
// its time, for the choice between kernels
double bits_estimate_us(int x_dtype, BitsAccess access, int rows, int inners, int columns, int sms);

}  // namespace tllm
