// mma_kernel.cuh -- the batched product on the tcgen05 tensor cores of sm_100a.
//
// The two-bit copy of W ("bit tiles") is expanded one slice of 128 columns x 64 rows at a time into fp16 / bf16 values in
// tensor memory and multiplied on the tensor cores:  D[n, m] = sum_k Wt[n, k] * X[m, k],  A = Wt slice (tensor memory, written
// by decoder warps with tcgen05.st), B = X slice (shared memory, K-major, 128-byte swizzle, written by TMA), D in tensor
// memory (fp32).  The ternary values are exact in both formats and products are exact; sums are accumulated in fp32.
//
// Why tensor memory for A: with the expanded slice in shared memory a slice of 64 rows and Nt activation rows moved
// 32 KiB of A (written and read) and Nt * 256 bytes of B through a shared memory of 128 bytes per clock -- 768 clocks at
// Nt = 256 for the 512 that the MMAs take, 320 for 64 at Nt = 32.  Without A it is Nt * 2 clocks beside MMAs of Nt * 2.
//
// X comes in one or three planes of 16-bit values.  fp16 / bf16 activations whose rows TMA can address are read where they
// are (one plane).  Everything else passes through stage_acts_kernel: int8 becomes fp16 (exact), rows on odd addresses and
// column-major activations are copied straight, and an fp32 value becomes three bf16 values of eight significant bits that
// add up to it exactly.  The planes of a row tile are rows of one B operand, 3 * Nt of them, each with its own columns of D, so
// an MMA does the three at once (three MMAs of Nt columns each instead were bound by their issue: 20 us against 12 for 256 rows
// of 2048 x 2048); D's planes are added in the epilogue, the small ones first.  (The tensor core truncates its sums: with the
// planes in one accumulator every step would cut bits, 1e-5 of the result at K = 4096 against 1e-7.)
//
// One persistent block per SM, alone or as one of a pair, twenty-seven warps (and one that has nothing to do):
//   warp 0        streams this block's range of bit tiles into a shared-memory ring (TMA, one thread)
//   warp 1        owns tensor memory and issues tcgen05.mma (one thread; a pair's second block has none)
//   warp 2        loads the activation slices by TMA (one thread)
//   warps 4..11   epilogue: tensor memory -> registers -> Y (or partial sums), four warps for every other sixteen rows (one warp per
//                 scheduler waits most of its time: 1700 clocks for sixteen rows of three planes, 780 of one; fp32 MLP module of 256 rows,
//                 2048 / 8192: 84 us with four warps, 74 with eight)
//   warps 12..27  decoders: bit tile -> tensor memory, one slice of 32 columns per warp and second unit (a warp can only write the 32
//                 lanes of tensor memory that its number modulo 4 selects)
// A unit is two consecutive slices of K.  What bounds a launch of many tiles is that the tensor core is never without an MMA:
//   * one thread issues (13 clocks an MMA), and it finds the next unit's operands ready: A has a ring of two or four units in tensor memory
//     beside two sets of accumulators, so that the sums of one tile (fp32: of one leg) leave while the next one's MMAs run; the decoders have
//     the values in registers when a place is free;
//   * a pair of blocks shares the MMAs (tcgen05 cta_group::2): 256 columns of W, 128 in each block's tensor memory, by Nt activation
//     rows, half of them in each block's shared memory.  For a block by itself writing and reading the activations takes all of the
//     128 bytes that its shared memory moves per clock.
// An MMA of N columns then takes 0.52 N + 13 to 25 clocks, the latter while decoders write to tensor memory.  Measured against a unit of four
// slices, one block per tile, a warp that elects a lane per MMA and one set of accumulators for three planes: 2048 rows of 5120 x 15360
// bf16 233 us (276; both at the power cap), 256 rows of fp32 2048 x 16384 42 us with its planes (55), 2048 x 8192 28 us (36).
// Work is either whole output tiles or, where those would leave SMs idle, the flattened list of (output tile, unit) pairs
// cut into equal contiguous ranges, one per block or pair.  Tiles that straddle two or more blocks are summed in block order by the
// last block to arrive, which makes the result independent of scheduling; a block does its two shared tiles first, so that
// this adding-up hides behind the tiles it has to itself.
// With few tiles a third way: a cluster of two, four or eight blocks, or of two or four pairs, cuts the units of one tile.  Each block sends its sums
// of the rows that another one is to write straight into that one's shared memory, so that a hand-over costs one trip between SMs, not
// partial sums to L2, a counter and partial sums back, and every block adds and writes a share of the tile.  (A block of a pair deals with
// the blocks of the other pairs that have its 128 columns.  256 rows of fp32 on 8192 x 2048: 26.6 us, 31.2 in equal ranges of units.)
//
// Every wait is bounded (see bounded_wait); on a time-out the block raises its abort flag, every role leaves
// its loop, tensor memory is released and the status word reports the failure.
#pragma once
#include <cuda.h>

#include <type_traits>

#include "column_sum.cuh"
#include "kernels.cuh"

namespace tllm {

#define MM_TILE_N 128                 // output columns per tile  (the MMA's M)
#define MM_TILE_K 64                  // rows of W per slice      (four MMAs of K = 16); a unit is two slices
#define MM_UNIT_BYTES 4096            // bit tiles of one unit: eight groups of sixteen columns, 512 bytes each
#define MM_UK 2
#define MM_RAW_UNITS 8                // ring of bit tiles: a power of two, at most MM_MAX_STAGES
#define MM_MAX_STAGES 8
// Units of a leg.  The tensor core cuts bits off its running sum at every MMA, always toward zero, so that a sum of many MMAs comes out too
// small: by 3.6e-7 of the result for fp32 activations of the spread that a gated MLP makes and 432 MMAs, where fp32 additions
// rounded to nearest are off by 7e-8.  The sums of fp32 activations therefore leave the accumulators after every 64 MMAs and
// are added up in fp32: 8e-8.
#define MM_LEG 8
#define MM_THREADS (28 * 32)
#define MM_MAX_COLS 192               // columns of D of a tile = planes * Nt, Nt (activation rows) a multiple of sixteen
#define MM_OWN_NT 64                  // a handle's own hand-over scratch is for tiles of up to this many rows
#define MM_MAX_M_TILES 16             // row tiles of one launch
static_assert(MM_RAW_UNITS <= MM_MAX_STAGES && (MM_RAW_UNITS & (MM_RAW_UNITS - 1)) == 0, "as many barriers as places; positions are masked");
static_assert(MM_MAX_STAGES == 8, "the barriers of the rings lie eight apart in shared memory");
// what a result is stored as
#define MM_OUT_F32 0
#define MM_OUT_I32 1
#define MM_OUT_F16 2
#define MM_OUT_BF16 3
#define MM_OUT_F16_PAIRS 4            // row-major, whole tiles of columns, rows on 4 bytes: two columns per store
#define MM_OUT_BF16_PAIRS 5
#define MM_OUT_F32_COL4 6             // column-major on 16 bytes: four rows per store
#define MM_OUT_I32_COL4 7
#define MM_OUT_PLANES 8               // the three bf16 values that add up to an fp32 result (see stage_acts_kernel)
#define MM_ERR_WAIT 3                 // status word: a bounded wait of the tensor-core kernel ran out

struct MmParams {
    void* Y;
    float* partial;           // [2 * gridDim.x][Nt / 4][128][4] fp32: a block's first and last (partial) tile
    unsigned int* counters;   // [tiles][4], zero between launches
    int* status;
    int M, K, N;
    int KB;                   // ceil(K / 64): slices
    int KBU;                  // ceil(KB / 2): units per tile
    int n_tiles, m_tiles;
    int Nt;                   // activation rows per tile; planes * Nt is the MMA's N
    int split;                // 0: whole tiles; 1: equal unit ranges, tiles may be shared; 2: a cluster per tile
    int cluster;              // blocks (CG = 2: pairs) per tile, split 2
    // How the work is dealt out (split 0: tiles, 1: units): every one of the G blocks or pairs has `share`, `share_more` of them one more; and what divisions by
    // G, KBU and m_tiles multiply with (mm_div).  (64-bit divisions in the kernel took 1500 clocks before its first copy, and again at every shared tile.)
    int share, share_more, cluster_log;
    uint32_t g_inv, kbu_inv, mt_inv;
    int P;                    // planes of X
    int out;                  // MM_OUT_*
    int epilogue, y_ld;       // epilogue 1: columns are (gate, up) pairs, Y[c / 2] = silu(g * scale) * (u * scale2)
    long long y_step_n, y_step_m;   // elements from column to column and from row to row (epilogue 0)
    long long plane_y;        // MM_OUT_PLANES: elements from plane to plane
    int SB;                   // ring length: units of B
    int R;                    // mma_units4_kernel: ring length, units of bit tiles (MS_RAW_UNITS)
    int leg;                  // units that are summed in the tensor core before the sum goes on in fp32 (MM_LEG)
    uint32_t idesc;           // tcgen05 instruction descriptor
    uint32_t mul4, mul16;     // 4 and 16
    float scale, scale2;      // half the product's scales: the decoded weights are 0 / +-2
    // Sums that are not finite (column_sum.cuh).  0: stored as they are (int8, where there are none; fp16 read in place, which 0 / +-2 cannot
    // overflow); 1: taken again from the rows that a column uses; 2: the same over every row, 0 * Inf = NaN included (bf16 read
    // in place).
    int finite;
    const uint32_t* bits;     // the bit tiles, and X where TMA reads it: plane_x elements from plane to plane, ld_x from row to row
    const unsigned short* X;
    long long plane_x, ld_x;
    bool bf16;
    bool wait_bits;           // the bit tiles are the work of a kernel that may not have finished
};

// ---- tcgen05 / TMA wrappers ------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// CG: blocks that the tensor core works for at a time, 1 or 2 (a pair); a warp of each of them allocates and releases
template <int CG = 1>
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
    if (CG == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
}
template <int CG = 1>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    if (CG == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem], issued by one thread; A: lane = row, 32-bit column c = values 2c, 2c + 1 of K.  B is given by the
// low word of its shared-memory descriptor (start address >> 4; the upper word -- K-major, 128-byte swizzle, eight-row
// groups 1024 bytes apart, version 1 -- is a constant).  CG = 2: D and A at the same columns of both blocks' tensor memory, 128 rows each;
// B's rows half in this block's shared memory and half at the same place of the other's.
template <int CG>
__device__ __forceinline__ void umma_f16_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
#define MM_UMMA(group)                                                                   \
    asm volatile(                                                                        \
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"                                      \
        "setp.ne.b32 p, %4, 0;\n\t"                                                      \
        "mov.b64 db, {%2, %5};\n\t"                                                      \
        "tcgen05.mma.cta_group::" group ".kind::f16 [%0], [%1], db, %3, p;\n\t}" ::"r"(d), \
        "r"(a), "r"(b_lo | (1u << 16)), "r"(idesc), "r"(accumulate), "r"(0x40004040u)     \
        : "memory")
    if (CG == 1) MM_UMMA("1");
    else MM_UMMA("2");
#undef MM_UMMA
}
// 32 columns of the calling warp's 32 lanes
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, "
        "%23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]),
        "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]),
        "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// the barrier (CG = 2: that of the cluster's blocks `both`) receives one arrival when every MMA issued so far by this thread has completed
template <int CG = 1>
__device__ __forceinline__ void umma_commit(uint32_t bar, uint32_t both = 3u) {
    if (CG == 1) asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((unsigned short)both)
                     : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
          "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// sixteen columns of D (rows of X) of this lane's column of W, the planes (nt columns apart) added up, the small ones first
__device__ __forceinline__ void mm_load16(uint32_t at, int nt, int planes, float (&f)[16]) {
    if (planes == 1) {
        uint32_t v[16];
        tmem_ld16(at, v);
#pragma unroll
        for (int t = 0; t < 16; ++t) f[t] = __uint_as_float(v[t]);
    } else {
        float g[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
            "tcgen05.wait::ld.sync.aligned;"
            : "=f"(f[0]), "=f"(f[1]), "=f"(f[2]), "=f"(f[3]), "=f"(f[4]), "=f"(f[5]), "=f"(f[6]), "=f"(f[7]), "=f"(f[8]), "=f"(f[9]), "=f"(f[10]),
              "=f"(f[11]), "=f"(f[12]), "=f"(f[13]), "=f"(f[14]), "=f"(f[15]), "=f"(g[0]), "=f"(g[1]), "=f"(g[2]), "=f"(g[3]), "=f"(g[4]), "=f"(g[5]),
              "=f"(g[6]), "=f"(g[7]), "=f"(g[8]), "=f"(g[9]), "=f"(g[10]), "=f"(g[11]), "=f"(g[12]), "=f"(g[13]), "=f"(g[14]), "=f"(g[15])
            : "r"(at + (uint32_t)nt), "r"(at + (uint32_t)(2 * nt))
            : "memory");
#pragma unroll
        for (int t = 0; t < 16; ++t) f[t] += g[t];
        uint32_t v[16];                                       // (not with the other two: forty-eight registers at a time were too many)
        tmem_ld16(at, v);
#pragma unroll
        for (int t = 0; t < 16; ++t) f[t] = __uint_as_float(v[t]) + f[t];
    }
}
// the sum of the legs so far: sixteen values of this thread, 512 bytes apart in shared memory
__device__ __forceinline__ void mm_add_run(uint32_t at, float (&f)[16]) {
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        float r;
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(at + (uint32_t)t * 512u) : "memory");
        f[t] += r;
    }
}
__device__ __forceinline__ void mm_store_run(uint32_t at, const float (&f)[16]) {
#pragma unroll
    for (int t = 0; t < 16; ++t) asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (uint32_t)t * 512u), "f"(f[t]) : "memory");
}
// 2-D tiled TMA load into this block's own shared memory: coordinates are (element along K, activation row).  CG = 2: `bar` may be
// the other block's of the pair.
template <int CG = 1>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    if (CG == 2) {
        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                     "l"(map), "r"(bar), "r"(c0), "r"(c1)
                     : "memory");
        return;
    }
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(map), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}
// coordinates (element along K, activation row, plane)
template <int CG = 1>
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    if (CG == 2) {
        asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
                     "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
                     : "memory");
        return;
    }
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(dst),
                 "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

// Sixteen two-bit codes -> eight words of two 16-bit floats 0 / +-2 (bittile_format.h).  The shifts are multiplications by
// values in registers: they run on the FMA pipe beside the ANDs on the ALU pipe.
__device__ __forceinline__ void mm_decode_word(uint32_t x, uint32_t m4, uint32_t m16, uint32_t* o) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        o[2 * p] = x & 0xC000C000u;
        o[2 * p + 1] = (x * m4) & 0xC000C000u;
        if (p < 3) x *= m16;
    }
}
__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

// Non-blocking probe of a barrier phase: unlike try_wait it never suspends the thread, so a spinning waiter
// sees the completion within one loop iteration.
__device__ __forceinline__ uint32_t mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
__device__ __forceinline__ bool bounded_spin(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    if (mbar_test_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (uint32_t it = 1;; ++it) {
        if (mbar_test_wait(bar, parity)) return true;
        if ((it & 63u) == 0) {
            if (*abort_flag) return false;
            if (clock64() - t0 > TLLM_WAIT_LIMIT_CLOCKS) {
                *abort_flag = 1;
                return false;
            }
        }
    }
}

// a wait for the first phase of a barrier at which other blocks arrive behind their writes to this one's shared memory (with a fence behind a wait that acquires
// for the block alone, 950 clocks)
__device__ __forceinline__ bool mm_wait_cluster(uint32_t bar, volatile int* abort_flag) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar)
            : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
        if (clock64() - t0 > TLLM_WAIT_LIMIT_CLOCKS) {
            *abort_flag = 1;
            return false;
        }
    }
}
// waiting roles are parked (bounded_wait): spinning ones took issue slots from the epilogue; only the thread that issues MMAs spins
#define MM_WAIT(bar, par)                             \
    do {                                                    \
        if (!bounded_wait((bar), (par), abort_flag)) goto done; \
    } while (0)
#define MM_SPIN(bar, par)                                       \
    do {                                                        \
        if (!bounded_spin((bar), (par), abort_flag)) goto done; \
    } while (0)
// ring position and the parity of its current round
#define MM_ADVANCE(idx, ph, n) \
    do {                       \
        if (++(idx) == (n)) {  \
            (idx) = 0;         \
            (ph) ^= 1u;        \
        }                      \
    } while (0)

// true in exactly one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// ---- clusters (split 2) ----------------------------------------------------------------------------------
__device__ __forceinline__ void mm_cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void mm_cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mm_cluster_sync() {
    mm_cluster_arrive();
    mm_cluster_wait();
}
// barriers made by this thread, for the other blocks' arrivals and for the TMA unit's
__device__ __forceinline__ void mm_fence_barriers() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// address of this block's shared location in block `rank`
__device__ __forceinline__ uint32_t mm_peer(uint32_t addr, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void mm_st_peer(uint32_t addr, float a, float b, float c, float d) {
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// An arrival at the barrier of a pair's first block: what it stands for is tensor memory, which the tcgen05 waits and fences before it
// have taken care of, so that nothing has to be released with it.  (With release.cluster it waited for the thread's other writes too: 2500 clocks.)
__device__ __forceinline__ void mm_arrive_first(uint32_t bar, uint32_t first) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(mm_peer(bar, first)) : "memory");
}
__device__ __forceinline__ void mm_arrive_peer(uint32_t bar) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }

// column (of the 32 of a quarter tile) that lane `lane` of tensor memory's quarter holds
__device__ __forceinline__ int mm_column(int lane) { return ((lane >> 1) & 1) * 16 + (lane & 1) * 8 + (lane >> 2); }

// a / d, inv = ceil(2^32 / d)
__host__ __device__ __forceinline__ uint32_t mm_inverse(uint32_t d) { return d == 1 ? 0u : 0xFFFFFFFFu / d + 1u; }
__device__ __forceinline__ int mm_div(int a, int d, uint32_t inv) {
    if (d == 1) return a;
    const uint32_t q = __umulhi((uint32_t)a, inv);
    return (int)(q * (uint32_t)d > (uint32_t)a ? q - 1u : q);
}
// first tile or unit of block or pair c of G
__device__ __forceinline__ int mm_share(const MmParams& p, int c, int G) { return c * p.share + mm_div(c * p.share_more, G, p.g_inv); }
// whose unit u is (split 1)
__device__ __forceinline__ int mm_owner(const MmParams& p, int u, int G, int total) {
    int c = min(G - 1, (int)((float)u * (float)G / (float)total));
    while (c + 1 < G && mm_share(p, c + 1, G) <= u) ++c;
    while (mm_share(p, c, G) > u) --c;
    return c;
}

// The segments of a block's unit range [u0, u1): one per output tile it touches; the first and the last, which other blocks may
// share, come first.
struct MmSegs {
    int u0, u1, KBU, t0, n;
    __device__ __forceinline__ MmSegs(int a, int b, int kbu, uint32_t inv) : u0(a), u1(b), KBU(kbu), t0(mm_div(a, kbu, inv)), n(mm_div(b - 1, kbu, inv) - t0 + 1) {}
    // segment i: its tile, the tile's units [ua, ub), and which of the block's two slots a partial sum goes to
    __device__ __forceinline__ void get(int i, int& tile, int& ua, int& ub, int& slot) const {
        const int j = i < 2 ? (i ? n - 1 : 0) : i - 1;
        tile = t0 + j;
        const int f = tile * KBU;
        ua = max(u0 - f, 0), ub = min(u1 - f, KBU);
        slot = j ? 1 : 0;
    }
};

// the units of those segments one after the other, for the thread that loads bit tiles
struct MmBitsRange {
    const MmSegs& segs;
    const MmParams& p;
    int cg, member, i = 0, ku = 0, ub = 0, row0 = 0;
    __device__ __forceinline__ MmBitsRange(const MmSegs& s, const MmParams& q, int c, int m) : segs(s), p(q), cg(c), member(m) { open(); }
    __device__ __forceinline__ bool left() const { return i < segs.n; }
    __device__ __forceinline__ void next() {
        if (++ku == ub && ++i < segs.n) open();
    }
    __device__ __forceinline__ void open() {
        int tile, slot;
        segs.get(i, tile, ku, ub, slot);
        row0 = (mm_div(tile, p.m_tiles, p.mt_inv) * cg + member) * 8;
    }
};

// ---- results: sixteen rows m .. m+15 of column n, called by whole warps.  The kind of store is looked at once per sixteen
// rows and the stores of a kind are straight-line code: with the choice inside the loop a store took 220 to 390 clocks, and a
// tile of 128 rows spent longer in its epilogue than in its MMAs.
template <bool BF16>
__device__ __forceinline__ unsigned short mm_16bit(float v) {
    return BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
}
template <bool BF16>
__device__ __forceinline__ void mm_emit_16(const MmParams& p, const float (&f)[16], int n, int m) {
    unsigned short* y = (unsigned short*)p.Y + (size_t)n * p.y_step_n + (size_t)m * p.y_step_m;
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        if (n < p.N && m + t < p.M) *y = mm_16bit<BF16>(f[t] * p.scale);
        y += p.y_step_m;
    }
}
// the lanes of neighbouring columns trade one value per pair of rows, so that every lane writes two adjacent columns of one row
template <bool BF16>
__device__ __forceinline__ void mm_emit_pairs(const MmParams& p, const float (&f)[16], int n, int m) {
    const bool odd = n & 1;
    uint32_t* y = (uint32_t*)((unsigned short*)p.Y + (size_t)(m + (odd ? 1 : 0)) * p.y_step_m + (n & ~1));
#pragma unroll
    for (int t = 0; t < 16; t += 2) {
        const float got = __shfl_xor_sync(0xffffffffu, odd ? f[t] : f[t + 1], 4);
        const float lo = (odd ? got : f[t]) * p.scale, hi = (odd ? f[t + 1] : got) * p.scale;
        uint32_t w;
        if (BF16) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
            w = *reinterpret_cast<const uint32_t*>(&h);
        } else {
            const __half2 h = __floats2half2_rn(lo, hi);
            w = *reinterpret_cast<const uint32_t*>(&h);
        }
        if (m + t + (odd ? 1 : 0) < p.M) *y = w;
        y += p.y_step_m;                       // two rows of 16-bit values = y_step_m words
    }
}
template <int OUT>
__device__ __forceinline__ void mm_emit(const MmParams& p, const float (&f)[16], int n, int m) {
    uint32_t* y = (uint32_t*)p.Y + (size_t)n * p.y_step_n + (size_t)m * p.y_step_m;
    if constexpr (OUT == MM_OUT_F16 || OUT == MM_OUT_BF16) mm_emit_16<OUT == MM_OUT_BF16>(p, f, n, m);
    else if constexpr (OUT == MM_OUT_F16_PAIRS || OUT == MM_OUT_BF16_PAIRS) mm_emit_pairs<OUT == MM_OUT_BF16_PAIRS>(p, f, n, m);
    else if constexpr (OUT == MM_OUT_F32 || OUT == MM_OUT_I32) {
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const uint32_t w = OUT == MM_OUT_F32 ? __float_as_uint(f[t] * p.scale) : (uint32_t)(int)(f[t] * 0.5f);
            if (n < p.N && m + t < p.M) *y = w;
            y += p.y_step_m;
        }
    } else {
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = OUT == MM_OUT_F32_COL4 ? __float_as_uint(f[t + j] * p.scale) : (uint32_t)(int)(f[t + j] * 0.5f);
            if (n < p.N && m + t + 4 <= p.M) *(uint4*)(y + t) = make_uint4(w[0], w[1], w[2], w[3]);
            else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (n < p.N && m + t + j < p.M) y[t + j] = w[j];
            }
        }
    }
}
// An fp32 value as bf16 values of eight significant bits: the upper half of `w` is the next one, and what is left after it is exact.  Inf
// and NaN are the first value, with zeros behind them (Inf - Inf would be NaN).
__device__ __forceinline__ uint32_t mm_first_piece(uint32_t w) { return (w & 0x7FFFFFFFu) > 0x7F800000u ? w | 0x00400000u : w; }
__device__ __forceinline__ uint32_t mm_next_piece(uint32_t w) {
    return (w & 0x7F800000u) == 0x7F800000u ? 0u : __float_as_uint(__uint_as_float(w) - __uint_as_float(w & 0xFFFF0000u));
}
// Gate and up columns sit in neighbouring lanes: the even one takes row t, the odd one row t + 1.
template <int OUT>
__device__ __forceinline__ void mm_emit_silu(const MmParams& p, const float (&f)[16], int n, int m) {
    const bool odd = n & 1;
    const int row = m + (odd ? 1 : 0);
    const size_t at = (size_t)row * p.y_ld + (n >> 1);
    float y[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const float got = __shfl_xor_sync(0xffffffffu, odd ? f[2 * t] : f[2 * t + 1], 4);
        y[t] = silu_mul((odd ? got : f[2 * t]) * p.scale, (odd ? f[2 * t + 1] : got) * p.scale2);
    }
    const bool ok = (n | 1) < p.N;
    const size_t step = 2 * (size_t)p.y_ld;
    if constexpr (OUT == MM_OUT_F32) {
#pragma unroll
        for (int t = 0; t < 8; ++t)
            if (ok && row + 2 * t < p.M) ((float*)p.Y)[at + t * step] = y[t];
    } else if constexpr (OUT == MM_OUT_PLANES) {
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            uint32_t w = mm_first_piece(__float_as_uint(y[t]));
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) {
                if (ok && row + 2 * t < p.M) ((unsigned short*)p.Y)[(size_t)pl * p.plane_y + at + t * step] = (unsigned short)(w >> 16);
                w = mm_next_piece(w);
            }
        }
    } else {
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const unsigned short w = mm_16bit<OUT == MM_OUT_BF16>(y[t]);
            if (ok && row + 2 * t < p.M) ((unsigned short*)p.Y)[at + t * step] = w;
        }
    }
}

// Which of sixteen sums are not finite: none, nearly always, and then one multiply-add each is all it costs.
__device__ __forceinline__ uint32_t mm_not_finite(const MmParams& p, const float (&f)[16]) {
    if (p.finite == 0) return 0u;
    float z[4] = {};
#pragma unroll
    for (int t = 0; t < 16; ++t) z[t & 3] = fmaf(f[t], 0.f, z[t & 3]);      // 0, or NaN from the first Inf or NaN on
    uint32_t bad = 0u;
    if (z[0] + z[1] + z[2] + z[3] != 0.f)
#pragma unroll
        for (int t = 0; t < 16; ++t) bad |= finite_sum(f[t]) ? 0u : 1u << t;
    return bad;
}
__device__ __noinline__ float mm_column_sum(const MmParams& p, int n, int m) {
    return column_sum(p.bits, n, p.K, p.KB, p.finite == 2, [&](int k) {
        float v = 0.f;
        for (int pl = p.P - 1; pl >= 0; --pl) {
            const unsigned short x = __ldcg(p.X + (size_t)pl * p.plane_x + (size_t)m * p.ld_x + k);
            v += p.bf16 ? __bfloat162float(__ushort_as_bfloat16(x)) : __half2float(__ushort_as_half(x));
        }
        return v;
    });
}
// Stores those of rows m .. m + 15 of column n again, behind the stores of the whole warp.  Of a gate and an up column either may be the
// one, so both are summed.
__device__ __noinline__ void mm_store_again(const MmParams& p, uint32_t bad, int n, int m) {
    const bool half = p.out == MM_OUT_F16 || p.out == MM_OUT_F16_PAIRS, bf16 = p.out == MM_OUT_BF16 || p.out == MM_OUT_BF16_PAIRS;
    for (; bad; bad &= bad - 1) {
        const int row = m + __ffs(bad) - 1;
        if (n >= p.N || row >= p.M) continue;
        float y;
        size_t at;
        if (p.epilogue == 0) y = mm_column_sum(p, n, row) * (2.f * p.scale), at = (size_t)n * p.y_step_n + (size_t)row * p.y_step_m;
        else {
            if ((n | 1) >= p.N) continue;
            y = silu_mul(mm_column_sum(p, n & ~1, row) * (2.f * p.scale), mm_column_sum(p, n | 1, row) * (2.f * p.scale2));
            at = (size_t)row * p.y_ld + (n >> 1);
        }
        if (p.out == MM_OUT_PLANES) {
            uint32_t w = mm_first_piece(__float_as_uint(y));
            for (int pl = 0; pl < 3; ++pl, w = mm_next_piece(w)) ((unsigned short*)p.Y)[(size_t)pl * p.plane_y + at] = (unsigned short)(w >> 16);
        } else store_out(p.Y, half ? TLLM_F16 : bf16 ? TLLM_BF16 : TLLM_F32, at, y);
    }
}

// runs `f` with the kind of store as a type
template <typename F>
__device__ __forceinline__ void mm_with_out(const MmParams& p, F f) {
    if (p.epilogue == 0) {
        switch (p.out) {
            case MM_OUT_F32: f(std::integral_constant<int, MM_OUT_F32>{}, std::false_type{}); break;
            case MM_OUT_I32: f(std::integral_constant<int, MM_OUT_I32>{}, std::false_type{}); break;
            case MM_OUT_F16: f(std::integral_constant<int, MM_OUT_F16>{}, std::false_type{}); break;
            case MM_OUT_BF16: f(std::integral_constant<int, MM_OUT_BF16>{}, std::false_type{}); break;
            case MM_OUT_F16_PAIRS: f(std::integral_constant<int, MM_OUT_F16_PAIRS>{}, std::false_type{}); break;
            case MM_OUT_BF16_PAIRS: f(std::integral_constant<int, MM_OUT_BF16_PAIRS>{}, std::false_type{}); break;
            case MM_OUT_F32_COL4: f(std::integral_constant<int, MM_OUT_F32_COL4>{}, std::false_type{}); break;
            default: f(std::integral_constant<int, MM_OUT_I32_COL4>{}, std::false_type{});
        }
    } else {
        switch (p.out) {
            case MM_OUT_F32: f(std::integral_constant<int, MM_OUT_F32>{}, std::true_type{}); break;
            case MM_OUT_F16: f(std::integral_constant<int, MM_OUT_F16>{}, std::true_type{}); break;
            case MM_OUT_BF16: f(std::integral_constant<int, MM_OUT_BF16>{}, std::true_type{}); break;
            default: f(std::integral_constant<int, MM_OUT_PLANES>{}, std::true_type{});
        }
    }
}

// Tensor memory: two sets of accumulators, and behind them the ring of expanded units, 64 columns each: four, or two beside
// accumulators of more than 128 columns.
__host__ __device__ __forceinline__ uint32_t mm_a_units_log(uint32_t acc_cols) { return acc_cols <= 128 ? 2u : 1u; }

// PAIRS: pairs of blocks (CG = 2) in clusters of several; an instance of its own, since with the place of a pair in its cluster as a variable the others took
// 3 to 7 % longer (512 rows of fp16 on 2048 x 16384 34.5 us, 32.4 with constants)
template <int CG, bool PAIRS = false>
__global__ void __launch_bounds__(MM_THREADS, 1) mma_spmm_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap wmap,
                                                                 const __grid_constant__ MmParams p) {
    extern __shared__ unsigned char mm_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // ---- the unit range of this block or pair ------------------------------------------------------------
    const int G = (int)gridDim.x / CG, cta = (int)blockIdx.x / CG, member = CG == 2 ? (int)blockIdx.x & 1 : 0;
    const int KBU = p.KBU, KB = p.KB, tiles = (p.n_tiles + CG - 1) / CG * p.m_tiles;
    const int total = tiles * KBU;
    const bool clustered = PAIRS || (CG == 1 && p.split == 2);
    const int C = clustered ? p.cluster : 1, rank = clustered ? cta & (C - 1) : 0;
    const uint32_t first = PAIRS ? (uint32_t)(rank * CG) : 0u, both = 3u << first;              // the pair's blocks in the cluster
    int u0, u1;
    if (clustered) u0 = (cta >> p.cluster_log) * KBU, u1 = u0 + (KBU * (rank + 1) >> p.cluster_log), u0 += KBU * rank >> p.cluster_log;
    else {
        u0 = mm_share(p, cta, G), u1 = mm_share(p, cta + 1, G);
        if (!p.split) u0 *= KBU, u1 *= KBU;
    }
    if (u0 >= u1) return;                  // never in a cluster: KBU >= C
    const MmSegs segs(u0, u1, KBU, p.kbu_inv);

    // ---- shared memory ---------------------------------------------------------------------------------
    const uint32_t raw0 = smem_u32(mm_smem);
    const uint32_t base = (raw0 + 1023u) & ~1023u;                 // swizzled tiles need 1024-byte alignment
    const uint32_t SB = (uint32_t)p.SB, R = MM_RAW_UNITS;
    const int Nt = p.Nt;
    const uint32_t acc_cols = (uint32_t)(p.P * Nt), b_slice = acc_cols / CG * 128u, b_unit = MM_UK * b_slice;
    const uint32_t b_base = base, r_base = b_base + SB * b_unit;
    const uint32_t bar_base = r_base + R * MM_UNIT_BYTES, part_base = bar_base + 512u;      // part_base: the cluster's parts, [block][rows / 16][4][128] x 16 bytes
    const uint32_t run_base = part_base + (clustered ? (uint32_t)(C * ((Nt / 16 + C - 1) / C)) * 8192u : 0u);      // fp32: the sum of the legs so far, [row][128]
    const uint32_t a_log = mm_a_units_log(acc_cols), a_mask = (1u << a_log) - 1u;
    // Where the ring of expanded units has two places, each of their slices has barriers of its own, so that it is filled again while the
    // other three are multiplied (5120 x 15360, 2048 rows in tiles of 192: 198 us, 227 with one pair of barriers a unit); with four places
    // there is time enough, and fewer barriers are faster (2048 x 8192, 32 rows: 8.8 us against 9.6).
    const uint32_t fine = a_log == 1u ? 1u : 0u;
    volatile int* flags = (volatile int*)(mm_smem + (bar_base - raw0) + 8 * 60);   // [0] tensor-memory address, [1] abort
    volatile int* abort_flag = flags + 1;
#define A_FULL(s) (bar_base + 8u * (uint32_t)(s))
#define A_EMPTY(s) (bar_base + 8u * (8u + (uint32_t)(s)))
#define B_FULL(s) (bar_base + 8u * (16u + (uint32_t)(s)))
#define B_EMPTY(s) (bar_base + 8u * (24u + (uint32_t)(s)))
#define RAW_FULL(r) (bar_base + 8u * (32u + (uint32_t)(r)))
#define RAW_EMPTY(r) (bar_base + 8u * (40u + (uint32_t)(r)))
#define ACC_FULL(a) (bar_base + 8u * (48u + (uint32_t)(a)))
#define ACC_EMPTY(a) (bar_base + 8u * (50u + (uint32_t)(a)))
#define PART_FULL(q) (bar_base + 8u * (52u + (uint32_t)(q)))

    // Start: warp 0 has the first bit tiles on their way as soon as their barriers exist, warp 1 takes tensor memory, warps 2 and 3 make the other
    // barriers, a thread each, and one barrier of the block or cluster ends it.  (One thread making sixty barriers, then tensor memory, then the first copies took
    // 4000 to 4600 clocks to here, 2500 in mma_units4_kernel, and 2800 more to the first expanded slice; with 64-bit divisions gone as well, and the
    // cluster waited for later, us before / now: 24 rows of fp32 on 2048 x 2048 10.4 / 9.4, 256 on 2048 x 8192 24.8 / 24.0, 256 of fp16 on
    // 512 x 3000 6.4 / 6.1.)
    MmBitsRange load(segs, p, CG, member);
    if (warp == 0) {
        if (lane < 16) mbar_init(RAW_FULL(lane), lane < 8 ? 1 : 8);             // RAW_EMPTY: half of the decoder warps
        mm_fence_barriers();
        __syncwarp();
        // The weights do not depend on the preceding kernel.  A tile's eight groups of sixteen columns are eight streams along K; the tensor map sees them
        // as eight rows, and one box of 8 x 512 bytes is a unit; past the end of K it is filled with zeros, which count.  (Eight bulk copies
        // instead, one per lane, took 820 clocks a unit to issue.)
        if (!p.wait_bits && elect_one())
            for (uint32_t r = 0; r < R && load.left(); ++r, load.next()) {
                mbar_expect_tx(RAW_FULL(r), MM_UNIT_BYTES);
                tma_load_2d(r_base + r * MM_UNIT_BYTES, &wmap, load.ku * (MM_UK * 64), load.row0, RAW_FULL(r));
            }
        __syncwarp();
    } else if (warp == 1) {
        tmem_alloc<CG>(smem_u32((const void*)flags), 512);
    } else if (warp < 4) {
        const int i = tid - 64;                                                // the order of the names above
        if (i < 60 && (i < 32 || i >= 48)) {
            const int n = i < 8 ? (fine ? 4 : 8) * CG                          // the decoder warps of a slice or unit (of a pair: at the first block)
                        : i < 16 ? 1                                           // tcgen05.commit
                        : i < 24 ? 1                                           // the TMA thread's expect_tx arrival
                        : i < 50 ? 1                                           // tcgen05.commit
                        : i < 52 ? 8 * CG                                      // the epilogue warps
                                 : max(C - 1, 1);                              // the same warp of the other blocks
            mbar_init(bar_base + 8u * (uint32_t)i, (uint32_t)n);
        }
        if (i == 63) {
            flags[1] = 0;
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap) : "memory");
        }
        mm_fence_barriers();
    }
    // The other blocks' barriers are waited for where they are needed (join): blocks of a cluster start up to 1300 clocks apart, and the first tiles are expanded
    // meanwhile.
    if (CG == 2 || clustered) mm_cluster_arrive();
    bool joined = CG == 1 && !clustered;
    const auto join = [&] {
        if (!joined) mm_cluster_wait(), joined = true;
    };
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = (uint32_t)flags[0];
    const uint32_t a_base = tmem + (a_log == 2u ? 256u : 384u);
    pdl_launch_dependents();

    // Every role walks the same list of segments.  The producers and the issuer are one thread each: with the whole warp in the loop and a
    // lane elected per block of instructions, eight MMAs and two commits took 220 clocks to issue, by one thread 105.
    if (warp == 0) {
        // ---- bit-tile producer, behind the first round of its ring
        if (elect_one()) {
            uint32_t r = 0, rph = 0;
            if (p.wait_bits) pdl_wait();
            else rph = 1u;
            for (; load.left(); load.next()) {
                MM_WAIT(RAW_EMPTY(r), rph ^ 1u);
                mbar_expect_tx(RAW_FULL(r), MM_UNIT_BYTES);
                tma_load_2d(r_base + r * MM_UNIT_BYTES, &wmap, load.ku * (MM_UK * 64), load.row0, RAW_FULL(r));
                MM_ADVANCE(r, rph, R);
            }
        }
    } else if (warp == 2) {
        // ---- activation producer: a unit is two TMA boxes (all planes of a slice each) on one barrier
        if (CG == 2) join();
        if (elect_one()) {
            pdl_wait();
            uint32_t b = 0, bph = 0;
            const int rows = Nt / CG;                             // of a pair each block fetches half of the rows, for the first block's barrier
            for (int i = 0; i < segs.n; ++i) {
                int tile, ua, ub, sl;
                segs.get(i, tile, ua, ub, sl);
                const int row0 = (tile - mm_div(tile, p.m_tiles, p.mt_inv) * p.m_tiles) * Nt + member * rows;
                for (int ku = ua; ku < ub; ++ku) {
                    const bool two = ku * MM_UK + 1 < KB;
                    MM_WAIT(B_EMPTY(b), bph ^ 1u);
                    const uint32_t full = CG == 1 ? B_FULL(b) : mm_peer(B_FULL(b), first), to = b_base + b * b_unit;
                    if (member == 0) mbar_expect_tx(B_FULL(b), (two ? 2u : 1u) * CG * b_slice);
                    // (three planes as three boxes a slice would be six instructions to issue; one plane as a box of three dimensions
                    // measured 4 % slower than one of two)
                    if (p.P == 1) {
                        tma_load_2d<CG>(to, &tmap, ku * (MM_UK * MM_TILE_K), row0, full);
                        if (two) tma_load_2d<CG>(to + b_slice, &tmap, ku * (MM_UK * MM_TILE_K) + MM_TILE_K, row0, full);
                    } else {
                        tma_load_3d<CG>(to, &tmap, ku * (MM_UK * MM_TILE_K), row0, 0, full);
                        if (two) tma_load_3d<CG>(to + b_slice, &tmap, ku * (MM_UK * MM_TILE_K) + MM_TILE_K, row0, 0, full);
                    }
                    MM_ADVANCE(b, bph, SB);
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer; of a pair the first block's.  Nothing but the MMAs' own time lies between two of them as long as the next unit's
        // operands are there: the tensor core has some in its queue while this thread looks.
        if (CG == 2) join();
        if (member == 0 && elect_one()) {
            const uint32_t idesc = p.idesc, b_lo0 = (b_base >> 4) & 0x3FFFu;
            uint32_t u = 0, sb = 0, sbph = 0, a = 0, aph = 0;
            for (int i = 0; i < segs.n; ++i) {
                int tile, ua, ub, sl, left = 0;
                segs.get(i, tile, ua, ub, sl);
                uint32_t d = 0, acc = 0;
                for (int ku = ua; ku < ub; ++ku, ++u) {
                    const uint32_t sa = u & a_mask, saph = (u >> a_log) & 1u;
                    MM_SPIN(A_FULL(sa << fine), saph);
                    MM_SPIN(B_FULL(sb), sbph);
                    if (left == 0) {                             // a leg starts
                        MM_SPIN(ACC_EMPTY(a), aph ^ 1u);
                        d = tmem + a * acc_cols, acc = 0, left = min(p.leg, ub - ku);
                    }
                    tc_fence_after();
                    const uint32_t at = a_base + sa * (MM_UK * 32u), b_lo = b_lo0 + sb * (b_unit >> 4);
                    // 16 values = 8 columns of A, 32 bytes = 2 descriptor address units of B
#pragma unroll
                    for (uint32_t k4 = 0; k4 < MM_TILE_K / 16; ++k4) umma_f16_ts<CG>(d, at + 8u * k4, b_lo + 2u * k4, idesc, k4 == 0 ? acc : 1u);
                    if (fine) {
                        umma_commit<CG>(A_EMPTY(2u * sa), both);
                        MM_SPIN(A_FULL(2u * sa + 1u), saph);
                        tc_fence_after();
                    }
                    if (ku * MM_UK + 1 < KB) {
#pragma unroll
                        for (uint32_t k4 = 0; k4 < MM_TILE_K / 16; ++k4) umma_f16_ts<CG>(d, at + 32u + 8u * k4, b_lo + (b_slice >> 4) + 2u * k4, idesc, 1u);
                    }
                    umma_commit<CG>(A_EMPTY(fine ? 2u * sa + 1u : sa), both);
                    umma_commit<CG>(B_EMPTY(sb), both);
                    MM_ADVANCE(sb, sbph, SB);
                    acc = 1;
                    if (--left == 0) {
                        umma_commit<CG>(ACC_FULL(a), both);
                        MM_ADVANCE(a, aph, 2u);
                    }
                }
            }
        }
    } else if (warp >= 12) {
        // ---- decoders: eight warps take the even units and eight the odd ones, and a warp expands 32 columns of W of one slice into its 32
        // lanes of tensor memory.  Lane 4g + u holds column 16 * (u >> 1) + 8 * (u & 1) + g of them (see mm_column).  The values are in
        // registers before the place in the ring is free: from there on they are a store away.
        const int q = warp & 3, h = ((warp - 12) >> 2) & 1;
        const uint32_t mine = (uint32_t)(warp - 12) >> 3;
        const uint32_t g = (uint32_t)lane >> 2, u = (uint32_t)lane & 3u;
        const uint32_t raw_lane = r_base + (uint32_t)(2 * q + (u >> 1)) * 512u;
        const uint32_t a_lane = a_base + ((uint32_t)(q * 32) << 16) + (uint32_t)h * 32u;
        uint32_t m4, m16;
        asm volatile("mov.b32 %0, %2;\n\tmov.b32 %1, %3;" : "=r"(m4), "=r"(m16) : "r"(p.mul4), "r"(p.mul16));
        uint32_t n = 0;                                       // units so far
        if (CG == 2) join();                                  // (in the loop, behind the first unit's values, it cost every unit 1 %)
        for (int i = 0; i < segs.n; ++i) {
            int tile, ua, ub, sl;
            segs.get(i, tile, ua, ub, sl);
            for (int ku = ua; ku < ub; ++ku, ++n) {
                if ((n & 1u) != mine) continue;
                const int slice = ku * MM_UK + h;
                const uint32_t r = n & (R - 1u), at = raw_lane + r * MM_UNIT_BYTES, sa = n & a_mask, bar = fine ? 2u * sa + (uint32_t)h : sa;
                MM_WAIT(RAW_FULL(r), (n / R) & 1u);
                uint32_t w[4] = {};
                if ((slice | 1) < KB) {
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        uint32_t lo, hi;
                        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(at + (uint32_t)mm_chunk((int)g, t) * 16u + (uint32_t)h * 8u) : "memory");
                        w[t] = u & 1u ? hi : lo;
                    }
                } else if (slice < KB) {                      // an odd last slice
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w[t]) : "r"(at + (4u * g + (uint32_t)t) * 8u + (u & 1u) * 4u) : "memory");
                }
                uint32_t o[32];
#pragma unroll
                for (int t = 0; t < 4; ++t) mm_decode_word(w[t], m4, m16, o + 8 * t);
                __syncwarp();
                if (lane == 0) mbar_arrive(RAW_EMPTY(r));
                MM_WAIT(A_EMPTY(bar), ((n >> a_log) & 1u) ^ 1u);
                if (slice < KB) {
                    tc_fence_after();
                    tmem_st32(a_lane + sa * (MM_UK * 32u), o);
                    tmem_wait_st();
                    tc_fence_before();
                }
                __syncwarp();
                if (lane == 0) {
                    if (CG == 1) mbar_arrive(A_FULL(bar));
                    else mm_arrive_first(A_FULL(bar), first);
                }
            }
        }
    } else if (warp >= 4) {
        // ---- epilogue: a warp may read the 32 tensor-memory lanes selected by warp % 4; of the sixteens of rows it has every other one (of
        // those that a block of a cluster writes, too)
        const int q = warp & 3, odd = (warp >> 2) - 1, nl = q * 32 + lane, ncol = q * 32 + mm_column(lane);
        join();
        pdl_wait();
        uint32_t a = 0, aph = 0;
        const auto acc_free = [&](uint32_t bar) {
            if (CG == 1) mbar_arrive(bar);
            else mm_arrive_first(bar, first);
        };
        // Columns of D: rows [0, Nt / 2) of X of each plane, which a pair's first block holds, and then the other's.
        const int rows = Nt / CG;
        const auto column = [&](int c16) { return (uint32_t)(CG == 2 && c16 >= rows ? c16 + (p.P - 1) * rows : c16); };
        for (int i = 0; i < segs.n; ++i) {
            int tile, ua, ub, sl;
            segs.get(i, tile, ua, ub, sl);
            const int ct = mm_div(tile, p.m_tiles, p.mt_inv), mt = tile - ct * p.m_tiles, nt = ct * CG + member;      // nt: this block's tile of 128 columns; the last of an odd number has no pair
            const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16), run = run_base + (uint32_t)nl * 4u;
            // all legs but the last join the sum in shared memory
            bool legs = false;
            for (int left = ub - ua; left > p.leg; left -= p.leg) {
                MM_WAIT(ACC_FULL(a), aph);
                tc_fence_after();
                for (int c16 = 16 * odd; c16 < Nt; c16 += 32) {
                    float f[16];
                    mm_load16(lanes + a * acc_cols + column(c16), rows, p.P, f);
                    if (legs) mm_add_run(run + (uint32_t)c16 * 512u, f);
                    mm_store_run(run + (uint32_t)c16 * 512u, f);
                }
                legs = true;
                tc_fence_before();
                __syncwarp();
                if (lane == 0) acc_free(ACC_EMPTY(a));
                MM_ADVANCE(a, aph, 2u);
            }
            MM_WAIT(ACC_FULL(a), aph);
            tc_fence_after();
            const bool full = ua == 0 && ub == KBU;
            const uint32_t taddr = lanes + a * acc_cols;
            const size_t slot_floats = (size_t)MM_TILE_N * Nt;
            float* slot = p.partial + (size_t)(2 * (cta * CG + member) + sl) * slot_floats + nl * 4;
            const int n = nt * MM_TILE_N + ncol;
            // sixteen accumulator columns (rows of X) of this lane's column of W
            auto load16 = [&](int c16, float (&f)[16]) {
                mm_load16(taddr + column(c16), rows, p.P, f);
                if (legs) mm_add_run(run + (uint32_t)c16 * 512u, f);
            };
            auto finish16 = [&](auto out, auto silu, const float (&f)[16], int n, int m) {
                const uint32_t bad = mm_not_finite(p, f);
                if constexpr (decltype(silu)::value) mm_emit_silu<decltype(out)::value>(p, f, n, m);
                else mm_emit<decltype(out)::value>(p, f, n, m);
                if (__any_sync(0xffffffffu, bad)) {
                    __syncwarp();
                    mm_store_again(p, bad, n, m);
                }
            };
            bool sum = false;                    // this block adds up the parts of a shared tile
            int cf = 0, cl = 0;
            if (clustered) {
                // sixteen c of the rows is block c % C's to write
                const int sixteens = Nt / 16, own = (sixteens + C - 1) / C;
                for (int c = 0; c < sixteens; ++c) {
                    const int o = c % C;
                    if (o == rank || ((c / C) & 1) != odd) continue;
                    float f[16];
                    load16(16 * c, f);
                    const uint32_t to = mm_peer(part_base + (uint32_t)(((rank * own + c / C) * 4) * 128 + nl) * 16u, (uint32_t)(o * CG + member));
#pragma unroll
                    for (int t = 0; t < 4; ++t) mm_st_peer(to + (uint32_t)t * 2048u, f[4 * t], f[4 * t + 1], f[4 * t + 2], f[4 * t + 3]);
                }
                __syncwarp();
                if (lane < C && lane != rank && lane < sixteens) mm_arrive_peer(mm_peer(PART_FULL(4 * odd + q), (uint32_t)(lane * CG + member)));
                if (rank < sixteens) {
                    if (!mm_wait_cluster(PART_FULL(4 * odd + q), abort_flag)) goto done;
                    mm_with_out(p, [&](auto out, auto silu) {
                        uint32_t at0 = part_base + (uint32_t)nl * 16u + (uint32_t)odd * 8192u;
                        for (int c = rank + odd * C; c < sixteens; c += 2 * C, at0 += 16384u) {
                            float f[16];
                            load16(16 * c, f);                          // its own part, then the others in block order
                            uint32_t at = at0;
#pragma unroll 1
                            for (int cc = 0; cc < C; ++cc, at += (uint32_t)own * 8192u)
                                if (cc != rank) {
#pragma unroll
                                    for (int t = 0; t < 4; ++t) {
                                        const uint4 x = ld_shared_v4(at + (uint32_t)t * 2048u);
                                        f[4 * t] += __uint_as_float(x.x), f[4 * t + 1] += __uint_as_float(x.y), f[4 * t + 2] += __uint_as_float(x.z), f[4 * t + 3] += __uint_as_float(x.w);
                                    }
                                }
                            if (CG == 1 || nt < p.n_tiles) finish16(out, silu, f, n, mt * Nt + 16 * c);
                        }
                    });
                }
            } else if (!full && (CG == 1 || nt < p.n_tiles)) {
                // The last of the blocks that share this tile to arrive adds the partial sums, in block order.  Each epilogue warp owns 32
                // columns of the tile and runs the hand-over for them by itself.  The last block's own part stays in tensor memory;
                // a block that finds all the others there already does not even write it.
                cf = mm_owner(p, tile * KBU, G, total), cl = mm_owner(p, tile * KBU + KBU - 1, G, total);
                unsigned int* ctr = p.counters + ((size_t)nt * p.m_tiles + mt) * 4 + q;
                const unsigned int others = (unsigned int)(cl - cf);
                const uint32_t field = 16u * (uint32_t)odd;      // the two warps of a column count in halves of one word
                unsigned int there = 0;
                if (lane == 0) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(there) : "l"(ctr) : "memory");
                sum = (__shfl_sync(0xffffffffu, there, 0) >> field & 0xFFFFu) == others;
                if (!sum) {
                    for (int c16 = 16 * odd; c16 < Nt; c16 += 32) {
                        float f[16];
                        load16(c16, f);
#pragma unroll
                        for (int t = 0; t < 16; t += 4) __stcg((float4*)(slot + (size_t)(c16 + t) * MM_TILE_N), make_float4(f[t], f[t + 1], f[t + 2], f[t + 3]));
                    }
                    __threadfence();
                    __syncwarp();
                    if (lane == 0) there = atomicAdd(ctr, 1u << field);
                    sum = (__shfl_sync(0xffffffffu, there, 0) >> field & 0xFFFFu) == others;
                }
                if (sum) {
                    if (lane == 0) atomicAnd(ctr, ~(0xFFFFu << field));
                    __threadfence();
                }
            }
            if (!clustered && (full || sum) && (CG == 1 || nt < p.n_tiles)) {
                // A part lies in its block's slot 0, except that the first block may have come from an earlier tile.
                const float* part0 = p.partial + (size_t)(2 * (cf * CG + member) + (!full && mm_share(p, cf, G) >= tile * KBU ? 0 : 1)) * slot_floats + nl * 4;
                const float* rest = p.partial + (size_t)(2 * ((cf + 1) * CG + member)) * slot_floats + nl * 4;
                mm_with_out(p, [&](auto out, auto silu) {
                    for (int c16 = 16 * odd; c16 < Nt; c16 += 32) {
                        float f[16];
                        if (full) load16(c16, f);
                        else {
#pragma unroll
                            for (int t = 0; t < 16; ++t) f[t] = 0.f;
                            const float* ps = part0 + (size_t)c16 * MM_TILE_N;
                            for (int cc = cf; cc <= cl; ++cc) {
                                if (cc == cta) {
                                    float mine[16];
                                    load16(c16, mine);
#pragma unroll
                                    for (int t = 0; t < 16; ++t) f[t] += mine[t];
                                } else {
                                    float4 x[4];
#pragma unroll
                                    for (int t = 0; t < 4; ++t) x[t] = __ldcg((const float4*)(ps + (size_t)(4 * t) * MM_TILE_N));
#pragma unroll
                                    for (int t = 0; t < 4; ++t) f[4 * t] += x[t].x, f[4 * t + 1] += x[t].y, f[4 * t + 2] += x[t].z, f[4 * t + 3] += x[t].w;
                                }
                                ps = rest + (size_t)(cc - cf) * 2 * CG * slot_floats + (size_t)c16 * MM_TILE_N;
                            }
                        }
                        finish16(out, silu, f, n, mt * Nt + c16);
                    }
                });
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) acc_free(ACC_EMPTY(a));
            MM_ADVANCE(a, aph, 2u);
        }
    }
done:
    __syncwarp();
    join();
    tc_fence_before();
    if (CG == 2) mm_cluster_sync();        // the pair's MMAs read both blocks' shared and tensor memory
    else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<CG>(tmem, 512);
    }
    if (tid == 0 && flags[1]) atomicExch(p.status, MM_ERR_WAIT);
    if (clustered) mm_cluster_sync();      // nobody leaves while the others may still write to its shared memory
#undef A_FULL
#undef A_EMPTY
#undef B_FULL
#undef B_EMPTY
#undef RAW_FULL
#undef RAW_EMPTY
#undef ACC_FULL
#undef ACC_EMPTY
#undef PART_FULL
}

// ---- activations as planes of 16-bit values for the kernel above: rows of k_pad values, zero beyond K ------------------
struct StageParams {
    const void* X;
    unsigned short* out;      // [planes][M][k_pad]
    int x_dtype, x_layout, x_ld;
    int M, K, k_pad;
    bool late;                // neither X nor `out` has to do with the preceding kernel: it is waited for at the end
};
// eight consecutive values of one row -> 16 bytes of each plane
template <int XT>
__device__ __forceinline__ void stage_eight(const StageParams& p, const uint32_t (&w)[8], int m, int k) {
    constexpr int PL = XT == TLLM_F32 ? 3 : 1;
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = XT == TLLM_F32 ? mm_first_piece(w[i]) : w[i];
#pragma unroll
    for (int pl = 0; pl < PL; ++pl) {
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (XT == TLLM_F32) o[i] = __byte_perm(v[2 * i], v[2 * i + 1], 0x7632);       // eight significant bits of each, truncated
            else if (XT == TLLM_I8)
                o[i] = (uint32_t)__half_as_ushort(__int2half_rn((int)(int8_t)v[2 * i])) | ((uint32_t)__half_as_ushort(__int2half_rn((int)(int8_t)v[2 * i + 1])) << 16);
            else o[i] = (v[2 * i] & 0xFFFFu) | (v[2 * i + 1] << 16);
        }
        *(uint4*)(p.out + ((size_t)pl * p.M + m) * p.k_pad + k) = make_uint4(o[0], o[1], o[2], o[3]);
        if (XT == TLLM_F32) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = mm_next_piece(v[i]);
        }
    }
}
// raw bits of one element
template <int XT>
__device__ __forceinline__ uint32_t stage_load(const void* X, size_t at) {
    if (XT == TLLM_F32) return __ldcg((const unsigned int*)X + at);
    if (XT == TLLM_I8) return (uint32_t)__ldcg((const unsigned char*)X + at);
    return (uint32_t)__ldcg((const unsigned short*)X + at);
}
// Row-major: a thread takes eight values of one row.  Column-major: a block turns a tile of 64 values of k by 32 rows through
// shared memory.  Bound by the bytes it moves: 1 x in, 1.5 x (fp32) or 2 x (int8) out, all of it L2-resident.
template <int XT>
__global__ void __launch_bounds__(256) stage_acts_kernel(const __grid_constant__ StageParams p) {
    pdl_launch_dependents();
    if (!p.late) pdl_wait();
    uint32_t w[8];
    if (p.x_layout == TLLM_ROW_MAJOR) {
        const long long per_row = p.k_pad / 8, i = (long long)blockIdx.x * 256 + threadIdx.x;
        if (i >= per_row * p.M) return;
        const int m = (int)(i / per_row), k = (int)(i - m * per_row) * 8;
        const size_t at = (size_t)m * p.x_ld + k;
        if (XT == TLLM_F32 && k + 8 <= p.K && (((uintptr_t)p.X + at * 4) & 15u) == 0) {
            const uint4 a = __ldcg((const uint4*)((const float*)p.X + at)), b = __ldcg((const uint4*)((const float*)p.X + at) + 1);
            w[0] = a.x, w[1] = a.y, w[2] = a.z, w[3] = a.w, w[4] = b.x, w[5] = b.y, w[6] = b.z, w[7] = b.w;
        } else if (XT == TLLM_I8 && k + 8 <= p.K && (((uintptr_t)p.X + at) & 7u) == 0) {
            const uint2 a = __ldcg((const uint2*)((const char*)p.X + at));
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = (a.x >> (8 * j)) & 0xFFu, w[4 + j] = (a.y >> (8 * j)) & 0xFFu;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) w[j] = k + j < p.K ? stage_load<XT>(p.X, at + j) : 0u;
        }
        stage_eight<XT>(p, w, m, k);
    } else {
        __shared__ uint32_t tile[64][33];
        const int k_tiles = p.k_pad / 64, kt = (int)(blockIdx.x % k_tiles), m0 = (int)(blockIdx.x / k_tiles) * 32;
        for (int i = threadIdx.x; i < 64 * 32; i += 256) {
            const int kk = i >> 5, m = m0 + (i & 31), k = kt * 64 + kk;
            tile[kk][i & 31] = k < p.K && m < p.M ? stage_load<XT>(p.X, (size_t)k * p.x_ld + m) : 0u;
        }
        __syncthreads();
        const int m = threadIdx.x & 31, k8 = (threadIdx.x >> 5) * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = tile[k8 + j][m];
        if (m0 + m < p.M) stage_eight<XT>(p, w, m0 + m, kt * 64 + k8);
    }
    if (p.late) pdl_wait();           // so that whoever waits for this kernel has waited for that one too
}

}  // namespace tllm
