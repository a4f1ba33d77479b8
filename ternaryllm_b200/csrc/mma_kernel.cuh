// mma_kernel.cuh -- the batched product on the tcgen05 tensor cores of sm_100a.
//
// The two-bit copy of W ("bit tiles") is expanded one slice of 128 columns x 64 rows at a time into fp16 / bf16 values in
// shared memory and multiplied on the tensor cores:  D[n, m] = sum_k Wt[n, k] * X[m, k],  A = Wt slice (K-major, 128-byte
// swizzle, written by decoder warps), B = X slice (K-major, the same swizzle, written by TMA), D in tensor memory (fp32).
// The ternary values are exact in both formats and products are exact; sums are accumulated in fp32.
//
// X comes in one or three planes of 16-bit values.  fp16 / bf16 activations whose rows TMA can address are read where they
// are (one plane).  Everything else passes through stage_acts_kernel: int8 becomes fp16 (exact), rows on odd addresses and
// column-major activations are copied straight, and an fp32 value becomes three bf16 values of eight significant bits that
// add up to it exactly; the three planes of a slice are multiplied with the same expanded slice of W, the first into one
// accumulator, the two small ones into another: the tensor core truncates its sums, and with all three in one accumulator
// every step would cut bits (1e-5 of the result at K = 4096, against 1e-7).
//
// One persistent block per SM, twenty-three warps:
//   warp 0        streams this block's range of bit tiles into a shared-memory ring (bulk copies)
//   warp 1        owns tensor memory and issues tcgen05.mma (one lane)
//   warps 2..5    epilogue: tensor memory -> registers -> Y (or partial sums)
//   warp 6        loads the activation slices by TMA
//   warps 7..22   decoders: bit tile -> swizzled fp16 / bf16 slices (two groups of eight warps, alternate units; with four
//                 warps a group the latency of load -> decode -> store -> fence, 1500 clocks a unit, set the pace)
// A unit is two consecutive slices of K: one hand-over between the roles for eight MMAs.  (With one for four the barriers, not
// the tensor core, set the pace: 244 against 159 us without any of them at 5120 x 15360, 2048 rows.)  A has a ring of
// units, B one of (unit, plane); with one plane they are the same ring and one commit frees both.
// Work is either whole output tiles or, where those would leave SMs idle, the flattened list of (output tile, unit) pairs
// cut into equal contiguous ranges, one per block.  Tiles that straddle two or more blocks are summed in block order by the
// last block to arrive, which makes the result independent of scheduling; a block does its two shared tiles first, so that
// this adding-up hides behind the tiles it has to itself.
//
// Every wait is bounded (see bounded_wait); on a time-out the block raises its abort flag, every role leaves
// its loop, tensor memory is released and the status word reports the failure.
#pragma once
#include <cuda.h>

#include "kernels.cuh"

namespace tllm {

#define MM_TILE_N 128                 // output columns per tile  (the MMA's M)
#define MM_TILE_K 64                  // rows of W per slice      (four MMAs of K = 16); a unit is two slices
#define MM_UNIT_BYTES 4096            // bit tiles of one unit: eight groups of sixteen columns, 512 bytes each
#define MM_A_BYTES (MM_TILE_N * MM_TILE_K * 2)
#define MM_A_UNIT (2 * MM_A_BYTES)
#define MM_MAX_STAGES 8
#define MM_THREADS (23 * 32)
#define MM_MAX_NT 256                 // activation rows per tile (the MMA's N), a multiple of sixteen; half of it with three planes
#define MM_OWN_NT 64                  // a handle's own hand-over scratch is for tiles of up to this many rows
#define MM_MAX_M_TILES 16             // row tiles of one launch
#define MM_ERR_WAIT 3                 // status word: a bounded wait of the tensor-core kernel ran out

struct MmParams {
    const uint4* bits;        // bit tiles: groups of sixteen columns, KB slices of 256 bytes each (bittile_format.h)
    void* Y;
    float* partial;           // [2 * gridDim.x][Nt / 4][128][4] fp32: a block's first and last (partial) tile
    unsigned int* counters;   // [tiles][4], zero between launches
    int* status;
    int M, K, N;
    int KB;                   // ceil(K / 64): slices
    int KBU;                  // ceil(KB / 2): units per tile
    int n_tiles, m_tiles;
    int Nt;                   // activation rows per tile
    int split;                // 1: equal unit ranges, tiles may be shared; 0: whole tiles
    int P, plane_rows;        // planes of X; rows from one plane to the next in the tensor map
    int y_dtype, epilogue, y_ld;
    int y_col;                // 1: Y is column-major, y_ld elements from column to column (epilogue 0); 2: and 16-byte stores reach it
    int y_planes;             // 1: Y is three planes of bf16 (the pieces of an fp32 result), plane_y elements apart
    long long plane_y;
    int SA, SB, R;            // ring lengths: units of A, (unit, plane) pairs of B (SA = SB with one plane), units of bit tiles
    uint32_t idesc;           // tcgen05 instruction descriptor
    uint32_t mul4, mul16;     // 4 and 16
    uint32_t tmem_cols;       // power of two >= 2 * Nt (4 * Nt with three planes)
    float scale, scale2;      // half the product's scales: the decoded weights are 0 / +-2
};

// ---- tcgen05 / TMA wrappers ------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem], issued by one thread
__device__ __forceinline__ void umma_f16(uint32_t d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// the barrier receives one arrival when every MMA issued so far by this thread has completed
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
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
// 2-D tiled TMA load into this block's own shared memory: coordinates are (element along K, activation row)
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(map), "r"(bar), "r"(c0), "r"(c1)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

// Shared-memory matrix descriptor of a K-major tile with 128-byte swizzle: rows of 128 bytes, groups of
// eight rows 1024 bytes apart (stride byte offset), descriptor version 1, layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

// Sixteen two-bit codes -> eight words of two 16-bit floats 0 / +-2 (bittile_format.h).  The shifts are multiplications by
// values in registers: they run on the FMA pipe beside the ANDs on the ALU pipe.
__device__ __forceinline__ void mm_decode_word(uint32_t x, uint32_t m4, uint32_t m16, uint32_t (&o)[8]) {
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

// single-lane roles (producers, MMA issuer) spin on the non-blocking probe; warps that wait with all their
// lanes use the blocking try_wait of bounded_wait, which parks them instead of spending issue slots
#define MM_WAIT(bar, par)                                   \
    do {                                                    \
        if (!bounded_spin((bar), (par), abort_flag)) goto done; \
    } while (0)
#define MM_WAIT_BLOCK(bar, par)                             \
    do {                                                    \
        if (!bounded_wait((bar), (par), abort_flag)) goto done; \
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

// The segments of a block's unit range [u0, u1): one per output tile it touches; the first and the last, which other blocks may
// share, come first.
struct MmSegs {
    int u0, u1, KBU, t0, n;
    __device__ __forceinline__ MmSegs(int a, int b, int kbu) : u0(a), u1(b), KBU(kbu), t0(a / kbu), n((b - 1) / kbu - a / kbu + 1) {}
    // segment i: its tile, the tile's units [ua, ub), and which of the block's two slots a partial sum goes to
    __device__ __forceinline__ void get(int i, int& tile, int& ua, int& ub, int& slot) const {
        const int j = i < 2 ? (i ? n - 1 : 0) : i - 1;
        tile = t0 + j;
        const int f = tile * KBU;
        ua = max(u0 - f, 0), ub = min(u1 - f, KBU);
        slot = j ? 1 : 0;
    }
};

__global__ void __launch_bounds__(MM_THREADS, 1) mma_spmm_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ MmParams p) {
    extern __shared__ unsigned char mm_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // ---- this block's unit range -----------------------------------------------------------------------
    const int G = (int)gridDim.x, cta = (int)blockIdx.x, KBU = p.KBU, KB = p.KB, tiles = p.n_tiles * p.m_tiles;
    const long long total = (long long)tiles * KBU;
    const int u0 = p.split ? (int)(total * cta / G) : (int)((long long)tiles * cta / G) * KBU;
    const int u1 = p.split ? (int)(total * (cta + 1) / G) : (int)((long long)tiles * (cta + 1) / G) * KBU;
    if (u0 >= u1) return;
    const MmSegs segs(u0, u1, KBU);

    // ---- shared memory ---------------------------------------------------------------------------------
    const uint32_t raw0 = smem_u32(mm_smem);
    const uint32_t base = (raw0 + 1023u) & ~1023u;                 // swizzled tiles need 1024-byte alignment
    const uint32_t SA = (uint32_t)p.SA, SB = (uint32_t)p.SB, R = (uint32_t)p.R;
    const int Nt = p.Nt;
    const uint32_t b_slice = (uint32_t)Nt * 128u, b_unit = 2u * b_slice;
    const uint32_t a_base = base, b_base = a_base + SA * MM_A_UNIT, r_base = b_base + SB * b_unit;
    const uint32_t bar_base = r_base + R * MM_UNIT_BYTES;
    volatile int* flags = (volatile int*)(mm_smem + (bar_base - raw0) + 8 * 52);   // [0] tensor-memory address, [1] abort
    volatile int* abort_flag = flags + 1;
#define A_FULL(s) (bar_base + 8u * (uint32_t)(s))
#define A_EMPTY(s) (bar_base + 8u * (8u + (uint32_t)(s)))
#define B_FULL(s) (bar_base + 8u * (16u + (uint32_t)(s)))
#define B_EMPTY(s) (bar_base + 8u * (24u + (uint32_t)(s)))
#define RAW_FULL(r) (bar_base + 8u * (32u + (uint32_t)(r)))
#define RAW_EMPTY(r) (bar_base + 8u * (40u + (uint32_t)(r)))
#define ACC_FULL(a) (bar_base + 8u * (48u + (uint32_t)(a)))
#define ACC_EMPTY(a) (bar_base + 8u * (50u + (uint32_t)(a)))

    if (tid == 0) {
        for (int s = 0; s < MM_MAX_STAGES; ++s) {
            mbar_init(A_FULL(s), 8);       // the eight decoder warps of a group
            mbar_init(A_EMPTY(s), 1);      // tcgen05.commit
            mbar_init(B_FULL(s), 1);       // the TMA thread's expect_tx arrival
            mbar_init(B_EMPTY(s), 1);      // tcgen05.commit
            mbar_init(RAW_FULL(s), 1);
            mbar_init(RAW_EMPTY(s), 8);    // the eight decoder warps of the group that took the unit
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(ACC_FULL(a), 1);
            mbar_init(ACC_EMPTY(a), 4);    // the four epilogue warps
        }
        flags[0] = 0;
        flags[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    if (warp == 1) tmem_alloc(smem_u32((const void*)flags), p.tmem_cols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = (uint32_t)flags[0];
    const uint32_t acc_cols = p.P == 1 ? (uint32_t)Nt : 2u * (uint32_t)Nt;
    pdl_launch_dependents();

    // Every role walks the same list of segments.
    if (warp == 0) {
        // ---- bit-tile producer: the weights do not depend on the preceding kernel, so this starts at once.  A tile's eight
        // groups of sixteen columns are eight streams along K: lanes 0..7 copy one each.
        uint32_t r = 0, rph = 0;
        for (int i = 0; i < segs.n; ++i) {
            int tile, ua, ub, sl;
            segs.get(i, tile, ua, ub, sl);
            const char* src = (const char*)p.bits + ((size_t)(tile / p.m_tiles * 8 + (lane & 7)) * KB + (size_t)ua * 2) * 256u;
            for (int ku = ua; ku < ub; ++ku, src += 512) {
                if (!__all_sync(0xffffffffu, bounded_wait(RAW_EMPTY(r), rph ^ 1u, abort_flag))) goto done;
                const uint32_t bytes = (uint32_t)min(2, KB - ku * 2) * 256u;
                if (lane == 0) mbar_expect_tx(RAW_FULL(r), 8u * bytes);
                __syncwarp();
                if (lane < 8) bulk_g2s(r_base + r * MM_UNIT_BYTES + (uint32_t)lane * 512u, src, bytes, RAW_FULL(r));
                MM_ADVANCE(r, rph, R);
            }
        }
    } else if (warp == 6) {
        // ---- activation producer: a unit and plane is two TMA boxes on one barrier
        if (lane == 0) {
            pdl_wait();
            uint32_t b = 0, bph = 0;
            for (int i = 0; i < segs.n; ++i) {
                int tile, ua, ub, sl;
                segs.get(i, tile, ua, ub, sl);
                const int row0 = (tile % p.m_tiles) * Nt;
                for (int ku = ua; ku < ub; ++ku) {
                    const int nk = min(2, KB - ku * 2);
                    for (int pl = 0; pl < p.P; ++pl) {
                        MM_WAIT(p.P == 1 ? A_EMPTY(b) : B_EMPTY(b), bph ^ 1u);
                        mbar_expect_tx(B_FULL(b), (uint32_t)nk * b_slice);
                        for (int h = 0; h < nk; ++h)
                            tma_load_2d(b_base + b * b_unit + (uint32_t)h * b_slice, &tmap, (ku * 2 + h) * MM_TILE_K, pl * p.plane_rows + row0, B_FULL(b));
                        MM_ADVANCE(b, bph, SB);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer (whole warp converged, one elected lane per instruction)
        const uint32_t idesc = p.idesc;
        const uint64_t ad0 = umma_desc_sw128(a_base), bd0 = umma_desc_sw128(b_base);
        uint32_t sa = 0, saph = 0, sb = 0, sbph = 0, a = 0, aph = 0;
        for (int i = 0; i < segs.n; ++i) {
            int tile, ua, ub, sl;
            segs.get(i, tile, ua, ub, sl);
            MM_WAIT(ACC_EMPTY(a), aph ^ 1u);
            tc_fence_after();
            const uint32_t d = tmem + a * acc_cols;
            uint32_t acc = 0;
            for (int ku = ua; ku < ub; ++ku) {
                const bool two = ku * 2 + 1 < KB;
                MM_WAIT(A_FULL(sa), saph);
                const uint64_t ad = ad0 + sa * (MM_A_UNIT >> 4);
                for (int pl = 0; pl < p.P; ++pl) {
                    MM_WAIT(B_FULL(sb), sbph);
                    tc_fence_after();
                    const uint64_t bd = bd0 + sb * (b_unit >> 4);
                    const uint32_t dp = pl == 0 ? d : d + (uint32_t)Nt, keep = pl < 2 ? acc : 1u;
                    if (elect_one()) {
#pragma unroll
                        for (uint32_t k4 = 0; k4 < MM_TILE_K / 16; ++k4)      // 16 values = 32 bytes = 2 descriptor address units
                            umma_f16(dp, ad + 2u * k4, bd + 2u * k4, idesc, k4 == 0 ? keep : 1u);
                        if (two) {
#pragma unroll
                            for (uint32_t k4 = 0; k4 < MM_TILE_K / 16; ++k4)
                                umma_f16(dp, ad + (MM_A_BYTES >> 4) + 2u * k4, bd + (b_slice >> 4) + 2u * k4, idesc, 1u);
                        }
                        if (p.P > 1) umma_commit(B_EMPTY(sb));
                        if (pl == p.P - 1) umma_commit(A_EMPTY(sa));          // with one plane this frees the unit of B too
                    }
                    __syncwarp();
                    MM_ADVANCE(sb, sbph, SB);
                }
                acc = 1;
                MM_ADVANCE(sa, saph, SA);
            }
            if (elect_one()) umma_commit(ACC_FULL(a));
            __syncwarp();
            a ^= 1u;
            aph ^= (a == 0);
        }
    } else if (warp >= 7) {
        // ---- decoders: group 0 (warps 7..14) takes even units, group 1 (warps 15..22) odd units; warp dw of a group takes sixteen
        // columns: a lane decodes the words it would feed to mma.sync
        const int dw = (warp - 7) & 7, group = (warp - 7) >> 3;
        const uint32_t g = (uint32_t)lane >> 2, t = (uint32_t)lane & 3u;
        const uint32_t ch0 = ((2u * t) ^ g) << 4, ch1 = ((2u * t + 1u) ^ g) << 4;      // swizzled 16-byte chunks of rows 16t .. 16t+15
        uint32_t m4, m16;
        asm volatile("mov.b32 %0, %2;\n\tmov.b32 %1, %3;" : "=r"(m4), "=r"(m16) : "r"(p.mul4), "r"(p.mul16));
        uint32_t sa = 0, saph = 0, r = 0, rph = 0, turn = 0;
        for (int i = 0; i < segs.n; ++i) {
            int tile, ua, ub, sl;
            segs.get(i, tile, ua, ub, sl);
            for (int ku = ua; ku < ub; ++ku, turn ^= 1u) {
                if ((int)turn == group) {
                    const bool two = ku * 2 + 1 < KB;
                    const uint32_t at = r_base + r * MM_UNIT_BYTES + (uint32_t)dw * 512u;
                    MM_WAIT_BLOCK(RAW_FULL(r), rph);
                    uint4 rw;
                    if (two) rw = ld_shared_v4(at + (uint32_t)lane * 16u);
                    else asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(rw.x), "=r"(rw.y) : "r"(at + (uint32_t)lane * 8u) : "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(RAW_EMPTY(r));
                    MM_WAIT_BLOCK(A_EMPTY(sa), saph ^ 1u);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (h == 0 || two) {
                            const uint32_t arow = a_base + sa * MM_A_UNIT + (uint32_t)h * MM_A_BYTES + ((uint32_t)(dw * 16) + g) * 128u;
#pragma unroll
                            for (int hi = 0; hi < 2; ++hi) {
                                uint32_t o[8];
                                mm_decode_word(h ? (hi ? rw.w : rw.z) : (hi ? rw.y : rw.x), m4, m16, o);
                                st_shared_v4(arow + (uint32_t)hi * 1024u + ch0, o[0], o[1], o[2], o[3]);
                                st_shared_v4(arow + (uint32_t)hi * 1024u + ch1, o[4], o[5], o[6], o[7]);
                            }
                        }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // make the slices visible to the tensor core's reads
                    __syncwarp();
                    if (lane == 0) mbar_arrive(A_FULL(sa));
                }
                MM_ADVANCE(sa, saph, SA);
                MM_ADVANCE(r, rph, R);
            }
        }
    } else {
        // ---- epilogue (warps 2..5): a warp may read the 32 tensor-memory lanes selected by warp % 4
        const int q = warp & 3, nl = q * 32 + lane;
        pdl_wait();
        uint32_t a = 0, aph = 0;
        for (int i = 0; i < segs.n; ++i) {
            int tile, ua, ub, sl;
            segs.get(i, tile, ua, ub, sl);
            const int nt = tile / p.m_tiles, mt = tile - nt * p.m_tiles;
            MM_WAIT_BLOCK(ACC_FULL(a), aph);
            tc_fence_after();
            const bool full = ua == 0 && ub == KBU;
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + a * acc_cols;
            const size_t slot_floats = (size_t)MM_TILE_N * Nt;
            float* slot = p.partial + (size_t)(2 * cta + sl) * slot_floats + nl * 4;
            const int n = nt * MM_TILE_N + nl;
            const bool in_n = n < p.N;
            // four consecutive rows m .. m+3 of this lane's column
            auto emit4 = [&](const float (&v)[4], int m) {
                if (p.y_col == 2 && in_n && m + 4 <= p.M && p.y_dtype != TLLM_F16 && p.y_dtype != TLLM_BF16) {
                    // column-major results of four bytes: the rows are neighbours
                    uint4 w;
                    if (p.y_dtype == TLLM_I32) w = make_uint4((uint32_t)(int)(v[0] * 0.5f), (uint32_t)(int)(v[1] * 0.5f), (uint32_t)(int)(v[2] * 0.5f), (uint32_t)(int)(v[3] * 0.5f));
                    else w = make_uint4(__float_as_uint(v[0] * p.scale), __float_as_uint(v[1] * p.scale), __float_as_uint(v[2] * p.scale), __float_as_uint(v[3] * p.scale));
                    *(uint4*)((uint32_t*)p.Y + (size_t)n * p.y_ld + m) = w;
                    return;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float y;
                    bool ok;
                    size_t at;
                    if (p.epilogue == 0) {
                        y = v[j] * p.scale;
                        ok = in_n;
                        at = p.y_col ? (size_t)n * p.y_ld + m + j : (size_t)(m + j) * p.y_ld + n;
                    } else {
                        const float other = __shfl_xor_sync(0xffffffffu, v[j], 1);
                        y = silu_mul(v[j] * p.scale, other * p.scale2);
                        ok = !(nl & 1) && n + 1 < p.N;
                        at = (size_t)(m + j) * p.y_ld + (n >> 1);
                    }
                    if (!ok || m + j >= p.M) continue;
                    if (p.y_planes) {
                        // the three bf16 values that add up to y (see stage_acts_kernel)
                        uint32_t w = __float_as_uint(y);
#pragma unroll
                        for (int pl = 0; pl < 3; ++pl) {
                            ((unsigned short*)p.Y)[(size_t)pl * p.plane_y + at] = (unsigned short)(w >> 16);
                            w = __float_as_uint(__uint_as_float(w) - __uint_as_float(w & 0xFFFF0000u));
                        }
                    } else if (p.y_dtype == TLLM_I32) ((int*)p.Y)[at] = (int)(v[j] * 0.5f);
                    else store_out(p.Y, p.y_dtype, at, y);
                }
            };
            // sixteen accumulator columns (rows of X) of this lane's column of W
            auto load16 = [&](int c16, float (&f)[16]) {
                uint32_t v[16];
                tmem_ld16(taddr + (uint32_t)c16, v);
#pragma unroll
                for (int t = 0; t < 16; ++t) f[t] = __uint_as_float(v[t]);
                if (p.P > 1) {
                    tmem_ld16(taddr + (uint32_t)(Nt + c16), v);
#pragma unroll
                    for (int t = 0; t < 16; ++t) f[t] += __uint_as_float(v[t]);
                }
            };
            bool sum = false;                    // this block adds up the parts of a shared tile
            int cf = 0, cl = 0;
            if (!full) {
                // The last of the blocks that share this tile to arrive adds the partial sums, in block order.  Each epilogue warp owns 32
                // columns of the tile and runs the hand-over for them by itself.  The last block's own part stays in tensor memory;
                // a block that finds all the others there already does not even write it.
                const long long first_unit = (long long)tile * KBU, last_unit = first_unit + KBU - 1;
                cf = (int)(((first_unit + 1) * G + total - 1) / total - 1), cl = (int)(((last_unit + 1) * G + total - 1) / total - 1);
                unsigned int* ctr = p.counters + (size_t)tile * 4 + q;
                const unsigned int others = (unsigned int)(cl - cf);
                unsigned int there = 0;
                if (lane == 0) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(there) : "l"(ctr) : "memory");
                sum = __shfl_sync(0xffffffffu, there, 0) == others;
                if (!sum) {
                    for (int c16 = 0; c16 < Nt; c16 += 16) {
                        float f[16];
                        load16(c16, f);
#pragma unroll
                        for (int t = 0; t < 16; t += 4) __stcg((float4*)(slot + (size_t)(c16 + t) * MM_TILE_N), make_float4(f[t], f[t + 1], f[t + 2], f[t + 3]));
                    }
                    __threadfence();
                    __syncwarp();
                    if (lane == 0) there = atomicAdd(ctr, 1u);
                    sum = __shfl_sync(0xffffffffu, there, 0) == others;
                }
                if (sum) {
                    if (lane == 0) *ctr = 0;
                    __threadfence();
                }
            }
            if (full || sum) {
                // A part lies in its block's slot 0, except that the first block may have come from an earlier tile.
                const float* part0 = p.partial + (size_t)(2 * cf + (!full && total * cf / G >= (long long)tile * KBU ? 0 : 1)) * slot_floats + nl * 4;
                const float* rest = p.partial + (size_t)(2 * cf + 2) * slot_floats + nl * 4;
                const bool pairs = p.epilogue == 0 && !p.y_planes && !p.y_col && (p.y_dtype == TLLM_F16 || p.y_dtype == TLLM_BF16) && !(p.y_ld & 1) &&
                                   ((uintptr_t)p.Y & 3u) == 0 && nt * MM_TILE_N + MM_TILE_N <= p.N;
                for (int c16 = 0; c16 < Nt; c16 += 16) {
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
                            ps = rest + (size_t)(cc - cf) * 2 * slot_floats + (size_t)c16 * MM_TILE_N;
                        }
                    }
                    if (pairs) {
                        // 16-bit outputs: neighbouring lanes trade one value per pair of rows, so that every lane
                        // writes two adjacent columns of one row with a single 4-byte store
#pragma unroll
                        for (int t = 0; t < 16; t += 2) {
                            const float e0 = f[t] * p.scale, e1 = f[t + 1] * p.scale;
                            const float mine = (lane & 1) ? e1 : e0, send = (lane & 1) ? e0 : e1;
                            const float got = __shfl_xor_sync(0xffffffffu, send, 1);
                            const int m = mt * Nt + c16 + t + (lane & 1);
                            const float lo = (lane & 1) ? got : mine, hi = (lane & 1) ? mine : got;
                            if (m < p.M) {
                                uint32_t w;
                                if (p.y_dtype == TLLM_F16) w = (uint32_t)__half_as_ushort(__float2half_rn(lo)) | ((uint32_t)__half_as_ushort(__float2half_rn(hi)) << 16);
                                else w = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(lo)) | ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(hi)) << 16);
                                *(uint32_t*)((char*)p.Y + ((size_t)m * p.y_ld + (n & ~1)) * 2) = w;
                            }
                        }
                    } else {
#pragma unroll
                        for (int t = 0; t < 16; t += 4) {
                            const float e[4] = {f[t], f[t + 1], f[t + 2], f[t + 3]};
                            emit4(e, mt * Nt + c16 + t);
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ACC_EMPTY(a));
            a ^= 1u;
            aph ^= (a == 0);
        }
    }
done:
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, p.tmem_cols);
    }
    if (tid == 0 && flags[1]) atomicExch(p.status, MM_ERR_WAIT);
#undef A_FULL
#undef A_EMPTY
#undef B_FULL
#undef B_EMPTY
#undef RAW_FULL
#undef RAW_EMPTY
#undef ACC_FULL
#undef ACC_EMPTY
}
#undef MM_WAIT
#undef MM_WAIT_BLOCK
#undef MM_ADVANCE

// ---- activations as planes of 16-bit values for the kernel above: rows of k_pad values, zero beyond K ------------------
struct StageParams {
    const void* X;
    unsigned short* out;      // [planes][M][k_pad]
    int x_dtype, x_layout, x_ld;
    int M, K, k_pad;
};
// eight consecutive values of one row -> 16 bytes of each plane
template <int XT>
__device__ __forceinline__ void stage_eight(const StageParams& p, const uint32_t (&w)[8], int m, int k) {
    constexpr int PL = XT == TLLM_F32 ? 3 : 1;
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = w[i];
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
            for (int i = 0; i < 8; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) - __uint_as_float(v[i] & 0xFFFF0000u));   // exact
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
    pdl_wait();
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
}

}  // namespace tllm
