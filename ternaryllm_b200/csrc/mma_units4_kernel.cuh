// mma_units4_kernel.cuh -- the batched product of mma_kernel.cuh for launches of few units: a unit is four slices of K, one block per tile.
//
// Where a block has a handful of units, what counts is the time from its start to its first MMA and from its last one to the result, and how many
// barriers are passed between; sixteen decoder warps expand a whole unit at a time, four warps store, and a block has twenty-three warps to start.
// mma_kernel.cuh feeds the tensor core better and starts later (24 rows of fp16 on 2048 x 2048: 5.6 us here, 6.3 there; 256 rows on 4096 x 4096
// 15.1 and 16.5; but 256 rows of fp32 on 4096 x 11008, planes included, 67 and 52; 2048 rows of 5120 x 15360 276 and 233).  mm_plan has an
// estimate of either.
//
// Roles: warp 0 bit tiles and warp 6 activations by TMA, warp 1 MMAs (one thread each), warps 2..5 epilogue, warps 7..22 decoders.  A has a ring of
// two units (256 columns of tensor memory; the accumulators have the other 256: two of them where they fit, and behind them, for fp32
// activations, the sum of the legs so far).  Segments, clusters, the hand-over of parts and the stores are those of mma_kernel.cuh.
#pragma once
#include "mma_kernel.cuh"

namespace tllm {

#define MS_UK 4
#define MS_UNIT_BYTES 8192            // bit tiles of one unit: eight groups of sixteen columns, 1024 bytes each
#define MS_RAW_UNITS 4
#define MS_A_UNITS 2
#define MS_A_COL 256
#define MS_LEG 4
#define MS_THREADS (23 * 32)
static_assert(MS_RAW_UNITS <= MM_MAX_STAGES && MS_A_UNITS <= MM_MAX_STAGES, "as many barriers as places");
static_assert(MS_A_COL + MS_A_UNITS * MS_UK * 32 <= 512, "the ring of expanded units lies in tensor memory");

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "f"(v[0]), "f"(v[1]),
        "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
        : "memory");
}
// sixteen columns of the calling warp's lanes at each of two places, one wait for both; added up
__device__ __forceinline__ void tmem_sum16(uint32_t at, uint32_t at2, float (&f)[16]) {
    uint32_t v[16], u[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
          "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
          "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(at), "r"(at2)
        : "memory");
#pragma unroll
    for (int t = 0; t < 16; ++t) f[t] = __uint_as_float(v[t]) + __uint_as_float(u[t]);
}
// sixteen columns of D (rows of X) of this lane's column of W, the planes added up, the small ones first
__device__ __forceinline__ void ms_load16(uint32_t at, int nt, int planes, float (&f)[16]) {
    uint32_t v[16];
    if (planes == 1) {
        tmem_ld16(at, v);
#pragma unroll
        for (int t = 0; t < 16; ++t) f[t] = __uint_as_float(v[t]);
    } else {
        tmem_sum16(at + (uint32_t)nt, at + (uint32_t)(2 * nt), f);
        tmem_ld16(at, v);
#pragma unroll
        for (int t = 0; t < 16; ++t) f[t] = __uint_as_float(v[t]) + f[t];
    }
}
__device__ __forceinline__ void ms_add16(uint32_t at, float (&f)[16]) {
    uint32_t v[16];
    tmem_ld16(at, v);
#pragma unroll
    for (int t = 0; t < 16; ++t) f[t] += __uint_as_float(v[t]);
}

__host__ __device__ __forceinline__ uint32_t ms_acc_sets(int planes, int nt) { return (2 * planes + (planes > 1 ? 1 : 0)) * nt <= MS_A_COL ? 2u : 1u; }

__global__ void __launch_bounds__(MS_THREADS, 1) mma_units4_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ CUtensorMap wmap,
                                                                   const __grid_constant__ MmParams p) {
    extern __shared__ unsigned char mm_smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // ---- this block's unit range -----------------------------------------------------------------------
    const int G = (int)gridDim.x, cta = (int)blockIdx.x, KBU = p.KBU, KB = p.KB, tiles = p.n_tiles * p.m_tiles;
    const int total = tiles * KBU;
    const bool clustered = p.split == 2;
    const int C = clustered ? p.cluster : 1, rank = clustered ? cta & (C - 1) : 0;
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
    // The length of the ring of bit tiles is a parameter: as a constant ptxas allots other registers, and stores of results get slower (998 rows of
    // int8 on 320 x 7296 20.5 us, 19.5 so; 500 rows of fp32 on 312 x 12480 31.3 and 28.7; 192 rows of fp16 on 4096 x 4096 13.9 and 13.6).
    const uint32_t SB = (uint32_t)p.SB, R = (uint32_t)p.R;
    const int Nt = p.Nt;
    const uint32_t acc_cols = (uint32_t)(p.P * Nt), b_slice = acc_cols * 128u, b_unit = MS_UK * b_slice;
    const uint32_t b_base = base, r_base = b_base + SB * b_unit;
    const uint32_t bar_base = r_base + R * MS_UNIT_BYTES, part_base = bar_base + 512u;      // part_base: the cluster's parts, [block][rows / 16][4][128] x 16 bytes
    volatile int* flags = (volatile int*)(mm_smem + (bar_base - raw0) + 8 * 56);   // [0] tensor-memory address, [1] abort
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

    // Start, as in mma_kernel.cuh: the first bit tiles on their way, tensor memory and the other barriers beside one another.
    MmBitsRange load(segs, p, 1, 0);
    if (warp == 0) {
        if (lane < 16) mbar_init(RAW_FULL(lane), lane < 8 ? 1 : 16);            // RAW_EMPTY: the decoder warps
        mm_fence_barriers();
        __syncwarp();
        // The weights do not depend on the preceding kernel, unless that is the one that makes them.  A unit is one box of 8 x 1024 bytes; past the end
        // of K it is filled with zeros, which count.
        if (!p.wait_bits && elect_one())
            for (uint32_t r = 0; r < R && load.left(); ++r, load.next()) {
                mbar_expect_tx(RAW_FULL(r), MS_UNIT_BYTES);
                tma_load_2d(r_base + r * MS_UNIT_BYTES, &wmap, load.ku * (MS_UK * 64), load.row0, RAW_FULL(r));
            }
        __syncwarp();
    } else if (warp == 1) {
        tmem_alloc(smem_u32((const void*)flags), 512);
    } else if (warp < 4) {
        const int i = tid - 64;                                                // the order of the names above
        if (i < 56 && (i < 32 || i >= 48)) {
            const int n = i < 8 ? 16                                           // the decoder warps
                        : i < 50 ? 1                                           // tcgen05.commit; B_FULL: the TMA thread's expect_tx arrival
                        : i < 52 ? 4                                           // the four epilogue warps
                                 : max(C - 1, 1);                              // the same warp of the other blocks
            mbar_init(bar_base + 8u * (uint32_t)i, (uint32_t)n);
        }
        if (i == 63) {
            flags[1] = 0;
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap) : "memory");
        }
        mm_fence_barriers();
    }
    if (clustered) mm_cluster_arrive();    // the others' barriers are waited for where they are needed
    bool joined = !clustered;
    const auto join = [&] {
        if (!joined) mm_cluster_wait(), joined = true;
    };
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = (uint32_t)flags[0];
    // one or two sets of accumulators, and behind them, for fp32 activations, the sum of the legs so far
    const uint32_t accs = ms_acc_sets(p.P, Nt), run_col = accs * acc_cols;
    pdl_launch_dependents();

    // Every role walks the same list of segments.
    if (warp == 0) {
        // ---- bit-tile producer, behind the first round of its ring
        if (elect_one()) {
            uint32_t r = 0, rph = 0;
            if (p.wait_bits) pdl_wait();
            else rph = 1u;
            for (; load.left(); load.next()) {
                MM_WAIT(RAW_EMPTY(r), rph ^ 1u);
                mbar_expect_tx(RAW_FULL(r), MS_UNIT_BYTES);
                tma_load_2d(r_base + r * MS_UNIT_BYTES, &wmap, load.ku * (MS_UK * 64), load.row0, RAW_FULL(r));
                MM_ADVANCE(r, rph, R);
            }
        }
    } else if (warp == 6) {
        // ---- activation producer: a unit is four TMA boxes (all planes of a slice each) on one barrier
        if (elect_one()) {
            pdl_wait();
            uint32_t b = 0, bph = 0;
            for (int i = 0; i < segs.n; ++i) {
                int tile, ua, ub, sl;
                segs.get(i, tile, ua, ub, sl);
                const int row0 = (tile - mm_div(tile, p.m_tiles, p.mt_inv) * p.m_tiles) * Nt;
                for (int ku = ua; ku < ub; ++ku) {
                    const int nk = min(MS_UK, KB - ku * MS_UK);
                    MM_WAIT(B_EMPTY(b), bph ^ 1u);
                    mbar_expect_tx(B_FULL(b), (uint32_t)nk * b_slice);
                    for (int h = 0; h < nk; ++h) {
                        const uint32_t to = b_base + b * b_unit + (uint32_t)h * b_slice;
                        if (p.P == 1) tma_load_2d(to, &tmap, (ku * MS_UK + h) * MM_TILE_K, row0, B_FULL(b));
                        else tma_load_3d(to, &tmap, (ku * MS_UK + h) * MM_TILE_K, row0, 0, B_FULL(b));
                    }
                    MM_ADVANCE(b, bph, SB);
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        if (elect_one()) {
            const uint32_t idesc = p.idesc, b_lo0 = (b_base >> 4) & 0x3FFFu;
            uint32_t sa = 0, saph = 0, sb = 0, sbph = 0, a = 0, aph = 0;
            for (int i = 0; i < segs.n; ++i) {
                int tile, ua, ub, sl, left = 0;
                segs.get(i, tile, ua, ub, sl);
                uint32_t d = 0, acc = 0;
                for (int ku = ua; ku < ub; ++ku) {
                    MM_SPIN(A_FULL(sa), saph);
                    MM_SPIN(B_FULL(sb), sbph);
                    if (left == 0) {                             // a leg starts
                        MM_SPIN(ACC_EMPTY(a), aph ^ 1u);
                        d = tmem + a * acc_cols, acc = 0, left = min(p.leg, ub - ku);
                    }
                    tc_fence_after();
                    const int nk = min(MS_UK, KB - ku * MS_UK);
                    const uint32_t at = tmem + MS_A_COL + sa * (MS_UK * 32u), b_lo = b_lo0 + sb * (b_unit >> 4);
                    // 16 values = 8 columns of A, 32 bytes = 2 descriptor address units of B
#pragma unroll
                    for (uint32_t h = 0; h < MS_UK; ++h)
                        if ((int)h < nk) {
#pragma unroll
                            for (uint32_t k4 = 0; k4 < MM_TILE_K / 16; ++k4)
                                umma_f16_ts<1>(d, at + 32u * h + 8u * k4, b_lo + h * (b_slice >> 4) + 2u * k4, idesc, (h | k4) == 0 ? acc : 1u);
                        }
                    umma_commit(A_EMPTY(sa));
                    umma_commit(B_EMPTY(sb));
                    MM_ADVANCE(sb, sbph, SB);
                    MM_ADVANCE(sa, saph, MS_A_UNITS);
                    acc = 1;
                    if (--left == 0) {
                        umma_commit(ACC_FULL(a));
                        MM_ADVANCE(a, aph, accs);
                    }
                }
            }
        }
    } else if (warp >= 7) {
        // ---- decoders: a warp expands slice h of every unit, 32 columns of W, into its 32 lanes of tensor memory.  Lane 4g + u
        // holds column 16 * (u >> 1) + 8 * (u & 1) + g of them (see mm_column).
        const int q = warp & 3, h = (warp - 7) >> 2;
        const uint32_t g = (uint32_t)lane >> 2, u = (uint32_t)lane & 3u;
        const uint32_t raw_lane = (uint32_t)(2 * q + (u >> 1)) * 1024u + (uint32_t)(h >> 1) * 512u;
        const uint32_t a_lane = tmem + MS_A_COL + ((uint32_t)(q * 32) << 16) + (uint32_t)h * 32u;
        uint32_t m4, m16;
        asm volatile("mov.b32 %0, %2;\n\tmov.b32 %1, %3;" : "=r"(m4), "=r"(m16) : "r"(p.mul4), "r"(p.mul16));
        uint32_t sa = 0, saph = 0, r = 0, rph = 0;
        for (int i = 0; i < segs.n; ++i) {
            int tile, ua, ub, sl;
            segs.get(i, tile, ua, ub, sl);
            for (int ku = ua; ku < ub; ++ku) {
                const int slice = ku * MS_UK + h;
                const uint32_t at = r_base + r * MS_UNIT_BYTES + raw_lane;
                MM_WAIT(RAW_FULL(r), rph);
                uint32_t w[4] = {};
                if ((slice | 1) < KB) {
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        uint32_t lo, hi;
                        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(lo), "=r"(hi) : "r"(at + (uint32_t)mm_chunk((int)g, t) * 16u + (uint32_t)(h & 1) * 8u) : "memory");
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
                MM_WAIT(A_EMPTY(sa), saph ^ 1u);
                if (slice < KB) {
                    tc_fence_after();
                    tmem_st32(a_lane + sa * (MS_UK * 32u), o);
                    tmem_wait_st();
                    tc_fence_before();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(A_FULL(sa));
                MM_ADVANCE(sa, saph, MS_A_UNITS);
                MM_ADVANCE(r, rph, R);
            }
        }
    } else {
        // ---- epilogue (warps 2..5): a warp may read the 32 tensor-memory lanes selected by warp % 4
        const int q = warp & 3, nl = q * 32 + lane, ncol = q * 32 + mm_column(lane);
        join();
        pdl_wait();
        uint32_t a = 0, aph = 0;
        for (int i = 0; i < segs.n; ++i) {
            int tile, ua, ub, sl;
            segs.get(i, tile, ua, ub, sl);
            const int nt = mm_div(tile, p.m_tiles, p.mt_inv), mt = tile - nt * p.m_tiles;
            const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16);
            // all legs but the last join the sum in tensor memory
            bool legs = false;
            for (int left = ub - ua; left > p.leg; left -= p.leg) {
                MM_WAIT(ACC_FULL(a), aph);
                tc_fence_after();
                for (int c16 = 0; c16 < Nt; c16 += 16) {
                    float f[16];
                    ms_load16(lanes + a * acc_cols + (uint32_t)c16, Nt, p.P, f);
                    if (legs) ms_add16(lanes + run_col + (uint32_t)c16, f);
                    tmem_st16(lanes + run_col + (uint32_t)c16, f);
                }
                tmem_wait_st();
                legs = true;
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(ACC_EMPTY(a));
                MM_ADVANCE(a, aph, accs);
            }
            MM_WAIT(ACC_FULL(a), aph);
            tc_fence_after();
            const bool full = ua == 0 && ub == KBU;
            const uint32_t taddr = lanes + a * acc_cols;
            const size_t slot_floats = (size_t)MM_TILE_N * Nt;
            float* slot = p.partial + (size_t)(2 * cta + sl) * slot_floats + nl * 4;
            const int n = nt * MM_TILE_N + ncol;
            // sixteen accumulator columns (rows of X) of this lane's column of W
            auto load16 = [&](int c16, float (&f)[16]) {
                ms_load16(taddr + (uint32_t)c16, Nt, p.P, f);
                if (legs) ms_add16(lanes + run_col + (uint32_t)c16, f);
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
                    if (o == rank) continue;
                    float f[16];
                    load16(16 * c, f);
                    const uint32_t to = mm_peer(part_base + (uint32_t)(((rank * own + c / C) * 4) * 128 + nl) * 16u, (uint32_t)o);
#pragma unroll
                    for (int t = 0; t < 4; ++t) mm_st_peer(to + (uint32_t)t * 2048u, f[4 * t], f[4 * t + 1], f[4 * t + 2], f[4 * t + 3]);
                }
                __syncwarp();
                if (lane < C && lane != rank && lane < sixteens) mm_arrive_peer(mm_peer(PART_FULL(q), (uint32_t)lane));
                if (rank < sixteens) {
                    if (!mm_wait_cluster(PART_FULL(q), abort_flag)) goto done;
                    mm_with_out(p, [&](auto out, auto silu) {
                        uint32_t at0 = part_base + (uint32_t)nl * 16u;
                        for (int c = rank; c < sixteens; c += C, at0 += 8192u) {
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
                            finish16(out, silu, f, n, mt * Nt + 16 * c);
                        }
                    });
                }
            } else if (!full) {
                // The last of the blocks that share this tile to arrive adds the partial sums, in block order.  Each epilogue warp owns 32
                // columns of the tile and runs the hand-over for them by itself.  The last block's own part stays in tensor memory;
                // a block that finds all the others there already does not even write it.
                cf = mm_owner(p, tile * KBU, G, total), cl = mm_owner(p, tile * KBU + KBU - 1, G, total);
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
            if (!clustered && (full || sum)) {
                // A part lies in its block's slot 0, except that the first block may have come from an earlier tile.
                const float* part0 = p.partial + (size_t)(2 * cf + (!full && mm_share(p, cf, G) >= tile * KBU ? 0 : 1)) * slot_floats + nl * 4;
                const float* rest = p.partial + (size_t)(2 * cf + 2) * slot_floats + nl * 4;
                mm_with_out(p, [&](auto out, auto silu) {
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
                        finish16(out, silu, f, n, mt * Nt + c16);
                    }
                });
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ACC_EMPTY(a));
            MM_ADVANCE(a, aph, accs);
        }
    }
done:
    __syncwarp();
    join();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
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
#undef MM_WAIT
#undef MM_SPIN
#undef MM_ADVANCE

}  // namespace tllm
