// bits.cu -- instantiations and launches of bits_spmm_kernel (bits_kernel.cuh), in a translation unit of their own so that
// they compile beside the rest.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "bits_kernel.cuh"
#include "util.h"

namespace tllm {
namespace {

#define BT_TRY(expr)                                                                                       \
    do {                                                                                                   \
        cudaError_t e_ = (expr);                                                                           \
        if (e_ != cudaSuccess) return fail(TLLM_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_)); \
    } while (0)

template <int XT, int NB, int GR, bool ASYNC, bool SHARED>
int launch(const BitsParams& p, int grid, size_t smem, int device, cudaStream_t st) {
    auto kern = bits_spmm_kernel<XT, NB, GR, ASYNC, SHARED>;
    static std::once_flag once[64];
    cudaError_t err = cudaSuccess;
    std::call_once(once[device & 63], [&] {
        err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        // An SM changes its split of L1 and shared memory only while it is idle: with the split left to each kernel, the next launch's blocks go
        // two to an SM where there happens to be room (fp16 MLP, one row, 4096 / 11008: 29 us instead of 18).
        if (err == cudaSuccess) err = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    });
    BT_TRY(err);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(BT_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = p.pdl ? 1 : 0;
    BT_TRY(cudaLaunchKernelEx(&cfg, kern, p));
    note_launch();
    return TLLM_OK;
}

// Rows on 16 bytes are shared only where the columns are cut (bits_share), which leaves a warp two groups or more, of four blocks of columns of B one.
template <int XT, bool ASYNC, bool SHARED>
int pick(const BitsParams& p, int nb, int gr, int grid, size_t smem, int device, cudaStream_t st) {
    if constexpr (!ASYNC || !SHARED) {
        if (nb == 1 && gr == 1) return launch<XT, 1, 1, ASYNC, SHARED>(p, grid, smem, device, st);
        if (nb == 2 && gr == 1) return launch<XT, 2, 1, ASYNC, SHARED>(p, grid, smem, device, st);
        if constexpr (XT == TLLM_F32) {
            if (nb == 3 && gr == 1) return launch<XT, 3, 1, ASYNC, SHARED>(p, grid, smem, device, st);
        }
    }
    if (nb == 1 && gr == 2) return launch<XT, 1, 2, ASYNC, SHARED>(p, grid, smem, device, st);
    if (nb == 1 && gr == 3) return launch<XT, 1, 3, ASYNC, SHARED>(p, grid, smem, device, st);
    if (nb == 2 && gr == 2) return launch<XT, 2, 2, ASYNC, SHARED>(p, grid, smem, device, st);
    if constexpr (XT == TLLM_I8) {
        if (nb == 4 && gr == 1) return launch<XT, 4, 1, ASYNC, SHARED>(p, grid, smem, device, st);
    }
    if constexpr (XT == TLLM_F32) {
        if (nb == 3 && gr == 2) return launch<XT, 3, 2, ASYNC, SHARED>(p, grid, smem, device, st);
    }
    return fail(TLLM_ERR_ARG, "bits_launch: no kernel for %d x %d", nb, gr);
}

}  // namespace

// How a product is cut.  One pass over the widest block's columns if GR = 3 (two for more than eight columns of B) and a split of up to four allow it; the
// narrowest split that does: every part of a split fetches the activations anew, or reads the shared ones again, and adds up fewer warps' sums.
namespace {
int dtype_bytes(int x_dtype) { return x_dtype == TLLM_F32 ? 4 : x_dtype == TLLM_I8 ? 1 : 2; }
struct BitsPlan {
    int nb, own, own_more, split_log, per_pass, passes, gr, pairs;     // pairs: pairs of slices a warp goes through, all passes together
};
BitsPlan bits_plan(int x_dtype, int rows, int columns, int kb, int sms) {
    BitsPlan q;
    const int cols = x_dtype == TLLM_F32 ? 3 * rows : rows, groups = (columns + 15) / 16;     // fp32: three bf16 columns a row
    q.nb = (cols + 7) / 8;
    if (x_dtype == TLLM_I8 && q.nb > 2) q.nb = 4;
    q.own = groups / sms, q.own_more = groups % sms;
    const int most = q.nb == 4 ? 1 : q.nb > 1 ? 2 : 3, own = q.own + (q.own_more ? 1 : 0);
    q.split_log = own <= most ? 0 : own <= 2 * most ? 1 : 2;
    const int split = 1 << q.split_log, passes = (own + split * most - 1) / (split * most), kparts = BT_WARPS / split;
    q.passes = passes, q.per_pass = (own + passes - 1) / passes;
    q.gr = (q.per_pass + split - 1) / split;
    q.pairs = ((kb + 1) / 2 + kparts - 1) / kparts * passes;
    return q;
}
// Whether the warps of a block share X in shared memory, loaded once a row by the TMA unit (rows that start anywhere and columns: by all threads),
// or each fetches its own pairs of slices of it.  Sharing saves what every part of a split, and every pass, would fetch again; a block's
// barrier and the later start cost 0.2 to 0.5 us, which a warp of a few pairs does not win back.  (16 rows of fp16 on 4096 x 11008 9.7 us, 12.1 apart;
// one on 8192 x 10240 9.3 and 10.3; 32 rows of int8 on 2048 x 8192 5.8 and 6.8, but 4.2 and 3.8 on 768 x 6912; 16 of fp16 on 2048 x 2048,
// no split, 3.1 and 2.7.  Two rows of fp16 on odd addresses, 2048 x 16384, 5.5 and 7.8; two columns of fp32 on 4096 x 11008 9.5 and 16.4.)
// Without a split the warps of rows and columns that start anywhere fetch nothing twice.  Shared, their loads of columns lie beside one another, and all 512 threads
// take part where K is short.  (Apart and shared, columns: nine of int8 on 1344 x 1152 12.1 and 6.5, seven of fp16 on 1183 x 332 5.5 and 3.7, four of fp32 on
// 616 x 3880 5.6 and 4.4; odd addresses: 24 rows of int8 on 1615 x 2056 5.8 and 4.9, six of fp16 on 440 x 4480 3.4 and 2.8, seven of fp32 on 216 x 1792
// 4.9 and 3.5.  Up to four columns of int8 over a short K lose 6 %, two of fp16 3 %, rows of fp32 over a longer K 4 %.)
bool bits_share(int x_dtype, BitsAccess access, bool async, const BitsPlan& q, int kp, int rows) {
    if (q.passes > 1) return true;
    if (!async && q.split_log > 0) return true;
    if (access == BITS_COLUMNS) return rows > 4 || kp > 16 || (rows > 2 ? x_dtype != TLLM_I8 : x_dtype == TLLM_F32 && kp <= 10);
    if (!async) return x_dtype == TLLM_I8 || (x_dtype == TLLM_F32 ? rows > 2 && kp <= 10 : rows > 2 || kp > 10);
    const bool two_bytes = x_dtype == TLLM_F16 || x_dtype == TLLM_BF16;
    if (q.split_log == 2) return q.pairs > 2;
    return q.split_log == 1 && (q.pairs > 4 || (q.pairs == 4 && two_bytes) || (q.pairs > 1 && (q.nb == 3 || (q.nb == 2 && two_bytes))));
}
// The whole cut of a launch.  Shared memory: X for all warps together, or a warp's pairs of it beside those of W.  Of these as many in flight as a warp has to
// fetch and as there is room for.
struct BitsCut : BitsPlan {
    bool async, share;             // X by rows that start on 16 bytes and are a multiple of them long; whether the warps share it
    int x_chunks, x_pairs, depth, slots;
    uint32_t x_pitch, slot_bytes, ring_at, red_at, bar_at, smem;
};
BitsCut bits_cut(int x_dtype, BitsAccess access, int rows, int inners, int columns, int sms) {
    const int e = dtype_bytes(x_dtype), kb = (inners + 63) / 64, kp = (kb + 1) / 2;
    BitsCut q{bits_plan(x_dtype, rows, columns, kb, sms)};
    q.async = access == BITS_ROWS16 && (size_t)inners * e % 16 == 0;
    q.share = bits_share(x_dtype, access, q.async, q, kp, rows);
    const uint32_t red = (uint32_t)(BT_WARPS >> q.split_log) * q.per_pass * (x_dtype == TLLM_F32 ? 3 * rows : rows) * 80;
    q.x_pitch = (uint32_t)kp * 128 * e + (e == 1 ? 64 : e == 2 ? 16 : 32);
    const auto all_x = [&] { return q.share ? ((size_t)rows * q.x_pitch + 127) / 128 * 128 : 0; };
    const auto slots = [&](int d) { return q.pairs <= d ? q.pairs : d + 1; };
    const auto slot = [&] { return (uint32_t)(q.gr * 512 + (q.share ? 0 : rows * 128 * e)); };
    const auto total = [&](int d) { return all_x() + (size_t)BT_WARPS * slots(d) * slot() + red + BT_BAR_BYTES; };
    if (q.share && total(std::min(q.pairs, 2)) > BT_SMEM_ALL) q.share = false;
    q.x_chunks = kp > 16 && (size_t)rows * inners * e > 16384 ? 2 : 1;
    q.x_pairs = q.x_chunks == 1 ? (kp + 15) / 16 * 16 : ((kp + 1) / 2 + 15) / 16 * 16;
    q.depth = 8;
    while (q.depth > 1 && (q.depth / 2 >= q.pairs || total(q.depth) > BT_SMEM_ALL)) q.depth /= 2;
    q.slots = slots(q.depth), q.slot_bytes = slot();
    q.ring_at = (uint32_t)all_x();
    q.red_at = q.ring_at + (uint32_t)BT_WARPS * q.slots * q.slot_bytes;
    q.bar_at = q.red_at + red;
    q.smem = q.bar_at + BT_BAR_BYTES;
    return q;
}
}  // namespace

// Microseconds of a launch as bits_cut makes it: its start, more of it the more of the sixteen warps have work; per pair of slices that a warp goes through a step
// of its own and what every block of columns of B and group of columns adds; the results; and the activations, of every pair again or, shared,
// of all of K once.  Fitted to 18000 products of 1 to 100 rows on 281 weights from 256 x 256 to 28672 x 8192 in graphs: 7 to 11 % off for rows; up to four
// columns and more of them apart, 8 to 22 %, since the addresses decide there.
double bits_estimate_us(int x_dtype, BitsAccess access, int rows, int inners, int columns, int sms) {
    struct Cost {
        double start, warps, step, groups, results, fetch, fetch_row;       // fetch and fetch_row, not shared: a row of a pair, less of it where blocks are few, and in any case
    };
    static const Cost costs[2][3][4] = {     // warps apart, sharing X; fp32, 16 bits, int8; rows on 16 bytes, rows, more than four columns, up to four
        {{{0.977, 0.904, 1.05, 0.145, 0, 0, 0}, {1.18, 0.781, 0.947, 0.238, 0.22, 0.0149, 0.242}, {0, 0, 0, 0.091, 5.77, 0, 1.7}, {0, 1.65, 0, 0.11, 1.25, 0.137, 1.01}},
         {{1.02, 0.499, 0.565, 0.189, 0.0258, 0, 0}, {0.706, 1.02, 0.953, 0.141, 0.227, 0.0336, 0.13}, {0, 0, 0, 1.08, 3.86, 0, 0.693}, {0.0118, 0.88, 1.69, 0.0865, 0.374, 0.235, 0.0594}},
         {{1.24, 0.431, 0.179, 0.191, 0.0162, 0, 0}, {0, 2.76, 0.725, 0.137, 0.275, 0.0184, 0.0558}, {0, 0, 0.527, 1.09, 2.7, 0.0458, 0.225}, {0, 2.87, 1.34, 0.0302, 0, 0.608, 0}}},
        {{{0, 1.1, 1.56, 0, 0.155, 0, 0.00279}, {1.45, 0.457, 0.946, 0.0593, 0.109, 0.0652, 0.0205}, {1.88, 0.783, 0.715, 0.113, 0.0789, 0.162, 0}, {2.09, 0.0933, 0.311, 0.311, 0.203, 0.0455, 0.0179}},
         {{0, 1.54, 0.655, 0.0522, 0.0795, 0.021, 0}, {1.53, 0.266, 0.496, 0.127, 0.0427, 0.0157, 0.0107}, {1.94, 1.57, 0, 0.294, 0, 0.144, 0}, {2.53, 0, 0.156, 0.297, 0.23, 0.0298, 0.0127}},
         {{2.05, 0.0528, 0.516, 0.0124, 0.0579, 0.00903, 0}, {1.65, 0.145, 0.309, 0.0754, 0.042, 0.0128, 0.00552}, {2.67, 1.06, 0, 0.239, 0, 0.166, 0}, {3.88, 0, 0, 0.337, 0.0102, 0.0042, 0.0139}}}};
    const BitsCut q = bits_cut(x_dtype, access, rows, inners, columns, sms);
    const int type = x_dtype == TLLM_F32 ? 0 : x_dtype == TLLM_I8 ? 2 : 1, how = access == BITS_COLUMNS ? (rows > 4 ? 2 : 3) : q.async ? 0 : 1;
    const Cost& c = costs[q.share][type][how];
    const double groups = (columns + 15) / 16, kp = ((inners + 63) / 64 + 1) / 2, each = kp / (BT_WARPS >> q.split_log);      // each: pairs of a warp and pass, in the mean
    const double pairs = q.passes > 1 ? (q.pairs + q.passes * each) / 2 : q.pairs;        // a warp that has one less goes on with the next pass
    const double fetch = q.share ? kp * (c.fetch + c.fetch_row * rows) : pairs * rows * (c.fetch * std::min(1.0, groups / (access == BITS_COLUMNS ? 128 : 256)) + c.fetch_row);
    // What columns take depends on the addresses (five of fp16 on 512 x 2568 9.7 us, four 5.6 before the warps shared them), so that they are priced above the mean, most
    // where every block reads all of X: of 6400 calls 60 became slower by more than 5 % with these prices in the place of the ones before, 202 without.
    const double doubt = access != BITS_COLUMNS ? 1.0 : rows <= 4 || columns < 1280 || q.split_log == 2 ? 1.1 : q.split_log == 1 ? 1.3 : 1.5;
    return doubt * (c.start + c.warps * std::min(1.0, each) + pairs * (c.step + c.groups * q.nb * q.gr) + c.results * groups * rows / 1000 + fetch);
}

thread_local int bits_last_plan[6];

int bits_launch(BitsParams& p, int sms, int device, void* stream) {
    if (p.x_dtype == TLLM_I8 && p.K >= BT_MAX_INT8_K) return fail(TLLM_ERR_ARG, "bits_launch: int8 over %d inners does not fit into 32-bit sums", p.K);
    const BitsCut q = bits_cut(p.x_dtype, bits_access(p.X, p.x_dtype, p.x_layout, p.x_ld), p.M, p.K, p.N, sms);
    const int nb = q.nb, gr = q.gr, grid = sms, ye = p.y_dtype == TLLM_F32 || p.y_dtype == TLLM_I32 ? 4 : 2;
    p.own = q.own, p.own_more = q.own_more, p.split_log = q.split_log, p.per_pass = q.per_pass;
    p.depth = q.depth, p.slots = q.slots, p.slot_bytes = q.slot_bytes;
    p.x_pairs = q.x_pairs, p.x_chunks = q.x_chunks, p.x_pitch = q.x_pitch, p.x_chunk = (uint32_t)q.x_pairs * 128u * (uint32_t)dtype_bytes(p.x_dtype);
    p.ring_at = q.ring_at, p.red_at = q.red_at, p.bar_at = q.bar_at;
    p.mul4 = 4, p.mul16 = 16;
    p.m_inv = (uint32_t)(((1ull << 32) + p.M - 1) / p.M);
    p.y_wide = p.epilogue == 0 && p.y_step_n == 1 && p.y_step_m % 4 == 0 && p.N % 4 == 0 && (uintptr_t)p.Y % (4 * ye) == 0;
    // A launch keeps an SM to itself.  With room for two blocks, those of the next launch came two to an SM as often as not, while other SMs waited: 4096 x 11008,
    // one row of fp16, called 400 times one after the other, 8.0 us in the median (5.9 to 8.2), alone 6.0 (6.0 to 6.1); an MLP of 2048 / 5632,
    // four rows, 10.7 and 8.5; 8192 x 2048, one row, in a graph 5.0 and 4.0.  What it costs is the next launch's start beside this one: 2048 x 16384,
    // one row, in a graph 4.7 and 5.1.
    const uint32_t smem = std::max(q.smem, BT_SMEM_ALONE);
    if (smem > 227u * 1024u) return fail(TLLM_ERR_ARG, "bits_launch: %u bytes of shared memory", smem);
    const int cut[6] = {gr, nb, 1 << q.split_log, q.passes, q.share ? q.x_chunks : 0, q.depth};
    std::memcpy(bits_last_plan, cut, sizeof cut);
    cudaStream_t st = (cudaStream_t)stream;
#define BT_PICK(XT)                                                                                                               \
    (q.async ? q.share ? pick<XT, true, true>(p, nb, gr, grid, smem, device, st) : pick<XT, true, false>(p, nb, gr, grid, smem, device, st) \
             : q.share ? pick<XT, false, true>(p, nb, gr, grid, smem, device, st) : pick<XT, false, false>(p, nb, gr, grid, smem, device, st))
    switch (p.x_dtype) {
        case TLLM_F32: return BT_PICK(TLLM_F32);
        case TLLM_F16: return BT_PICK(TLLM_F16);
        case TLLM_BF16: return BT_PICK(TLLM_BF16);
        default: return BT_PICK(TLLM_I8);
    }
#undef BT_PICK
}

}  // namespace tllm
