// bits.cu -- instantiations and launches of bits_spmm_kernel (bits_kernel.cuh), in a translation unit of their own so that
// they compile beside the rest.
#include <algorithm>
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

template <int XT, int NB, int GR, bool ASYNC>
int launch(const BitsParams& p, int grid, size_t smem, int device, cudaStream_t st) {
    auto kern = bits_spmm_kernel<XT, NB, GR, ASYNC>;
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

template <int XT, bool ASYNC>
int pick(const BitsParams& p, int nb, int gr, int grid, size_t smem, int device, cudaStream_t st) {
    if (nb == 1 && gr == 1) return launch<XT, 1, 1, ASYNC>(p, grid, smem, device, st);
    if (nb == 1 && gr == 2) return launch<XT, 1, 2, ASYNC>(p, grid, smem, device, st);
    if (nb == 1 && gr == 3) return launch<XT, 1, 3, ASYNC>(p, grid, smem, device, st);
    if (nb == 2 && gr == 1) return launch<XT, 2, 1, ASYNC>(p, grid, smem, device, st);
    if (nb == 2 && gr == 2) return launch<XT, 2, 2, ASYNC>(p, grid, smem, device, st);
    if constexpr (XT == TLLM_I8) {
        if (nb == 4 && gr == 1) return launch<XT, 4, 1, ASYNC>(p, grid, smem, device, st);
    }
    if constexpr (XT == TLLM_F32) {
        if (nb == 3 && gr == 1) return launch<XT, 3, 1, ASYNC>(p, grid, smem, device, st);
        if (nb == 3 && gr == 2) return launch<XT, 3, 2, ASYNC>(p, grid, smem, device, st);
    }
    return fail(TLLM_ERR_ARG, "bits_launch: no kernel for %d x %d", nb, gr);
}

}  // namespace

// How a product is cut.  One pass over the widest block's columns if GR = 3 (two for more than eight columns of B: 64 and 128
// registers) and a split of up to four allow it; the narrowest split that does, because every part of a split fetches the
// activations anew.
namespace {
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
}  // namespace

// Microseconds of a launch: a chain of 2 us, and per pair of slices that a warp goes through what it takes sixteen warps to fetch and
// turn the activations and to decode and multiply the columns, more of it where the activations are fetched once a pass.  Measured at 1 to 16 rows of 2048 x 2048 .. 8192 x 10240.
// Activations that cp.async cannot read pass through registers with every pair, and the blocks wait for them: 2.7 us a pair where 16 rows of
// fp16 start anywhere (bytes 1.6, 8 rows of fp32 2.4), and element by element from a column-major X, by all blocks
// from the same lines (16 rows of fp16, 4096 x 11008: 227 us; the batched kernel behind its planes 18.5).  Measured over the
// same sizes, 1 to 16 rows.
double bits_estimate_us(int x_dtype, BitsAccess access, int rows, int columns, int kb, int sms) {
    const BitsPlan q = bits_plan(x_dtype, rows, columns, kb, sms);
    const bool f32 = x_dtype == TLLM_F32, i8 = x_dtype == TLLM_I8;
    double step = f32 ? q.nb * (0.6 + 0.18 * q.gr) : !i8 || access != BITS_ROWS16 ? 0.25 + q.nb * (0.15 + 0.2 * q.gr) : q.nb == 4 ? 1.3 : 0.1 + q.nb * (0.02 + 0.16 * q.gr);
    const double groups = (columns + 15) / 16;               // of few columns few blocks read X
    if (access == BITS_ROWS) step += std::min(1.0, 0.6 + groups / 256) * (f32 ? 0.6 + 0.23 * rows : i8 ? 0.7 + 0.055 * rows : 0.35 + 0.15 * rows);
    else if (access == BITS_COLUMNS)
        step += std::min(1.0, 0.1 + groups / 128) * (i8 ? 1.6 + 0.5 * rows : (f32 ? 1.7 : 1.1) * rows * (rows <= 4 ? 0.65 : 1.0));
    return 2.0 + q.pairs * (step + (q.passes > 1 ? 0.15 : 0.0));
}

int bits_launch(BitsParams& p, int sms, int device, void* stream) {
    const int e = p.x_dtype == TLLM_F32 ? 4 : p.x_dtype == TLLM_I8 ? 1 : 2;
    const bool async = bits_access(p.X, p.x_dtype, p.x_layout, p.x_ld) == BITS_ROWS16;
    const BitsPlan q = bits_plan(p.x_dtype, p.M, p.N, p.KB, sms);
    const int nb = q.nb, gr = q.gr, grid = sms, kparts = BT_WARPS >> q.split_log, cols = p.x_dtype == TLLM_F32 ? 3 * p.M : p.M, pairs = q.pairs;
    p.own = q.own, p.own_more = q.own_more, p.split_log = q.split_log, p.per_pass = q.per_pass;
    p.mul4 = 4, p.mul16 = 16;
    p.m_inv = (uint32_t)(((1ull << 32) + p.M - 1) / p.M);
    p.slot_bytes = (uint32_t)(gr * 512 + p.M * 128 * e);
    // Pairs in flight: as many as a warp has to fetch and half of the shared memory holds (so that the next launch fits
    // beside this one); where not even two fit there, up to all of it.
    const size_t red = (size_t)kparts * p.per_pass * cols * 80;
    auto slots = [&](int d) { return pairs <= d ? pairs : d + 1; };
    auto total = [&](int d) { return (size_t)BT_WARPS * slots(d) * p.slot_bytes + red; };
    p.depth = 8;
    while (p.depth > 1 && (p.depth / 2 >= pairs || total(p.depth) > BT_SMEM_SHARED)) p.depth /= 2;
    if (p.depth == 1 && pairs > 1 && total(2) <= 220u * 1024u) p.depth = 2;
    p.slots = slots(p.depth);
    // A launch of some length keeps an SM to itself: behind one that does not fit beside it, its blocks would start two to an SM while
    // others wait (fp16 MLP, four rows, 4096 / 11008: 24 us instead of 19).
    size_t smem = total(p.depth);
    if (pairs > 4) smem = std::max(smem, (size_t)BT_SMEM_ALONE);
    if (smem > 227u * 1024u) return fail(TLLM_ERR_ARG, "bits_launch: %zu bytes of shared memory", smem);
    cudaStream_t st = (cudaStream_t)stream;
#define BT_PICK(XT) (async ? pick<XT, true>(p, nb, gr, grid, smem, device, st) : pick<XT, false>(p, nb, gr, grid, smem, device, st))
    switch (p.x_dtype) {
        case TLLM_F32: return BT_PICK(TLLM_F32);
        case TLLM_F16: return BT_PICK(TLLM_F16);
        case TLLM_BF16: return BT_PICK(TLLM_BF16);
        default: return BT_PICK(TLLM_I8);
    }
#undef BT_PICK
}

}  // namespace tllm
