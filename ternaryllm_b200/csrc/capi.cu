// capi.cu -- the C ABI of libtllm (declared in include/tllm.h): handles, launches, host staging.
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include <cudaTypedefs.h>

#include "attn_kernel.cuh"
#include "bits_kernel.cuh"
#include "bstream_kernel.cuh"
#include "kernels.cuh"
#include "lists_kernel.cuh"
#include "mma_kernel.cuh"
#include "mma_units4_kernel.cuh"
#include "nibble_format.h"
#include "nibble_kernel.cuh"
#include "nibble_rows_kernel.cuh"
#include "util.h"

namespace tllm {

static thread_local std::string g_err;
static std::atomic<int64_t> g_launches{0};

int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

#define CU_TRY(expr)                                                                                       \
    do {                                                                                                   \
        cudaError_t e_ = (expr);                                                                           \
        if (e_ != cudaSuccess) return fail(TLLM_ERR_CUDA, "%s failed: %s", #expr, cudaGetErrorString(e_)); \
    } while (0)

static size_t dtype_size(int dt) {
    switch (dt) {
        case TLLM_F32: case TLLM_I32: return 4;
        case TLLM_F16: case TLLM_BF16: return 2;
        case TLLM_I8: return 1;
    }
    return 0;
}

// Which kernel takes a call: -1 = decide per call from a cost model of the two kernels (the default), 0 = never the
// tensor-core kernel, n > 0 = from n activation rows on.  TLLM_MMA_MIN_ROWS sets the initial value.
static std::atomic<int> g_mm_min_rows{-2};
static std::atomic<int64_t> g_mm_launches{0};
static thread_local int g_mm_last_plan[5];      // of this thread's last launch: tllm_mma_last_plan
static std::atomic<int64_t> g_bits_launches{0};
static int mm_min_rows() {
    int v = g_mm_min_rows.load(std::memory_order_relaxed);
    if (v == -2) {
        const char* e = getenv("TLLM_MMA_MIN_ROWS");
        v = e ? atoi(e) : -1;
        if (v < -1) v = -1;
        g_mm_min_rows.store(v, std::memory_order_relaxed);
    }
    return v;
}
// Cost model measured on B200 (CUDA-graph replays of back-to-back products, weights streamed from HBM), microseconds:
// a gather launch of up to four rows costs about GATHER_FIXED + nnz * g(rows padded to 1, 2, 4), more rows take
// ceil(rows / 4) launches; the decode tensor-core kernel is modelled below, the two kernels on bit tiles beside theirs.
static const double GATHER_FIXED_US = 2.9;
static const double GATHER_PS_PER_NNZ[3] = {0.48, 0.68, 1.35};
// The decode tensor-core kernel: -1 = cost model, 0 = never, n > 0 = always for calls of up to n rows.
static std::atomic<int> g_nb_max_rows{-1};
static std::atomic<int64_t> g_nb_launches{0};
#ifdef NB_DEBUG
static int g_nb_debug_tx = 0;   // diagnostic builds only: bytes a weight tile's copy is expected to report
static int g_nb_debug_stages = 0, g_nb_debug_flags = 0;
#endif
// one launch of the decode tensor-core kernel: half a byte per entry at 5.2 TB/s around 6.7 us of start-up (building B
// once the preceding kernel has finished) and hand-over between blocks, 0.9 us more for every further row
static const double NB_FIXED_US = 6.7, NB_ROW_US = 0.9, NB_US_PER_ENTRY = 0.5 / 5.2e6;
static double gather_model_us(int64_t nnz, int rows) {
    const int full = rows / 4, tail = rows % 4;
    const int idx = tail <= 1 ? 0 : (tail == 2 ? 1 : 2);
    return full * (GATHER_FIXED_US + nnz * GATHER_PS_PER_NNZ[2] * 1e-6) + (tail ? GATHER_FIXED_US + nnz * GATHER_PS_PER_NNZ[idx] * 1e-6 : 0.0);
}
// more rows than one such launch takes: the pieces kernel + the many-row kernel, up to 64 (32 fp32) rows per launch.
// Measured per launch with 32 / 64 / 128 / 256 piece rows: start-up and hand-over grow with the rows, and the stream
// slows down as the B tiles it re-reads from L2 and the MMAs grow with the piece rows.
static const double NR_FIXED_US[4] = {13.5, 19.2, 26.9, 42.6}, NR_US_PER_MENTRY[4] = {0.081, 0.075, 0.090, 0.158};
static double nibble_model_us(int64_t entries, int rows, int rows_per_launch) {
    if (rows <= rows_per_launch) return NB_FIXED_US + entries * NB_US_PER_ENTRY + (rows - 1) * NB_ROW_US;
    const int per2 = rows_per_launch * (NR_MAX_NB / NB_ROWS), pieces = NB_ROWS / rows_per_launch;
    double t = 0;
    for (int r0 = 0; r0 < rows; r0 += per2) {
        const int m = rows - r0 < per2 ? rows - r0 : per2;
        int i = 0;
        while ((32 << i) < m * pieces) ++i;
        t += NR_FIXED_US[i] + entries * 1e-6 * NR_US_PER_MENTRY[i];
    }
    return t;
}

}  // namespace tllm

using namespace tllm;

struct tllm_weight {
    BsLayout lay;
    float scale = 1.f;
    int device = 0;
    int max_rows = 4;                 // rows of one gather launch
    uint32_t max_meta_words = 0;      // longest block table
    uint4* d_stream = nullptr;
    uint32_t* d_meta = nullptr;
    TsCtaDesc* d_cta = nullptr;
    void* d_partial = nullptr;
    unsigned int* d_counters = nullptr;
    int* d_status = nullptr;
    size_t stream_bytes = 0, meta_bytes = 0, scratch_bytes = 0;
    // staging for the host-buffer entry points
    void* d_x = nullptr;
    void* d_y = nullptr;
    void* d_bias = nullptr;
    int* h_status = nullptr;        // pinned copy of the status word, read back with every host-buffer call
    size_t x_cap = 0, y_cap = 0, bias_cap = 0;
    cudaStream_t own_stream = nullptr;
    cudaEvent_t part_event[TLLM_HOST_PARTS] = {};       // tllm_spmm_host_parts: a piece of the result has arrived
    // tensor-core kernel: dense two-bit copy of W and its split scratch
    uint4* d_bits = nullptr;
    float* d_mm_partial = nullptr;
    unsigned int* d_mm_counters = nullptr;
    size_t bits_bytes = 0;
    CUtensorMap bits_map[2];
    int mm_n_tiles = 0, mm_kb = 0, mm_grid = 0;
    // decode tensor-core kernel: transposed four-bit copy of W, its tensor map, schedule and hand-over scratch
    uint8_t* d_nib = nullptr;
    size_t nib_bytes = 0;
    CUtensorMap nib_map;
    int nb_kb = 0, nb_kbs = 0, nb_splits = 0, nb_tiles = 0, nb_gj = 0, nb_uk = 2;
    float* d_nb_partial = nullptr;
    unsigned int* d_nb_counters = nullptr;
    uint32_t* d_nb_sched = nullptr;
    // many-row variant: the activation pieces of a call, their tensor maps (32 / 64 / 128 / 256 piece rows), scratch
    uint8_t* d_nr_pieces = nullptr;
    float* d_nr_row_pow = nullptr;
    float* d_nr_partial = nullptr;
    unsigned int* d_nr_counters = nullptr;
    CUtensorMap nr_map[4];
    int nb_k_pad = 0, nr_grid = 0;
};

// What the two kernels that read bit tiles need of a weight: a handle's, or one made for a single call (tllm_ter_spmm).
struct BitsView {
    const uint4* bits;
    const CUtensorMap* map;       // bit tiles in boxes of a unit: [0] two slices, [1] four (mma_units4_kernel)
    int inners, columns, n_tiles, kb, sms, device;
    float* partial;               // 2 * sms hand-over slots for row tiles of up to MM_OWN_NT, or NULL
    unsigned int* counters;       // n_tiles * MM_MAX_M_TILES * 4, zero between launches
    int* status;
    bool lists;                   // made from lists by the preceding kernel: the product has to wait for it; else the tiles were there before
    bool fresh;                   // lists: nothing has been launched since
};

struct tllm_mlp {
    tllm_weight* gate_up = nullptr;   // columns interleaved: 2c = gate column c, 2c+1 = up column c
    tllm_weight* down = nullptr;
    int hidden = 0, inter = 0;
    float s_gate = 1.f, s_up = 1.f;
    void* d_h = nullptr;              // never replaced: graphs that were captured with it hold its address
    size_t h_cap = 0;
    // staging for the host-buffer entry point, grown as needed
    void* d_x = nullptr;
    void* d_y = nullptr;
    void* d_hh = nullptr;
    size_t x_cap = 0, y_cap = 0, hh_cap = 0;
};

namespace {

// scratch of one gather launch: the handle's own, or the library's built-in array (tllm_spmm_static_scratch)
struct Scratch {
    void* partial;
    unsigned int* counters;
};

template <typename ACC, int MP>
int launch_bs(const BsParams& p, int grid, size_t smem, cudaStream_t st) {
    auto kern = bstream_spmm_kernel<ACC, MP>;
    static std::mutex mu;
    static bool configured[64] = {};
    int dev = 0;
    CU_TRY(cudaGetDevice(&dev));
    {
        std::lock_guard<std::mutex> lk(mu);
        if (dev < 64 && !configured[dev]) {
            CU_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            configured[dev] = true;
        }
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(BS_WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CU_TRY(cudaLaunchKernelEx(&cfg, kern, p));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return TLLM_OK;
}

int check_types(int x_dtype, int y_dtype, const char* who) {
    if (x_dtype == TLLM_I8) {
        if (y_dtype != TLLM_I32) return fail(TLLM_ERR_ARG, "%s: int8 activations produce int32 results (y_dtype must be TLLM_I32)", who);
        return TLLM_OK;
    }
    if (x_dtype != TLLM_F32 && x_dtype != TLLM_F16 && x_dtype != TLLM_BF16) return fail(TLLM_ERR_ARG, "%s: unsupported x_dtype %d", who, x_dtype);
    if (y_dtype != TLLM_F32 && y_dtype != TLLM_F16 && y_dtype != TLLM_BF16) return fail(TLLM_ERR_ARG, "%s: unsupported y_dtype %d", who, y_dtype);
    return TLLM_OK;
}

// The handle's buffers live on one device; a call made with another device current would launch there with
// pointers from two GPUs.
int check_device(const tllm_weight* w, const char* who) {
    int dev = 0;
    CU_TRY(cudaGetDevice(&dev));
    if (dev != w->device) return fail(TLLM_ERR_ARG, "%s: the weight lives on device %d but device %d is current", who, w->device, dev);
    return TLLM_OK;
}

// ---- tensor-core path -----------------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

BitsView bits_view(const tllm_weight* w) {
    return BitsView{w->d_bits, w->bits_map, w->lay.inners, w->lay.columns, w->mm_n_tiles, w->mm_kb, w->mm_grid, w->device, w->d_mm_partial, w->d_mm_counters, w->d_status, false, false};
}

// true when TMA can read the activations where they are (rows on 16 bytes; a box is 64 values wide)
bool mm_direct(int inners, const void* X, int x_dtype, int x_layout, int x_ld) {
    return (x_dtype == TLLM_F16 || x_dtype == TLLM_BF16) && x_layout == TLLM_ROW_MAJOR && (uintptr_t)X % 16 == 0 && (size_t)x_ld * 2 % 16 == 0 &&
           inners >= MM_TILE_K;
}

// true when the batched tensor-core kernel is pinned: for fp16 / bf16 row-major activations whose rows TMA can address
bool mm_pinned(const tllm_weight* w, const void* X, int x_dtype, int x_layout, int x_ld, int rows) {
    const int thr = mm_min_rows();
    return thr > 0 && rows >= thr && w->d_bits && mm_direct(w->lay.inners, X, x_dtype, x_layout, x_ld) && tensor_map_encoder() != nullptr;
}

// ---- workspace of one call ---------------------------------------------------------------------------------------------
// Stream-ordered allocations from a pool of the library's own (one per device): a call takes what it needs, frees it behind its
// last kernel in stream order, and the next call on the stream gets the same memory without a synchronisation.  The pool
// is thread-safe, keeps at most WS_KEEP_BYTES across synchronisations and is trimmed to nothing when the last handle goes, or, where
// there never was one, by tllm_ter_spmm_forget(NULL, NULL).
constexpr uint64_t WS_KEEP_BYTES = 256ull << 20;
std::mutex g_ws_mu;
cudaMemPool_t g_ws_pool[64] = {};
std::atomic<int> g_handles{0};

int ws_pool(int device, cudaMemPool_t* out) {
    std::lock_guard<std::mutex> lk(g_ws_mu);
    if (device < 0 || device >= 64) return fail(TLLM_ERR_ARG, "device ordinal %d out of range", device);
    if (!g_ws_pool[device]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        cudaMemPool_t pool = nullptr;
        // the first call may come under stream capture, where making a pool is refused unless the thread says that it does not mind
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        CU_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
        uint64_t keep = WS_KEEP_BYTES;
        cudaError_t made = cudaMemPoolCreate(&pool, &props);
        if (made == cudaSuccess) made = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        CU_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
        CU_TRY(made);
        g_ws_pool[device] = pool;
    }
    *out = g_ws_pool[device];
    return TLLM_OK;
}
void ws_trim() {
    std::lock_guard<std::mutex> lk(g_ws_mu);
    for (cudaMemPool_t pool : g_ws_pool)
        if (pool) cudaMemPoolTrimTo(pool, 0);
}
struct Workspace {
    void* ptr = nullptr;
    cudaStream_t st = nullptr;
    int take(int device, size_t bytes, cudaStream_t stream) {
        cudaMemPool_t pool = nullptr;
        const int rc = ws_pool(device, &pool);
        if (rc) return rc;
        st = stream;
        CU_TRY(cudaMallocFromPoolAsync(&ptr, bytes, pool, stream));
        return TLLM_OK;
    }
    ~Workspace() {
        if (ptr) cudaFreeAsync(ptr, st);
    }
};

// How a product of `rows` rows (in `planes` planes) is cut: by which of the two kernels, row tiles of Nt rows each, and whole tiles, equal
// ranges of units, or a cluster per tile; by one block or by a pair of blocks.  Chosen by one estimate of what the call takes, microseconds, the
// kernel that makes planes included (`staged`: most of the product's start hides behind it); the choice between this product and the other kernels
// goes by the same figure.  Fitted to 21000 measured plans (100 weights from 256 x 256 to 8192 x 10240, 8 to 2048 rows, one plane and three): 3 % off
// in the mean.  (Separate estimates for the two choices, fitted to fewer and larger calls, picked plans 2 % slower than the best measured in the
// mean, now 0.5; 24 rows of fp16 on 1280 x 465 took 7.5 us where units of four slices take 5.7.)  In clocks of 1.85 GHz:
// Units of two slices: eight MMAs of 128 x (planes * Nt) x 16.  A block by itself takes as long as its shared memory needs to write and read the
// activations, a pair half of that; neither takes less than the 700 to 780 of decoding a unit.  A tile's epilogue is hidden behind the next one where
// that takes longer.
// Units of four slices: a slice never takes less than 250; where there is no room for two sets of accumulators a tile's epilogue and legs are not
// hidden.
// In a tile that `parts` blocks share the last one to arrive reads the other parts, a round trip to L2 for every sixteen rows of each.
// A cluster of C blocks per tile: every block's units, then what goes to the other blocks and the adding-up of its own share.
// A million results take half a microsecond to store, a million activations as much to turn into planes.
// A launch that holds more than half of the SMs, or of the clusters that fit, keeps the next one's blocks, one to an SM, from starting up beside it.
struct MmPlan {
    int Nt, m_tiles, split, cluster;
    int cg;                  // blocks that share a tile's MMAs: 1, or 2 (a pair: 256 columns of W, half of the activations in each block)
    bool units4;             // mma_units4_kernel
    double us;
};
constexpr int MM_SMEM = 227 * 1024;
// shared memory beside the units of B: bit tiles, barriers, a cluster's parts, the sum of the legs of three planes
int mm_other_bytes(int nt, int planes, int cluster, bool units4) {
    const int parts = cluster > 1 ? cluster * ((nt / 16 + cluster - 1) / cluster) * 8192 : 0;
    return 1024 + 512 + (units4 ? MS_RAW_UNITS * MS_UNIT_BYTES : MM_RAW_UNITS * MM_UNIT_BYTES) + parts + (planes > 1 && !units4 ? nt * 512 : 0);
}
using MmKernel = void (*)(CUtensorMap, CUtensorMap, MmParams);
MmKernel mm_kernel(int cg, bool units4, bool pairs) { return units4 ? mma_units4_kernel : cg == 1 ? mma_spmm_kernel<1> : pairs ? mma_spmm_kernel<2, true> : mma_spmm_kernel<2>; }
// clusters of `cluster` blocks (cg = 2: of one, two or four pairs) that fit on the device at a time: they do not span the groups of 16 to 20 SMs that a
// GPU is made of
int mm_clusters(int cluster, int cg, bool units4, int sms, int device) {
    static std::atomic<int> known[64][18];
    const int slot = (units4 ? 9 : 0) + (cg == 2 ? cluster - 1 : cluster);      // 2, 4, 8; pairs 1, 3, 7
    const MmKernel kern = mm_kernel(cg, units4, cg == 2 && cluster > 2);
    int n = device < 64 ? known[device][slot].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(sms / cluster * cluster));
        cfg.blockDim = dim3(units4 ? MS_THREADS : MM_THREADS);
        cfg.dynamicSmemBytes = MM_SMEM;
        cudaLaunchAttribute at[1] = {};
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)cluster, at[0].val.clusterDim.y = 1, at[0].val.clusterDim.z = 1;
        cfg.attrs = at, cfg.numAttrs = 1;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MM_SMEM) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
            cudaGetLastError();
            return 0;                                // no clusters for this call; the next one asks again
        }
        if (device < 64) known[device][slot].store(n, std::memory_order_relaxed);
    }
    return n;
}
int mm_max_nt(int planes) { return planes == 1 ? MM_MAX_COLS : MM_MAX_COLS / 3; }
// staged: planes made by the preceding kernel from rows (MM_FROM_ROWS) or columns (MM_FROM_COLUMNS).  asked: false where the device did not say how
// many clusters fit.
enum { MM_READY, MM_FROM_ROWS, MM_FROM_COLUMNS };
MmPlan mm_make_plan(int rows, int planes, int staged, int n_tiles, int kb, int sms, int device, bool* asked) {
    const auto clusters = [&](int c, int cg, bool units4) {
        const int n = mm_clusters(c, cg, units4, sms, device);
        if (n == 0) *asked = false;
        return n;
    };
    MmPlan best{0, 0, 0, 1, 1, false, 0};
    const bool one = planes == 1;
    const auto take = [&](int nt, int mt, int split, int c, int cg, bool units4, double start, double clocks) {
        const double us = start + clocks / 1850.0;
        if (best.Nt == 0 || us < best.us) best = MmPlan{nt, mt, split, c, cg, units4, us};
    };
    const double crowded = staged == MM_FROM_ROWS ? 900.0 : staged ? 2200.0 : 2500.0;
    const double results = (double)rows * n_tiles * MM_TILE_N / 1e6, planes_us = staged ? 0.55 * rows * kb * MM_TILE_K / 1e6 : 0.0;
    const double start2 = (!staged ? 1.3 : one ? 5.1 : 5.2) + 0.6 * results + planes_us, start4 = (!staged ? 1.7 : one ? 5.3 : 5.6) + 0.4 * results + planes_us;
    const int kbu = (kb + MM_UK - 1) / MM_UK, kbu4 = (kb + MS_UK - 1) / MS_UK, pairs = n_tiles > 1 ? clusters(2, 2, false) : 0;
    for (int nt = 16; nt <= mm_max_nt(planes); nt += 16) {
        const int mt = (rows + nt - 1) / nt, cols = planes * nt, sixteens = nt / 16, turns = (sixteens + 1) / 2;     // turns: sixteens of an epilogue warp
        if (mt > MM_MAX_M_TILES) continue;
        // units of two slices
        const double piece = one ? 740.0 : 1240.0, epilogue = 2000.0 + turns * piece, legs = one ? 0.0 : ((kbu + MM_LEG - 1) / MM_LEG - 1) * turns * 2000.0;
        const auto crowd = [&](double held, double fit) { return 2 * held > fit ? crowded : 0.0; };
        for (int cg = 1; cg <= 2; ++cg) {
            const double groups = cg == 1 ? sms : pairs, tiles = (double)((n_tiles + cg - 1) / cg) * mt, units = tiles * kbu;
            if (groups <= 0 || nt % (16 * cg) != 0) continue;
            const double unit = cg == 1 ? std::max(706.0, 500.0 + 3.36 * cols) : std::max(780.0, 240.0 + 3.23 * cols), extra = cg == 1 ? 0.0 : 1590.0;
            take(nt, mt, 0, 1, cg, false, start2, extra + (std::ceil(tiles / groups) - 1) * std::max(kbu * unit, epilogue + legs) + kbu * unit + epilogue + crowd(tiles * cg, sms));
            const double blocks = std::min(units, groups), parts = std::min((double)kbu, blocks / tiles + 1.0);
            take(nt, mt, 1, 1, cg, false, start2, extra + std::ceil(units / blocks) * unit + 7170.0 + turns * (4.4 * piece + 320.0 * (parts - 1)) + crowd(blocks * cg, sms));
            for (int c = 2; c * cg <= 8 && c <= kbu; c *= 2) {
                const int fit = clusters(c * cg, cg, false);
                // pairs: not where the last ones' second blocks would do nothing, nor for a few units, which do not pay for their start
                if (cg == 2 && (n_tiles % 2 != 0 || kbu < 16 * c)) continue;
                if (MM_SMEM - mm_other_bytes(nt, planes, c, false) < 2 * cols / cg * 128 * MM_UK || fit < tiles) continue;
                take(nt, mt, 2, c, cg, false, start2, extra + (kbu + c - 1) / c * unit + 6900.0 + sixteens * 400.0 + ((sixteens + c - 1) / c + 1) / 2 * piece + crowd(tiles, fit));
            }
        }
        // units of four slices
        const double tiles = (double)n_tiles * mt, units = tiles * kbu4;
        const double slice = std::max(245.0, one ? 200.0 + 1.26 * cols : 195.0 + 1.8 * cols), piece4 = one ? 520.0 : 580.0, epilogue4 = 1510.0 + sixteens * piece4;
        const bool two = ms_acc_sets(planes, nt) == 2;
        const auto legs4 = [&](double u) { return two || one ? 0.0 : (std::ceil(u / MS_LEG) - 1) * (500 + sixteens * 150.0); };
        const double tile = kb * slice + legs4(kbu4);
        take(nt, mt, 0, 1, 1, true, start4, tile + epilogue4 + (std::ceil(tiles / sms) - 1) * (two ? std::max(tile, epilogue4) : tile + epilogue4) + crowd(tiles, sms));
        const double blocks = std::min(units, (double)sms), parts = std::min((double)kbu4, blocks / tiles + 1.0);
        take(nt, mt, 1, 1, 1, true, start4,
             std::ceil(units / blocks) * MS_UK * slice + legs4(std::min(units / blocks, (double)kbu4)) + 3000.0 + sixteens * (8 * piece4 + 520.0 * (parts - 1)) + crowd(blocks, sms));
        for (int c = 2; c <= 8 && c <= kbu4; c *= 2) {
            const int fit = clusters(c, 1, true);
            if (MM_SMEM - mm_other_bytes(nt, planes, c, true) < 2 * cols * 128 * MS_UK || fit < tiles) continue;
            take(nt, mt, 2, c, 1, true, start4, (kbu4 + c - 1) / c * MS_UK * slice + legs4((kbu4 + c - 1) / c) + 5110.0 + sixteens * 470.0 + (sixteens + c - 1) / c * piece4 + crowd(tiles, fit));
        }
        if (nt >= rows) break;
    }
    return best;
}
// The plan depends on these sizes alone; a thread keeps those of the last sizes it asked for (making one takes 0.1 to 1 us of a call that takes 4).
MmPlan mm_plan(int rows, int planes, int staged, int n_tiles, int kb, int sms, int device) {
    struct Known {
        int rows, planes, n_tiles, kb, sms, device;
        int staged;
        MmPlan plan;
    };
    static thread_local Known known[64];
    const uint32_t h = ((uint32_t)rows * 31u + (uint32_t)n_tiles) * 31u + (uint32_t)kb * 16u + (uint32_t)planes * 4u + (uint32_t)staged;
    Known& e = known[(h * 2654435761u) >> 26];
    if (e.rows == rows && e.planes == planes && e.staged == staged && e.n_tiles == n_tiles && e.kb == kb && e.sms == sms && e.device == device) return e.plan;
    bool asked = true;
    const MmPlan plan = mm_make_plan(rows, planes, staged, n_tiles, kb, sms, device, &asked);
    if (asked) e = Known{rows, planes, n_tiles, kb, sms, device, staged, plan};
    return plan;
}

// X as planes of rows of K values (one plane: two dimensions); a box is 64 values of box_rows rows of every plane
int encode_rows_map(CUtensorMap* map, const void* base, bool bf16, int k, int rows, int planes, size_t pitch_bytes, size_t plane_bytes, int box_rows) {
    const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)rows, (cuuint64_t)planes};
    const cuuint64_t strides[2] = {(cuuint64_t)pitch_bytes, (cuuint64_t)plane_bytes};
    const cuuint32_t box[3] = {MM_TILE_K, (cuuint32_t)box_rows, (cuuint32_t)planes};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult cr = tensor_map_encoder()(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, planes == 1 ? 2 : 3, const_cast<void*>(base), dims, strides,
                                             box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return fail(TLLM_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)cr);
    return TLLM_OK;
}

// bit tiles as rows = groups of sixteen columns of KB * 64 words; a box is a unit: eight groups x two or four slices
int encode_bits_map(CUtensorMap* map, const void* bits, int n_tiles, int kb, int slices) {
    const cuuint64_t dims[2] = {(cuuint64_t)kb * 64, (cuuint64_t)n_tiles * 8};
    const cuuint64_t strides[1] = {(cuuint64_t)kb * 256};
    const cuuint32_t box[2] = {(cuuint32_t)slices * 64, 8}, estr[2] = {1, 1};
    const CUresult cr = tensor_map_encoder()(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(bits), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return fail(TLLM_ERR_CUDA, "cuTensorMapEncodeTiled (bit tiles) failed with code %d", (int)cr);
    return TLLM_OK;
}

cudaLaunchAttribute pdl_attribute() {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    return at;
}

int stage_pad(int k) { return (k + 63) / 64 * 64; }

int run_stage(const void* X, int x_dtype, int x_layout, int x_ld, int rows, int K, unsigned short* out, bool late, cudaStream_t st) {
    StageParams q{X, out, x_dtype, x_layout, x_ld, rows, K, stage_pad(K), late};
    void (*kern)(StageParams) = x_dtype == TLLM_F32 ? stage_acts_kernel<TLLM_F32> : x_dtype == TLLM_I8 ? stage_acts_kernel<TLLM_I8> : stage_acts_kernel<TLLM_F16>;
    cudaLaunchConfig_t cfg{};
    const long long blocks = x_layout == TLLM_ROW_MAJOR ? ((long long)rows * (q.k_pad / 8) + 255) / 256 : (long long)(q.k_pad / 64) * ((rows + 31) / 32);
    cfg.gridDim = dim3((unsigned)blocks);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute at[1] = {pdl_attribute()};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CU_TRY(cudaLaunchKernelEx(&cfg, kern, q));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return TLLM_OK;
}

// X of one launch as the kernel reads it: `planes` planes of 16-bit rows, plane_rows apart, pitch bytes per row
struct MmActs {
    const void* base;
    bool bf16;
    int planes, plane_rows;
    size_t pitch;
    int finite;              // MmParams::finite
    int staged;              // mm_plan
};
struct MmOut {
    void* Y;
    int dtype, ld, epilogue;
    float scale, scale2;
    bool col_major;          // Y[n * ld + m]
    bool planes;             // epilogue 1: three bf16 planes, plane elements apart, instead of dtype
    long long plane;
};

// rows [0, rows) of `x` (at most MM_MAX_M_TILES tiles) in one launch of the tensor-core kernel
int launch_mm(const BitsView& w, const MmActs& x, int rows, const MmOut& o, cudaStream_t st) {
    const MmPlan plan = mm_plan(rows, x.planes, x.staged, w.n_tiles, w.kb, w.sms, w.device);
    MmParams p{};
    p.Y = o.Y;
    p.counters = w.counters;
    p.status = w.status;
    p.M = rows, p.K = w.inners, p.N = w.columns;
    const int uk = plan.units4 ? MS_UK : MM_UK;
    p.KB = w.kb, p.KBU = (p.KB + uk - 1) / uk;
    p.n_tiles = w.n_tiles, p.m_tiles = plan.m_tiles, p.Nt = plan.Nt, p.split = plan.split, p.cluster = plan.cluster;
    p.P = x.planes;
    p.leg = x.planes > 1 ? (plan.units4 ? MS_LEG : MM_LEG) : 1 << 24;
    p.epilogue = o.epilogue, p.y_ld = o.ld, p.plane_y = o.plane;
    p.y_step_n = o.col_major ? o.ld : 1, p.y_step_m = o.col_major ? 1 : o.ld;
    p.out = o.planes ? MM_OUT_PLANES : o.dtype == TLLM_F32 ? MM_OUT_F32 : o.dtype == TLLM_I32 ? MM_OUT_I32 : o.dtype == TLLM_F16 ? MM_OUT_F16 : MM_OUT_BF16;
    if (o.epilogue == 0 && !o.planes) {
        const bool wide = o.dtype == TLLM_F32 || o.dtype == TLLM_I32;
        if (wide && o.col_major && (uintptr_t)o.Y % 16 == 0 && o.ld % 4 == 0) p.out = o.dtype == TLLM_F32 ? MM_OUT_F32_COL4 : MM_OUT_I32_COL4;
        if (!wide && !o.col_major && (uintptr_t)o.Y % 4 == 0 && o.ld % 2 == 0 && w.columns % MM_TILE_N == 0) p.out += MM_OUT_F16_PAIRS - MM_OUT_F16;
    }
    const int cg = plan.cg, b_unit = x.planes * p.Nt / cg * 128 * uk, other = mm_other_bytes(p.Nt, x.planes, p.cluster, plan.units4);
    p.SB = std::min(MM_MAX_STAGES, (MM_SMEM - other) / b_unit);
    p.R = MS_RAW_UNITS;
    p.mul4 = 4, p.mul16 = 16;
    const uint32_t fmt = x.bf16 ? 1u : 0u;
    // instruction descriptor: fp32 accumulate (bits 4-5 = 1), A and B formats (bits 7-9, 10-12), both K-major,
    // N / 8 in bits 17-22, M / 16 in bits 24-28
    p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(x.planes * p.Nt >> 3) << 17) | ((uint32_t)(cg * MM_TILE_N >> 4) << 24);
    p.scale = o.scale * 0.5f, p.scale2 = o.scale2 * 0.5f;          // the decoded weights are +-2
    p.finite = x.finite;
    p.bits = (const uint32_t*)w.bits, p.X = (const unsigned short*)x.base, p.bf16 = x.bf16;
    p.wait_bits = w.lists;
    p.ld_x = (long long)(x.pitch / 2), p.plane_x = x.plane_rows * p.ld_x;

    CUtensorMap map;
    int rc = encode_rows_map(&map, x.base, x.bf16, w.inners, rows, x.planes, x.pitch, (size_t)x.plane_rows * x.pitch, p.Nt / cg);
    if (rc) return rc;
    const size_t smem = (size_t)other + (size_t)p.SB * b_unit;
    if (smem > MM_SMEM || p.SB < 2) return fail(TLLM_ERR_ARG, "tensor-core kernel: ring configuration needs %zu bytes of shared memory", smem);
    const MmKernel kern = mm_kernel(cg, plan.units4, p.split == 2);
    static std::once_flag once[4][64];
    cudaError_t err = cudaSuccess;
    std::call_once(once[plan.units4 ? 2 : cg == 2 && p.split == 2 ? 3 : cg - 1][w.device & 63], [&] { err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MM_SMEM); });
    CU_TRY(err);
    // never more blocks than items: the hand-over between the blocks that share a tile counts on every block in a
    // tile's range of owners holding at least one unit of it
    const long long items = (long long)((p.n_tiles + cg - 1) / cg) * p.m_tiles * (p.split == 1 ? p.KBU : p.cluster);
    const long long most = p.split == 2 ? items : cg == 2 ? mm_clusters(2, 2, false, w.sms, w.device) : w.sms;      // (the plan has seen that a launch's clusters fit)
    const int groups = (int)std::min(items, most), grid = groups * cg, dealt = p.split == 0 ? (p.n_tiles + cg - 1) / cg * p.m_tiles : (p.n_tiles + cg - 1) / cg * p.m_tiles * p.KBU;
    p.share = dealt / groups, p.share_more = dealt % groups, p.g_inv = mm_inverse((uint32_t)groups);
    p.kbu_inv = mm_inverse((uint32_t)p.KBU), p.mt_inv = mm_inverse((uint32_t)p.m_tiles);
    p.cluster_log = p.cluster == 8 ? 3 : p.cluster / 2;
    Workspace ws;
    if ((p.Nt <= MM_OWN_NT && w.partial) || p.split != 1) p.partial = w.partial;
    else {
        rc = ws.take(w.device, (size_t)2 * grid * MM_TILE_N * p.Nt * sizeof(float), st);
        if (rc) return rc;
        p.partial = (float*)ws.ptr;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(plan.units4 ? MS_THREADS : MM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2] = {};
    int n_at = 0;
    at[n_at++] = pdl_attribute();
    if (p.split == 2 || cg == 2) {
        at[n_at].id = cudaLaunchAttributeClusterDimension;
        at[n_at].val.clusterDim.x = (unsigned)(cg * (p.split == 2 ? p.cluster : 1)), at[n_at].val.clusterDim.y = 1, at[n_at].val.clusterDim.z = 1;
        ++n_at;
    }
    cfg.attrs = at;
    cfg.numAttrs = (unsigned)n_at;
    CU_TRY(cudaLaunchKernelEx(&cfg, kern, map, w.map[plan.units4 ? 1 : 0], p));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    g_mm_launches.fetch_add(1, std::memory_order_relaxed);
    const int cut[5] = {uk, cg, p.split, p.cluster, p.Nt};
    std::memcpy(g_mm_last_plan, cut, sizeof cut);
    return TLLM_OK;
}

// fp32 activations that are three planes already ([3][rows][pitch / 2], pitch bytes per row)
int run_mm_planes(const BitsView& w, const unsigned short* planes, int plane_rows, size_t pitch, int rows, void* Y, int y_dtype, int y_ld, float scale, cudaStream_t st) {
    const int per = MM_MAX_M_TILES * mm_max_nt(3);
    for (int r0 = 0; r0 < rows; r0 += per) {
        const int rc = launch_mm(w, MmActs{(const char*)planes + (size_t)r0 * pitch, true, 3, plane_rows, pitch, 1, MM_FROM_ROWS}, std::min(rows - r0, per),
                                 MmOut{(char*)Y + (size_t)r0 * y_ld * dtype_size(y_dtype), y_dtype, y_ld, 0, scale, 0.f, false, false, 0}, st);
        if (rc) return rc;
    }
    return TLLM_OK;
}

// the whole product on the tensor-core kernel: activations that TMA cannot read as they are go through planes in a workspace
int run_mm(const BitsView& w, const void* X, int x_dtype, int x_layout, int x_ld, int rows, void* Y, int y_dtype, int y_ld, int epilogue, float scale,
           float scale2, cudaStream_t st, bool y_col = false, bool y_planes = false, long long plane_y = 0) {
    const int K = w.inners;
    const size_t xe = dtype_size(x_dtype), ye = dtype_size(y_dtype);
    const bool direct = mm_direct(w.inners, X, x_dtype, x_layout, x_ld);
    const int planes = x_dtype == TLLM_F32 ? 3 : 1, per = MM_MAX_M_TILES * mm_max_nt(planes);
    const int finite = x_dtype == TLLM_I8 ? 0 : !direct || w.lists ? 1 : x_dtype == TLLM_BF16 ? 2 : 0;
    Workspace ws;
    if (!direct) {
        const int rc = ws.take(w.device, (size_t)planes * std::min(rows, per) * stage_pad(K) * 2, st);
        if (rc) return rc;
    }
    for (int r0 = 0; r0 < rows; r0 += per) {
        const int m = std::min(rows - r0, per);
        const char* xp = (const char*)X + (x_layout == TLLM_ROW_MAJOR ? (size_t)r0 * x_ld : (size_t)r0) * xe;
        MmActs a{xp, x_dtype == TLLM_BF16 || x_dtype == TLLM_F32, planes, m, (size_t)x_ld * 2, finite, direct ? MM_READY : x_layout == TLLM_ROW_MAJOR ? MM_FROM_ROWS : MM_FROM_COLUMNS};
        if (!direct) {
            const int rc = run_stage(xp, x_dtype, x_layout, x_ld, m, K, (unsigned short*)ws.ptr, w.fresh && r0 == 0, st);
            if (rc) return rc;
            a.base = ws.ptr, a.pitch = (size_t)stage_pad(K) * 2;
        }
        const int rc = launch_mm(w, a, m, MmOut{(char*)Y + (y_col ? (size_t)r0 : (size_t)r0 * y_ld) * (y_planes ? 2 : ye), y_dtype, y_ld, epilogue, scale, scale2, y_col, y_planes, plane_y}, st);
        if (rc) return rc;
    }
    return TLLM_OK;
}

// ---- decode tensor-core path ---------------------------------------------------------------------------------
int nb_rows_per_launch(int x_dtype) { return x_dtype == TLLM_F32 ? NB_ROWS / 8 : NB_ROWS / 4; }

// true when the decode tensor-core kernel can and should take this call
bool nb_fits(const tllm_weight* w, int x_dtype, int x_layout) {
    return w->d_nib && (x_dtype == TLLM_F16 || x_dtype == TLLM_BF16 || x_dtype == TLLM_F32) && x_layout == TLLM_ROW_MAJOR && mm_min_rows() != 0 &&
           g_nb_max_rows.load(std::memory_order_relaxed) != 0;
}
// pinned, or ahead of the gather kernel
bool nb_usable(const tllm_weight* w, int x_dtype, int x_layout, int rows) {
    if (!nb_fits(w, x_dtype, x_layout)) return false;
    const int thr = g_nb_max_rows.load(std::memory_order_relaxed);
    if (thr > 0) return rows <= thr;
    const int64_t entries = (int64_t)w->lay.inners * w->lay.columns;
    return nibble_model_us(entries, rows, nb_rows_per_launch(x_dtype)) < gather_model_us(w->lay.nnz, rows);
}

int upload_nibbles(tllm_weight* w, const int8_t* dense, int inners, int columns, int sms) {
    if (tensor_map_encoder() == nullptr) return TLLM_OK;      // no driver entry point: the handle simply has no such copy
    NbHostImage img;
    nb_pack_dense(dense, inners, columns, &img);
    w->nib_bytes = img.codes.size();
    CU_TRY(cudaMalloc(&w->d_nib, w->nib_bytes));
    CU_TRY(cudaMemcpy(w->d_nib, img.codes.data(), w->nib_bytes, cudaMemcpyHostToDevice));
    const cuuint64_t dims[2] = {(cuuint64_t)img.k_pad, (cuuint64_t)img.n_pad};
    const cuuint64_t strides[1] = {(cuuint64_t)img.k_pad / 2};
    const cuuint32_t box[2] = {NB_TILE_K, NB_TILE_N};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult cr = tensor_map_encoder()(&w->nib_map, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, 2, w->d_nib, dims, strides, box, estr,
                                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) return fail(TLLM_ERR_CUDA, "cuTensorMapEncodeTiled (four-bit weight planes) failed with code %d", (int)cr);
    // One block per SM, two tiles per unit, K ranges of up to 32 blocks.  (Two blocks per SM with one tile per unit and
    // ranges of 16 -- a block's start-up and hand-over overlapping the other's streaming -- measured 5 to 35 % slower.)
    static_assert(NB_FMT_TILE == NB_TILE_K && NB_FMT_TILE == NB_TILE_N && NB_FMT_MAX_KBS == NB_MAX_KBS && NB_FMT_UK == 2,
                  "the host schedule and the kernel (launched as nibble_spmm_kernel<2>) disagree");
    NbSchedule plan;
    nb_make_schedule(img.k_pad, img.n_pad, sms, &plan);
    w->nb_uk = plan.uk, w->nb_kb = plan.kb, w->nb_tiles = plan.tiles, w->nb_kbs = plan.kbs, w->nb_splits = plan.splits, w->nb_gj = plan.gj;
    const std::vector<uint32_t>& sched = plan.words;
    const size_t partial_bytes = (size_t)w->nb_splits * ((size_t)w->nb_tiles + w->nb_gj) * (NB_ROWS / 4) * NB_TILE_N * sizeof(float);
    const size_t counter_bytes = (size_t)w->nb_tiles * 4 * sizeof(unsigned int);
    CU_TRY(cudaMalloc(&w->d_nb_sched, sched.size() * sizeof(uint32_t)));
    CU_TRY(cudaMemcpy(w->d_nb_sched, sched.data(), sched.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    CU_TRY(cudaMalloc(&w->d_nb_partial, partial_bytes));
    CU_TRY(cudaMalloc(&w->d_nb_counters, counter_bytes));
    CU_TRY(cudaMemset(w->d_nb_counters, 0, counter_bytes));
    w->scratch_bytes += partial_bytes + counter_bytes;
    // the many-row variant: pieces of up to NR_MAX_NB piece rows, one tensor map per B height, two hand-over slots per block
    w->nb_k_pad = img.k_pad;
    w->nr_grid = sms;
    const size_t pieces_bytes = (size_t)NR_MAX_NB * img.k_pad, nr_partial_bytes = (size_t)2 * sms * NB_TILE_N * NR_MAX_ROWS * sizeof(float);
    CU_TRY(cudaMalloc(&w->d_nr_pieces, pieces_bytes));
    CU_TRY(cudaMemset(w->d_nr_pieces, 0, pieces_bytes));
    CU_TRY(cudaMalloc(&w->d_nr_row_pow, NR_MAX_ROWS * sizeof(float)));
    CU_TRY(cudaMalloc(&w->d_nr_partial, nr_partial_bytes));
    CU_TRY(cudaMalloc(&w->d_nr_counters, counter_bytes));
    CU_TRY(cudaMemset(w->d_nr_counters, 0, counter_bytes));
    w->scratch_bytes += pieces_bytes + nr_partial_bytes + counter_bytes;
    for (int i = 0; i < 4; ++i) {
        const cuuint64_t pdims[2] = {(cuuint64_t)img.k_pad, (cuuint64_t)NR_MAX_NB};
        const cuuint64_t pstrides[1] = {(cuuint64_t)img.k_pad};
        const cuuint32_t pbox[2] = {NB_TILE_K, (cuuint32_t)(32 << i)};
        const CUresult pr = tensor_map_encoder()(&w->nr_map[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, w->d_nr_pieces, pdims, pstrides, pbox, estr,
                                                 CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                                 CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (pr != CUDA_SUCCESS) return fail(TLLM_ERR_CUDA, "cuTensorMapEncodeTiled (activation pieces) failed with code %d", (int)pr);
    }
    CU_TRY(cudaDeviceSynchronize());
    return TLLM_OK;
}

// more rows than one launch of nibble_spmm_kernel takes: the pieces kernel and the many-row kernel, up to NR_MAX_NB piece rows per pair
int run_nr(tllm_weight* w, const void* X, int x_dtype, int x_ld, int rows, void* Y, int y_dtype, int y_ld, int epilogue, float scale, float scale2,
           cudaStream_t st) {
    const BsLayout& L = w->lay;
    static std::mutex mu;
    static bool configured[64] = {};
    {
        std::lock_guard<std::mutex> lk(mu);
        if (w->device < 64 && !configured[w->device]) {
            CU_TRY(cudaFuncSetAttribute(nibble_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            configured[w->device] = true;
        }
    }
    const int P = x_dtype == TLLM_F32 ? 8 : 4, per = NR_MAX_NB / P;
    const size_t xe = dtype_size(x_dtype), ye = dtype_size(y_dtype);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    for (int r0 = 0; r0 < rows; r0 += per) {
        const int M = rows - r0 < per ? rows - r0 : per;
        int mi = 0;
        while ((32 << mi) < M * P) ++mi;
        const int NB = 32 << mi;
        NpParams q{};
        q.X = (const char*)X + (size_t)r0 * x_ld * xe;
        q.pieces = w->d_nr_pieces;
        q.row_pow = w->d_nr_row_pow;
        q.M = M, q.K = L.inners, q.k_pad = w->nb_k_pad, q.x_dtype = x_dtype, q.x_ld = x_ld, q.P = P;
        cudaLaunchConfig_t c1{};
        c1.gridDim = dim3((unsigned)M);
        c1.blockDim = dim3(256);
        c1.stream = st;
        c1.attrs = at;
        c1.numAttrs = 1;
        CU_TRY(cudaLaunchKernelEx(&c1, nibble_pieces_kernel, q));
        NrParams p{};
        p.row_pow = w->d_nr_row_pow;
        p.Y = (char*)Y + (size_t)r0 * y_ld * ye;
        p.partial = w->d_nr_partial;
        p.counters = w->d_nr_counters;
        p.status = w->d_status;
        p.M = M, p.N = L.columns;
        p.y_dtype = y_dtype, p.y_ld = y_ld, p.epilogue = epilogue;
        p.P = P, p.NB = NB, p.KB = w->nb_kb, p.n_tiles = w->nb_tiles;
        const size_t stage = (size_t)NR_UK * (NB_A_STAGE_BYTES + (size_t)NB * 128);
        p.S = (int)std::min<size_t>(NB_MAX_STAGES, (200 * 1024) / stage);
        p.idesc = (1u << 4) | (5u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) | ((uint32_t)(NB_TILE_N >> 4) << 24);
        p.tmem_cols = (uint32_t)(2 * NB);
        p.scale = scale, p.scale2 = scale2;
        const long long units = (long long)p.n_tiles * ((p.KB + NR_UK - 1) / NR_UK);
        cudaLaunchConfig_t c2{};
        c2.gridDim = dim3((unsigned)(units < w->nr_grid ? units : w->nr_grid));
        c2.blockDim = dim3(NR_THREADS);
        c2.dynamicSmemBytes = 1024 + (size_t)p.S * stage + 1024;
        c2.stream = st;
        c2.attrs = at;
        c2.numAttrs = 1;
        CU_TRY(cudaLaunchKernelEx(&c2, nibble_rows_kernel, w->nib_map, w->nr_map[mi], p));
        g_launches.fetch_add(2, std::memory_order_relaxed);
        g_nb_launches.fetch_add(1, std::memory_order_relaxed);
    }
    return TLLM_OK;
}

// `rows` activation rows through the decode tensor-core kernel: one launch for up to four rows (two for fp32), the many-row
// pair of kernels above that
int run_nb(tllm_weight* w, const void* X, int x_dtype, int x_ld, int rows, void* Y, int y_dtype, int y_ld, int epilogue, float scale, float scale2,
           cudaStream_t st) {
    if (rows > nb_rows_per_launch(x_dtype)) return run_nr(w, X, x_dtype, x_ld, rows, Y, y_dtype, y_ld, epilogue, scale, scale2, st);
    const BsLayout& L = w->lay;
    static std::mutex mu;
    static bool configured[64] = {};
    {
        std::lock_guard<std::mutex> lk(mu);
        if (w->device < 64 && !configured[w->device]) {
            CU_TRY(cudaFuncSetAttribute(nibble_spmm_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
            configured[w->device] = true;
        }
    }
    NbParams p{};
    p.partial = w->d_nb_partial;
    p.counters = w->d_nb_counters;
    p.sched = w->d_nb_sched;
    p.status = w->d_status;
    p.K = L.inners;
    p.N = L.columns;
    p.x_dtype = x_dtype;
    p.x_ld = x_ld;
    p.y_dtype = y_dtype;
    p.y_ld = y_ld;
    p.epilogue = epilogue;
    p.P = x_dtype == TLLM_F32 ? 8 : 4;
    p.KB = w->nb_kb;
    p.KBS = w->nb_kbs;
    p.k_splits = w->nb_splits;
    p.n_tiles = w->nb_tiles;
    p.Gj = w->nb_gj;
    p.S = NB_MAX_STAGES;
    // instruction descriptor: fp32 accumulate (bits 4-5 = 1), A = e2m1 (5, bits 7-9), B = e5m2 (1, bits 10-12), both
    // K-major, N / 8 in bits 17-22, M / 16 in bits 24-28
    p.idesc = (1u << 4) | (5u << 7) | (1u << 10) | ((uint32_t)(NB_ROWS >> 3) << 17) | ((uint32_t)(NB_TILE_N >> 4) << 24);
    p.tmem_cols = 32;
    p.tx_bytes = NB_A_TILE_BYTES;
#ifdef NB_DEBUG
    if (g_nb_debug_tx) p.tx_bytes = (uint32_t)g_nb_debug_tx;
    if (g_nb_debug_stages) p.S = g_nb_debug_stages;
    p.debug = g_nb_debug_flags;
#endif
    p.scale = scale;
    p.scale2 = scale2;
    const size_t smem = 1024 + (size_t)p.S * w->nb_uk * NB_A_STAGE_BYTES + (size_t)p.KBS * NB_ROWS * 128 + 512;
    const size_t xe = dtype_size(x_dtype), ye = dtype_size(y_dtype);
    const int per = nb_rows_per_launch(x_dtype);
    for (int r0 = 0; r0 < rows; r0 += per) {
        p.M = rows - r0 < per ? rows - r0 : per;
        p.X = (const char*)X + (size_t)r0 * x_ld * xe;
        p.Y = (char*)Y + (size_t)r0 * y_ld * ye;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)(p.k_splits * p.Gj));
        cfg.blockDim = dim3(NB_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        CU_TRY(cudaLaunchKernelEx(&cfg, nibble_spmm_kernel<2>, w->nib_map, p));
        g_launches.fetch_add(1, std::memory_order_relaxed);
        g_nb_launches.fetch_add(1, std::memory_order_relaxed);
    }
    return TLLM_OK;
}

// ---- two-bit tiles decoded in registers ----------------------------------------------------------------------------
// rows one launch takes: 16, fp32 (three bf16 values each) 8, int8 32
int bt_rows_per_launch(int x_dtype) { return x_dtype == TLLM_F32 ? BT_MAX_ROWS / 2 : x_dtype == TLLM_I8 ? BT_MAX_ROWS * 2 : BT_MAX_ROWS; }

int run_bits(const BitsView& w, const void* X, int x_dtype, int x_layout, int x_ld, int rows, void* Y, int y_dtype, int y_ld, int epilogue, float scale,
             float scale2, cudaStream_t st, bool y_col = false) {
    BitsParams p{};
    p.pdl = !w.lists;
    p.bits = w.bits, p.status = w.status;
    p.x_dtype = x_dtype, p.x_layout = x_layout, p.x_ld = x_ld;
    p.y_dtype = y_dtype, p.epilogue = epilogue;
    p.y_step_n = y_col ? y_ld : 1, p.y_step_m = y_col ? 1 : y_ld;
    p.K = w.inners, p.N = w.columns, p.KB = w.kb;
    p.scale = scale * 0.5f, p.scale2 = scale2 * 0.5f;            // the decoded weights are +-2
    const size_t xe = dtype_size(x_dtype), ye = dtype_size(y_dtype);
    const int per = bt_rows_per_launch(x_dtype);
    for (int r0 = 0; r0 < rows; r0 += per) {
        p.M = rows - r0 < per ? rows - r0 : per;
        p.X = (const char*)X + (x_layout == TLLM_ROW_MAJOR ? (size_t)r0 * x_ld : (size_t)r0) * xe;
        p.Y = (char*)Y + (size_t)r0 * p.y_step_m * ye;
        const int rc = bits_launch(p, w.sms, w.device, st);
        if (rc) return rc;
    }
    g_bits_launches.fetch_add((rows + per - 1) / per, std::memory_order_relaxed);
    return TLLM_OK;
}

// Cost models of the two kernels that read the two-bit tiles, microseconds.
double bt_model_us(int inners, int columns, int sms, int x_dtype, BitsAccess access, int rows) {
    const int per = bt_rows_per_launch(x_dtype);
    const auto us = [&](int m) { return bits_estimate_us(x_dtype, access, m, inners, columns, sms); };
    return (rows >= per ? rows / per * us(per) : 0.0) + (rows % per ? us(rows % per) : 0.0);
}
double mm_tiles_model_us(int inners, int columns, int sms, int device, bool direct, int x_dtype, BitsAccess access, int rows) {
    const int planes = x_dtype == TLLM_F32 ? 3 : 1, per = MM_MAX_M_TILES * mm_max_nt(planes), staged = direct ? MM_READY : access == BITS_COLUMNS ? MM_FROM_COLUMNS : MM_FROM_ROWS;
    double t = access == BITS_COLUMNS ? 0.1 + 1.3 * rows * inners / 1e6 : 0.0;        // columns take longer to turn into planes
    for (int r0 = 0; r0 < rows; r0 += per)
        t += mm_plan(std::min(rows - r0, per), planes, staged, (columns + 127) / 128, (inners + 63) / 64, sms, device).us;
    // (the plans' figures are from before the batched kernels started earlier; in the mean of 6000 products not far from the decoder's time)
    return t * (direct ? 0.94 : access == BITS_COLUMNS ? 0.91 : 0.89);
}
// which of the two: true = decode in registers
bool bits_prefer_registers(int inners, int columns, int sms, int device, bool direct, int x_dtype, BitsAccess access, int rows) {
    if (rows == 1 && access == BITS_ROWS16) return true;
    if (rows > 8 * BT_MAX_ROWS) return false;
    // (Against the fastest kernel over 18000 drawn products, by type, access and 1, 2 to 4, 5 to 16 and more rows: mean loss 0 to 1 % for rows, 0 to 4 % for columns; 0 to 6 and
    // 0 to 16 % with estimates that counted on shared activations whether or not a launch shares them, and on those of the kernels before.)
    return bt_model_us(inners, columns, sms, x_dtype, access, rows) <= mm_tiles_model_us(inners, columns, sms, device, direct, x_dtype, access, rows);
}

enum KernelChoice { KERNEL_GATHER, KERNEL_MMA, KERNEL_NIBBLE, KERNEL_BITS };
KernelChoice choose_kernel(const tllm_weight* w, const void* X, int x_dtype, int x_layout, int x_ld, int rows) {
    const bool nb = nb_usable(w, x_dtype, x_layout, rows);
    if (nb && g_nb_max_rows.load(std::memory_order_relaxed) > 0) return KERNEL_NIBBLE;     // pinned
    if (mm_pinned(w, X, x_dtype, x_layout, x_ld, rows)) return KERNEL_MMA;
    const int64_t entries = (int64_t)w->lay.inners * w->lay.columns;
    // int8: the batched kernel's fp32 sums are exact while K * 128 stays within 2^24; the register decoder's int32 sums of 64 * x while K stays below
    // 2^18 (BT_MAX_INT8_K), which this bound takes care of too
    if (w->d_bits && mm_min_rows() == -1 && (x_dtype != TLLM_I8 || w->lay.inners <= 131072) && tensor_map_encoder() != nullptr) {
        const int inners = w->lay.inners, columns = w->lay.columns, sms = w->mm_grid;
        const BitsAccess access = bits_access(X, x_dtype, x_layout, x_ld);
        const double bits = bt_model_us(inners, columns, sms, x_dtype, access, rows), gather = gather_model_us(w->lay.nnz, rows);
        const int per = nb_rows_per_launch(x_dtype);
        const bool nibbles = nb_fits(w, x_dtype, x_layout) && rows <= 8 && (rows <= per || access == BITS_ROWS16);
        const double nibble = nibbles ? nibble_model_us(entries, rows, per) : 1e9;
        const auto tiles = [&] { return mm_tiles_model_us(inners, columns, sms, w->device, false, x_dtype, access, rows); };
        // One row of a large, very sparse weight: the index lists are shorter than two bits an entry (13456 x 9088, 90 % zeros, fp32: 13.1 us against 19.0; 4096 x 11008,
        // 95 % zeros, fp16 5.0 against 6.1; 8192 x 57344, 90 % zeros, bf16 34.5 against 44.7).  The gather model is 0.2 too low up to K = 4096, beyond that 0.4 to 0.6 for
        // the largest weights and 0.5 to 0.9 (thrice more) for others, and 0.6 or more for rows on odd addresses.
        // Two rows of int8 too, which the gather kernel reads in either layout, with sums that are exact as well (column-major, 21504 x 5828, 90 % zeros:
        // 16.6 us against 25.8); two columns over a short K as before the decoder's warps shared them (2048 x 8192, 70 % zeros: 6.0 us, 4.3 decoded).
        const bool short_k = inners <= 4096;
        const double gather_times = short_k && access == BITS_ROWS16 ? 1.3 : entries > 150000000 ? 1.6 : 1.85;
        if (columns >= 4096 && rows == 1 && gather_times * gather < std::min(bits, nibble)) return KERNEL_GATHER;
        if (columns >= 4096 && rows == 2 && x_dtype == TLLM_I8 &&
            (short_k && access == BITS_COLUMNS && w->lay.nnz * 3 < entries ? 0.97 : 1.6) * gather < std::min(bits, tiles()))
            return KERNEL_GATHER;
        // Four bits an entry, which no thread touches.  16 bits: where a block of the register decoder makes several passes (more than twelve groups of sixteen columns to an SM)
        // the two are level (8192 x 28672, one row of bf16 26.9 us, 26.5 decoded); with more rows, more columns or a longer K the decoder is ahead (eight rows
        // 32.1 and 27.4; 8192 x 57344, one row 46.4 and 44.8; 28672 x 8192 31.1 and 24.2).  fp32: faster than the three pieces in registers (8192 x 28672, one row
        // 27.1 and 38.4; 10056 x 15232 21.2 and 24.5).  The model is 10 to 20 % low for fp32 and for rows on odd addresses.  More than one launch's rows (4, fp32 2)
        // have to start on 16 bytes: its planes are made from X element by element else (28672 x 8192, eight rows: 82 us, the batched kernel 43).  Of fp32
        // these compete with the batched kernel (three rows on 5120 x 23512 20.1 us against 24.9, on 2240 x 23936 12.8 against 18.6), over a K that is
        // not too long: 28672 x 8192, four rows 59 against 40.
        if (nibbles) {
            if (x_dtype == TLLM_F32 && rows > per) {
                if (inners <= 16384 && 0.95 * nibble < std::min(bits, tiles())) return KERNEL_NIBBLE;
            } else if (x_dtype == TLLM_F32 ? 1.2 * nibble < bits : nb && columns > 12 * 16 * sms && (access == BITS_ROWS16 ? 0.92 : 1.2) * nibble < bits)
                return KERNEL_NIBBLE;
        }
        return bits_prefer_registers(inners, columns, sms, w->device, mm_direct(inners, X, x_dtype, x_layout, x_ld), x_dtype, access, rows) ? KERNEL_BITS : KERNEL_MMA;
    }
    return nb ? KERNEL_NIBBLE : KERNEL_GATHER;           // no bit tiles, or the kernels on them switched off
}

// K-tiles whose activation tables one launch keeps in shared memory at the same time (the rest follow, one barrier-
// separated group after the other): small tables leave room for four blocks per SM
#ifndef BS_RESIDENT_MAX
#define BS_RESIDENT_MAX 2
#endif
int resident_tiles(int mp, int tiles_per_cta) {
    const int fit = BS_RESIDENT_MAX / mp > 0 ? BS_RESIDENT_MAX / mp : 1;
    return tiles_per_cta < fit ? tiles_per_cta : fit;
}

// one gather launch of at most four rows
int run_bs(tllm_weight* w, const void* X, int x_dtype, int x_layout, int x_ld, int rows, void* Y, int y_dtype, int y_ld,
           int epilogue, float scale, float scale2, const Scratch& scr, cudaStream_t st) {
    const BsLayout& L = w->lay;
    const int mp = rows <= 1 ? 1 : (rows == 2 ? 2 : 4);
    BsParams p{};
    p.stream = w->d_stream;
    p.meta = w->d_meta;
    p.X = X;
    p.Y = Y;
    p.partial = scr.partial;
    p.counters = scr.counters;
    p.status = w->d_status;
    p.x_dtype = x_dtype;
    p.x_layout = x_layout;
    p.y_dtype = y_dtype;
    p.M = rows;
    p.K = L.inners;
    p.N = L.columns;
    p.T = L.tile_rows;
    p.col_blocks = L.col_blocks;
    p.k_splits = L.k_splits;
    p.tiles_per_cta = L.tiles_per_cta;
    p.max_cols = L.max_cols_per_block;
    p.resident = resident_tiles(mp, L.tiles_per_cta);
    p.epilogue = epilogue;
    p.y_ld = y_ld;
    p.x_ld = x_ld;
    const size_t e = dtype_size(x_dtype);
    p.x_vec = x_layout == TLLM_ROW_MAJOR && ((uintptr_t)X % 16 == 0) && ((size_t)x_ld * e % 16 == 0) && (L.inners % 16 == 0) && (L.tile_rows % 16 == 0);
    p.l2_prefetch_bytes = 256u * 1024u;
    p.scale = scale;
    p.scale2 = scale2;
    const BsSmem sm = bs_smem_layout(mp, p.resident, L.tiles_per_cta, L.max_cols_per_block, w->max_meta_words, BS_STAGE_BYTES);
    p.off_table = sm.off_table, p.off_cells = sm.off_cells, p.off_meta = sm.off_meta, p.off_bars = sm.off_bars, p.off_stage = sm.off_stage;
    if (sm.total > 227u * 1024u) return fail(TLLM_ERR_ARG, "gather kernel: this weight needs %u bytes of shared memory per block", sm.total);
    p.cta_ext = w->d_cta;
    std::memcpy(p.cta, L.cta.data(), sizeof(TsCtaDesc) * (size_t)(L.num_ctas < BS_MAX_PARAM_BLOCKS ? L.num_ctas : BS_MAX_PARAM_BLOCKS));
    if (x_dtype == TLLM_I8) {
        if (mp == 1) return launch_bs<int, 1>(p, L.num_ctas, sm.total, st);
        if (mp == 2) return launch_bs<int, 2>(p, L.num_ctas, sm.total, st);
        return launch_bs<int, 4>(p, L.num_ctas, sm.total, st);
    }
    if (mp == 1) return launch_bs<float, 1>(p, L.num_ctas, sm.total, st);
    if (mp == 2) return launch_bs<float, 2>(p, L.num_ctas, sm.total, st);
    return launch_bs<float, 4>(p, L.num_ctas, sm.total, st);
}

// the gather product of any number of rows: launches of up to max_rows rows
int run_gather(tllm_weight* w, const void* X, int x_dtype, int x_layout, int x_ld, int rows, void* Y, int y_dtype, int y_ld, int epilogue,
               float scale, float scale2, const Scratch& scr, cudaStream_t st) {
    const size_t xe = dtype_size(x_dtype), ye = dtype_size(y_dtype);
    for (int r0 = 0; r0 < rows; r0 += w->max_rows) {
        const int m = rows - r0 < w->max_rows ? rows - r0 : w->max_rows;
        const char* xp = (const char*)X + (x_layout == TLLM_ROW_MAJOR ? (size_t)r0 * x_ld : (size_t)r0) * xe;
        char* yp = (char*)Y + (size_t)r0 * y_ld * ye;
        const int r = run_bs(w, xp, x_dtype, x_layout, x_ld, m, yp, y_dtype, y_ld, epilogue, scale, scale2, scr, st);
        if (r) return r;
    }
    return TLLM_OK;
}

// [rows][columns] -> [columns][ld], elements of e bytes, on the device
int turn_out(const void* src, void* dst, int rows, int columns, int ld, int e, cudaStream_t st) {
    const dim3 grid((columns + 31) / 32, std::min((rows - 1) / 32 + 1, 65535)), block(32, 8);
    if (e == 4) turn_kernel<uint32_t><<<grid, block, 0, st>>>((const uint32_t*)src, (uint32_t*)dst, rows, columns, ld);
    else turn_kernel<uint16_t><<<grid, block, 0, st>>>((const uint16_t*)src, (uint16_t*)dst, rows, columns, ld);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return TLLM_OK;
}

// the product of `rows` rows on the kernel that choose_kernel names.  y_col: Y is column-major (y_ld elements from column to
// column), which the two kernels on bit tiles write themselves; for the others it is turned out of a workspace.
int run_product(tllm_weight* w, const void* X, int x_dtype, int x_layout, int x_ld, int rows, void* Y, int y_dtype, int y_ld, int epilogue, float scale,
                float scale2, cudaStream_t st, bool y_col = false) {
    const KernelChoice kc = choose_kernel(w, X, x_dtype, x_layout, x_ld, rows);
    if (kc == KERNEL_BITS) return run_bits(bits_view(w), X, x_dtype, x_layout, x_ld, rows, Y, y_dtype, y_ld, epilogue, scale, scale2, st, y_col);
    if (kc == KERNEL_MMA) return run_mm(bits_view(w), X, x_dtype, x_layout, x_ld, rows, Y, y_dtype, y_ld, epilogue, scale, scale2, st, y_col);
    Workspace ws;
    void* out = Y;
    int ld = y_ld;
    if (y_col) {
        ld = w->lay.columns;
        const int rc = ws.take(w->device, (size_t)rows * ld * dtype_size(y_dtype), st);
        if (rc) return rc;
        out = ws.ptr;
    }
    const int rc = kc == KERNEL_NIBBLE ? run_nb(w, X, x_dtype, x_ld, rows, out, y_dtype, ld, epilogue, scale, scale2, st)
                                       : run_gather(w, X, x_dtype, x_layout, x_ld, rows, out, y_dtype, ld, epilogue, scale, scale2, Scratch{w->d_partial, w->d_counters}, st);
    if (rc || !y_col) return rc;
    return turn_out(out, Y, rows, ld, y_ld, (int)dtype_size(y_dtype), st);
}

int upload(tllm_weight* w, const BsHostImage& img, float scale, int max_rows) {
    w->lay = img.lay;
    w->scale = scale;
    w->max_rows = max_rows;
    w->max_meta_words = 0;
    for (const TsCtaDesc& d : img.lay.cta) w->max_meta_words = d.meta_words > w->max_meta_words ? d.meta_words : w->max_meta_words;
    CU_TRY(cudaGetDevice(&w->device));
    w->stream_bytes = img.stream.size();
    w->meta_bytes = img.meta.size() * sizeof(uint32_t);
    CU_TRY(cudaMalloc(&w->d_stream, w->stream_bytes + 512));
    CU_TRY(cudaMalloc(&w->d_meta, w->meta_bytes + 16));
    CU_TRY(cudaMemcpy(w->d_stream, img.stream.data(), w->stream_bytes, cudaMemcpyHostToDevice));
    CU_TRY(cudaMemcpy(w->d_meta, img.meta.data(), w->meta_bytes, cudaMemcpyHostToDevice));
    CU_TRY(cudaMalloc(&w->d_cta, img.lay.cta.size() * sizeof(TsCtaDesc)));
    CU_TRY(cudaMemcpy(w->d_cta, img.lay.cta.data(), img.lay.cta.size() * sizeof(TsCtaDesc), cudaMemcpyHostToDevice));
    const size_t partial_bytes = img.lay.k_splits > 1 ? (size_t)img.lay.k_splits * max_rows * img.lay.columns * 4 : 16;
    const size_t counter_bytes = (size_t)img.lay.col_blocks * sizeof(unsigned int);
    w->scratch_bytes = partial_bytes + counter_bytes + sizeof(int);
    CU_TRY(cudaMalloc(&w->d_partial, partial_bytes));
    CU_TRY(cudaMalloc(&w->d_counters, counter_bytes));
    CU_TRY(cudaMalloc(&w->d_status, sizeof(int)));
    CU_TRY(cudaMemset(w->d_counters, 0, counter_bytes));
    CU_TRY(cudaMemset(w->d_status, 0, sizeof(int)));
    CU_TRY(cudaDeviceSynchronize());
    return TLLM_OK;
}

int upload_bit_tiles(tllm_weight* w, const std::vector<uint32_t>& bits, int sms) {
    w->bits_bytes = bits.size() * sizeof(uint32_t);
    w->mm_grid = sms;
    CU_TRY(cudaMalloc(&w->d_bits, w->bits_bytes));
    CU_TRY(cudaMemcpy(w->d_bits, bits.data(), w->bits_bytes, cudaMemcpyHostToDevice));
    if (tensor_map_encoder() != nullptr) {
        int rc = encode_bits_map(&w->bits_map[0], w->d_bits, w->mm_n_tiles, w->mm_kb, MM_UK);
        if (!rc) rc = encode_bits_map(&w->bits_map[1], w->d_bits, w->mm_n_tiles, w->mm_kb, MS_UK);
        if (rc) return rc;
    }
    const size_t partial_bytes = (size_t)2 * sms * MM_TILE_N * MM_OWN_NT * sizeof(float);
    const size_t counter_bytes = (size_t)w->mm_n_tiles * MM_MAX_M_TILES * 4 * sizeof(unsigned int);
    CU_TRY(cudaMalloc(&w->d_mm_partial, partial_bytes));
    CU_TRY(cudaMalloc(&w->d_mm_counters, counter_bytes));
    CU_TRY(cudaMemset(w->d_mm_counters, 0, counter_bytes));
    w->scratch_bytes += partial_bytes + counter_bytes;
    CU_TRY(cudaDeviceSynchronize());
    return TLLM_OK;
}

int upload_bits(tllm_weight* w, const int8_t* dense, int inners, int columns, int sms) {
    std::vector<uint32_t> bits;
    mm_pack_bits(dense, inners, columns, &bits, &w->mm_n_tiles, &w->mm_kb);
    return upload_bit_tiles(w, bits, sms);
}

int device_sms(int* sms) {
    int dev = 0;
    CU_TRY(cudaGetDevice(&dev));
    CU_TRY(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
    int max_smem = 0;
    CU_TRY(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    if (max_smem < 227 * 1024)
        return fail(TLLM_ERR_ARG, "this device offers %d bytes of shared memory per block; the kernels need 232448 (built for sm_100a)", max_smem);
    return TLLM_OK;
}

int create_from_dense(const int8_t* dense, int inners, int columns, float scale, const tllm_pack_opts* opts, tllm_weight** out) {
    if (!out) return fail(TLLM_ERR_ARG, "weight create: out is NULL");
    *out = nullptr;
    int sms = 0;
    int rc = device_sms(&sms);
    if (rc) return rc;
    BsHostImage img;
    const char* msg = bs_pack_dense(dense, inners, columns, opts, sms, &img);
    if (msg) return fail(TLLM_ERR_ARG, "%s", msg);
    int max_rows = (opts && opts->max_rows > 0) ? opts->max_rows : 4;
    if (max_rows > 4) max_rows = 4;
    tllm_weight* w = new tllm_weight();
    g_handles.fetch_add(1, std::memory_order_relaxed);
    rc = upload(w, img, scale, max_rows);
    if (rc == TLLM_OK && !(opts && opts->no_bit_tiles)) rc = upload_bits(w, dense, inners, columns, sms);
    if (rc == TLLM_OK && !(opts && opts->no_nibbles)) rc = upload_nibbles(w, dense, inners, columns, sms);
    if (rc != TLLM_OK) {
        tllm_weight_destroy(w);
        return rc;
    }
    *out = w;
    return TLLM_OK;
}

int ensure(void** p, size_t* cap, size_t need, bool pinned) {
    if (*cap >= need) return TLLM_OK;
    if (*p) {
        if (pinned) CU_TRY(cudaFreeHost(*p));
        else CU_TRY(cudaFree(*p));
        *p = nullptr;
        *cap = 0;
    }
    size_t n = need < 4096 ? 4096 : need;
    if (pinned) CU_TRY(cudaMallocHost(p, n));
    else CU_TRY(cudaMalloc(p, n));
    *cap = n;
    return TLLM_OK;
}

// Y[rows][columns] (row-major, on the device) += bias[columns], both of y_dtype
int add_bias(void* Y, const void* bias, int y_dtype, int rows, int columns, cudaStream_t st) {
    const long long n = (long long)rows * columns;
    bias_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(Y, bias, y_dtype, n, columns);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return TLLM_OK;
}

int device_sms_cached(int dev, int* sms) {
    static std::atomic<int> known[64];
    int v = dev < 64 ? known[dev].load(std::memory_order_relaxed) : 0;
    if (!v) {
        const int rc = device_sms(&v);
        if (rc) return rc;
        if (dev < 64) known[dev].store(v, std::memory_order_relaxed);
    }
    *sms = v;
    return TLLM_OK;
}

// ---- the product on the reference's arrays as they are --------------------------------------------------------------
// one warp per column; with `flags`, `blocks` thread blocks that do it only if one of the nflags words is not zero
int run_mcsc(const void* X, int x_dtype, int x_layout, const int16_t* row_idx, const int32_t* col_off, void* Y, int y_dtype, int batch, int rows, int columns,
             int inners, int tile_k, float scale, const int* flags, int nflags, int blocks, cudaStream_t st) {
    const dim3 grid((columns + 7) / 8, (rows + MCSC_ROWS - 1) / MCSC_ROWS, batch);
#define MCSC_ARGS rows, columns, inners, tile_k, scale
    if (flags) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)blocks);
        cfg.blockDim = dim3(256);
        cfg.stream = st;
        cudaLaunchAttribute at[1] = {pdl_attribute()};
        cfg.attrs = at;
        cfg.numAttrs = 1;
        auto kern = x_dtype == TLLM_I8 ? mcsc_spmm_if_kernel<int, MCSC_ROWS> : mcsc_spmm_if_kernel<float, MCSC_ROWS>;
        CU_TRY(cudaLaunchKernelEx(&cfg, kern, X, x_dtype, x_layout, row_idx, col_off, Y, y_dtype, batch, MCSC_ARGS, flags, nflags));
    } else {
        if (grid.y > 65535) return fail(TLLM_ERR_ARG, "tllm_ter_spmm: too many rows for one call");
        if (x_dtype == TLLM_I8) mcsc_spmm_kernel<int, MCSC_ROWS><<<grid, 256, 0, st>>>(X, x_dtype, x_layout, row_idx, col_off, Y, y_dtype, MCSC_ARGS);
        else mcsc_spmm_kernel<float, MCSC_ROWS><<<grid, 256, 0, st>>>(X, x_dtype, x_layout, row_idx, col_off, Y, y_dtype, MCSC_ARGS);
    }
#undef MCSC_ARGS
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return TLLM_OK;
}

// Whether the arrays are turned into bit tiles first, on every call.  The per-column kernel reads the lists again for every four
// rows; the conversion and the kernels behind it cost 13 to 24 us at least.  2048 x 8192, 80 % zeros, fp32: 5 rows 24 us turned into tiles, 41 per
// column; 256 rows 39 and 1393.  The two meet at about 6e6 entries times passes: 24 rows of fp32 17.5 us and 16.6 on 1024 x 1024, 14.7 and 14.9 on
// 512 x 2048 (bf16 16.8 and 18.7, 13.3 and 16.7), 9 rows on 2048 x 1024, half zeros, 24.8 and 26.0.
bool lists_worth_converting(long long entries, int rows) { return rows > MCSC_ROWS && entries * ((rows + MCSC_ROWS - 1) / MCSC_ROWS) >= 6000000; }

int run_lists(const void* X, int x_dtype, int x_layout, const int16_t* row_idx, const int32_t* col_off, void* Y, int y_dtype, int batch, int rows, int columns,
              int inners, int tile_k, float scale, int dev, int sms, cudaStream_t st) {
    const int n_tiles = (columns + 127) / 128, kb = (inners + 63) / 64, groups = n_tiles * 8;
    const size_t bits_bytes = (size_t)groups * kb * 256, counter_words = (size_t)n_tiles * MM_MAX_M_TILES * 4;
    Workspace ws;
    int rc = ws.take(dev, bits_bytes + (counter_words + groups + 1) * 4, st);
    if (rc) return rc;
    uint32_t* bits = (uint32_t*)ws.ptr;
    unsigned int* counters = (unsigned int*)((char*)ws.ptr + bits_bytes);
    int* flags = (int*)(counters + counter_words);          // one per group of columns, then the status word of the product
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)groups);
    cfg.blockDim = dim3(LB_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute at[1] = {pdl_attribute()};
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CU_TRY(cudaLaunchKernelEx(&cfg, lists_to_bits_kernel, row_idx, col_off, bits, counters, (int)counter_words, flags, columns, inners, tile_k, kb));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    CUtensorMap map[2];
    rc = encode_bits_map(&map[0], bits, n_tiles, kb, MM_UK);
    if (!rc) rc = encode_bits_map(&map[1], bits, n_tiles, kb, MS_UK);
    if (rc) return rc;
    BitsView view{(const uint4*)bits, map, inners, columns, n_tiles, kb, sms, dev, nullptr, counters, flags + groups, true, true};
    const size_t xe = dtype_size(x_dtype), ye = dtype_size(y_dtype);
    const bool one = x_layout == TLLM_ROW_MAJOR && (long long)batch * rows <= 0x7fffffffLL;      // the batch is contiguous: one product
    const int parts = one ? 1 : batch, m = one ? batch * rows : rows, x_ld = x_layout == TLLM_ROW_MAJOR ? inners : rows;
    for (int b = 0; b < parts; ++b) {
        const char* xp = (const char*)X + (size_t)b * rows * inners * xe;
        char* yp = (char*)Y + (size_t)b * rows * columns * ye;
        if (bits_prefer_registers(inners, columns, sms, dev, mm_direct(inners, xp, x_dtype, x_layout, x_ld), x_dtype, bits_access(xp, x_dtype, x_layout, x_ld), m))
            rc = run_bits(view, xp, x_dtype, x_layout, x_ld, m, yp, y_dtype, columns, 0, scale, 0.f, st);
        else rc = run_mm(view, xp, x_dtype, x_layout, x_ld, m, yp, y_dtype, columns, 0, scale, 0.f, st);
        if (rc) return rc;
        view.fresh = false;
    }
    // lists that two bits an entry cannot hold (an entry named twice) are computed as before
    return run_mcsc(X, x_dtype, x_layout, row_idx, col_off, Y, y_dtype, batch, rows, columns, inners, tile_k, scale, flags, groups + 1, 2 * sms, st);
}

}  // namespace

namespace tllm {
void bs_fill_info(const BsLayout& L, tllm_weight_info* info) {
    info->inners = L.inners;
    info->columns = L.columns;
    info->tile_rows = L.tile_rows;
    info->tiles = L.tiles;
    info->col_blocks = L.col_blocks;
    info->k_splits = L.k_splits;
    info->tiles_per_cta = L.tiles_per_cta;
    info->num_ctas = L.num_ctas;
    info->units = (int)L.units;
    info->nnz = L.nnz;
    info->algorithmic_bytes = 2 * L.nnz + 16 * (int64_t)L.columns * ((L.inners + 511) / 512);
}
}  // namespace tllm

#ifdef BS_TRACE
extern "C" int tllm_debug_set_trace(void* device_buffer) {
    CU_TRY(cudaMemcpyToSymbol(tllm::g_bs_trace, &device_buffer, sizeof(void*)));
    return TLLM_OK;
}
#endif

extern "C" {

const char* tllm_last_error(void) { return g_err.c_str(); }
int tllm_version(void) { return 200; }
int64_t tllm_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }
int64_t tllm_bits_launch_count(void) { return g_bits_launches.load(std::memory_order_relaxed); }
int64_t tllm_mma_launch_count(void) { return g_mm_launches.load(std::memory_order_relaxed); }
int tllm_mma_last_plan(int plan[5]) {
    if (!plan || g_mm_last_plan[0] == 0) return fail(TLLM_ERR_ARG, "tllm_mma_last_plan: %s", plan ? "this thread has launched none" : "plan is NULL");
    std::memcpy(plan, g_mm_last_plan, sizeof g_mm_last_plan);
    return TLLM_OK;
}
int tllm_bits_last_plan(int plan[6]) {
    if (!plan || bits_last_plan[0] == 0) return fail(TLLM_ERR_ARG, "tllm_bits_last_plan: %s", plan ? "this thread has launched none" : "plan is NULL");
    std::memcpy(plan, bits_last_plan, sizeof bits_last_plan);
    return TLLM_OK;
}
int tllm_set_mma_min_rows(int rows) {
    const int prev = mm_min_rows();
    g_mm_min_rows.store(rows < 0 ? -1 : rows, std::memory_order_relaxed);
    return prev;
}

// ---- packed copies of the reference's device arrays, keyed by the arrays' addresses and the shape --------------------
namespace {
struct TerCacheEntry {
    const void* row_idx;
    const void* col_off;
    int columns, inners, tile_k, device;
    tllm_weight* w;
};
std::mutex g_ter_mu;
std::vector<TerCacheEntry> g_ter_cache;

tllm_weight* ter_cache_find(const void* row_idx, const void* col_off, int columns, int inners, int tile_k) {
    std::lock_guard<std::mutex> lk(g_ter_mu);
    if (g_ter_cache.empty()) return nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    for (const TerCacheEntry& e : g_ter_cache)
        if (e.row_idx == row_idx && e.col_off == col_off && e.columns == columns && e.inners == inners && e.tile_k == tile_k && e.device == dev) return e.w;
    return nullptr;
}
}  // namespace

int tllm_ter_spmm_prepare(const int16_t* row_idx, const int32_t* col_off, int columns, int inners, int tile_k) {
    if (!row_idx || !col_off || columns <= 0 || inners <= 0 || tile_k <= 0) return fail(TLLM_ERR_ARG, "tllm_ter_spmm_prepare: bad argument");
    if (ter_cache_find(row_idx, col_off, columns, inners, tile_k)) return TLLM_OK;
    // the row-index array's length is the largest list end
    const size_t n_off = (size_t)columns * ((size_t)(inners + tile_k - 1) / tile_k) * 4;
    std::vector<int32_t> off(n_off);
    CU_TRY(cudaMemcpy(off.data(), col_off, n_off * sizeof(int32_t), cudaMemcpyDeviceToHost));
    int64_t len = 0;
    for (size_t i = 0; i < n_off; i += 4) len = std::max<int64_t>(len, off[i + 2]);
    tllm_weight* w = nullptr;
    const int rc = tllm_weight_create_mcsc_device(row_idx, len, col_off, columns, inners, tile_k, 1.0f, nullptr, &w);
    if (rc) return rc;
    std::lock_guard<std::mutex> lk(g_ter_mu);
    g_ter_cache.push_back(TerCacheEntry{row_idx, col_off, columns, inners, tile_k, w->device, w});
    return TLLM_OK;
}

int tllm_ter_spmm_forget(const int16_t* row_idx, const int32_t* col_off) {
    std::vector<tllm_weight*> dead;
    {
        std::lock_guard<std::mutex> lk(g_ter_mu);
        for (size_t i = 0; i < g_ter_cache.size();) {
            if ((!row_idx && !col_off) || (g_ter_cache[i].row_idx == row_idx && g_ter_cache[i].col_off == col_off)) {
                dead.push_back(g_ter_cache[i].w);
                g_ter_cache.erase(g_ter_cache.begin() + (long)i);
            } else ++i;
        }
    }
    for (tllm_weight* w : dead) tllm_weight_destroy(w);
    if (!row_idx && !col_off && g_handles.load(std::memory_order_relaxed) == 0) ws_trim();      // calls on arrays as they are need no handle
    return (int)dead.size();
}

int tllm_set_nibble_max_rows(int rows) {
    return g_nb_max_rows.exchange(rows < 0 ? -1 : rows, std::memory_order_relaxed);
}

#ifdef NB_DEBUG
int tllm_debug_set_nb_tx(int bytes) {
    g_nb_debug_tx = bytes;
    return 0;
}
int tllm_debug_set_nb_flags(int flags) {
    g_nb_debug_flags = flags;
    return 0;
}
int tllm_debug_set_nb_stages(int stages) {
    g_nb_debug_stages = stages;
    return 0;
}
int tllm_debug_set_nb_trace(void* device_buffer) {
    CU_TRY(cudaMemcpyToSymbol(tllm::g_nb_trace, &device_buffer, sizeof(void*)));
    return TLLM_OK;
}
#endif
int64_t tllm_nibble_launch_count(void) { return g_nb_launches.load(std::memory_order_relaxed); }

int tllm_ter_spmm(const void* X, int x_dtype, int x_layout, const int16_t* row_idx, const int32_t* col_off,
                  const int16_t* col_tile_idx, void* Y, int y_dtype, int batch, int rows, int columns,
                  int inners, int tile_k, float scale, int uniformed, int padded, void* stream) {
    (void)col_tile_idx;
    (void)uniformed;
    (void)padded;
    if (batch == 0) return TLLM_OK;   // the reference launches nothing for a 2-D input (TernaryLinear.py:168)
    if (!X || !row_idx || !col_off || !Y) return fail(TLLM_ERR_ARG, "tllm_ter_spmm: NULL pointer");
    if (batch < 0 || rows <= 0 || columns <= 0 || inners <= 0 || tile_k <= 0) return fail(TLLM_ERR_ARG, "tllm_ter_spmm: bad shape");
    const int rc = check_types(x_dtype, y_dtype, "tllm_ter_spmm");
    if (rc) return rc;
    if (batch > 65535) return fail(TLLM_ERR_ARG, "tllm_ter_spmm: batch too large");
    if (rows == 1) x_layout = TLLM_ROW_MAJOR;        // one row per batch item: both layouts are the same memory
    if (tllm_weight* w = ter_cache_find(row_idx, col_off, columns, inners, tile_k)) {
        // these arrays were repacked by tllm_ter_spmm_prepare: the product runs on the packed copy
        cudaStream_t st = (cudaStream_t)stream;
        const size_t xe = dtype_size(x_dtype), ye = dtype_size(y_dtype);
        if (x_layout == TLLM_ROW_MAJOR) {
            const long long m = (long long)batch * rows;      // the batch is contiguous: one product of batch * rows rows
            if (m > 0x7fffffffLL) return fail(TLLM_ERR_ARG, "tllm_ter_spmm: batch * rows too large");
            return run_product(w, X, x_dtype, x_layout, inners, (int)m, Y, y_dtype, columns, 0, scale, 0.f, st);
        }
        for (int b = 0; b < batch; ++b) {
            const int rc2 = run_product(w, (const char*)X + (size_t)b * rows * inners * xe, x_dtype, x_layout, rows, rows,
                                        (char*)Y + (size_t)b * rows * columns * ye, y_dtype, columns, 0, scale, 0.f, st);
            if (rc2) return rc2;
        }
        return TLLM_OK;
    }
    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0, sms = 0;
    CU_TRY(cudaGetDevice(&dev));
    if (mm_min_rows() == -1 && lists_worth_converting((long long)columns * inners, x_layout == TLLM_ROW_MAJOR ? (int)std::min(rows * (long long)batch, 0x7fffffffLL) : rows) && (x_dtype != TLLM_I8 || inners <= 131072) && tensor_map_encoder() != nullptr) {
        const int rc2 = device_sms_cached(dev, &sms);
        if (rc2) return rc2;
        return run_lists(X, x_dtype, x_layout, row_idx, col_off, Y, y_dtype, batch, rows, columns, inners, tile_k, scale, dev, sms, st);
    }
    return run_mcsc(X, x_dtype, x_layout, row_idx, col_off, Y, y_dtype, batch, rows, columns, inners, tile_k, scale, nullptr, 0, 0, st);
}

int tllm_weight_create_dense(const int8_t* w, int inners, int columns, float scale, const tllm_pack_opts* opts, tllm_weight** out) {
    if (!w || inners <= 0 || columns <= 0) return fail(TLLM_ERR_ARG, "tllm_weight_create_dense: bad argument");
    const size_t n = (size_t)inners * columns;
    for (size_t i = 0; i < n; ++i)
        if (w[i] < -1 || w[i] > 1) return fail(TLLM_ERR_ARG, "tllm_weight_create_dense: entry %zu is %d, not ternary", i, (int)w[i]);
    return create_from_dense(w, inners, columns, scale, opts, out);
}

int tllm_weight_create_mcsc(const int32_t* row_idx, const int32_t* col_off, int columns, int inners, int tile_k, float scale,
                            const tllm_pack_opts* opts, tllm_weight** out) {
    if (!row_idx || !col_off || columns <= 0 || inners <= 0 || tile_k <= 0) return fail(TLLM_ERR_ARG, "tllm_weight_create_mcsc: bad argument");
    std::vector<int8_t> dense;
    const char* msg = decode_mcsc(row_idx, col_off, columns, inners, tile_k, &dense);
    if (msg) return fail(TLLM_ERR_ARG, "%s", msg);
    return create_from_dense(dense.data(), inners, columns, scale, opts, out);
}

int tllm_weight_create_ssr(const uint8_t* image, size_t bytes, int inners, int columns, float scale, const tllm_pack_opts* opts, tllm_weight** out) {
    if (!image || inners <= 0 || columns <= 0) return fail(TLLM_ERR_ARG, "tllm_weight_create_ssr: bad argument");
    std::vector<int8_t> dense((size_t)inners * (size_t)columns);
    const int rc = tllm_ssr_decode(image, bytes, inners, columns, dense.data());      // validates the whole image first
    if (rc != TLLM_OK) return rc;
    return create_from_dense(dense.data(), inners, columns, scale, opts, out);
}

int tllm_weight_create_mcsc_device(const int16_t* row_idx, int64_t row_idx_len, const int32_t* col_off, int columns, int inners, int tile_k,
                                   float scale, const tllm_pack_opts* opts, tllm_weight** out) {
    if (!row_idx || !col_off || columns <= 0 || inners <= 0 || tile_k <= 0 || row_idx_len < 0)
        return fail(TLLM_ERR_ARG, "tllm_weight_create_mcsc_device: bad argument");
    const size_t n_off = (size_t)columns * ((size_t)(inners + tile_k - 1) / tile_k) * 4;
    std::vector<int16_t> ri16((size_t)row_idx_len);
    std::vector<int32_t> off(n_off);
    if (row_idx_len) CU_TRY(cudaMemcpy(ri16.data(), row_idx, ri16.size() * sizeof(int16_t), cudaMemcpyDeviceToHost));
    CU_TRY(cudaMemcpy(off.data(), col_off, off.size() * sizeof(int32_t), cudaMemcpyDeviceToHost));
    for (size_t i = 0; i < n_off; i += 4)
        if (off[i] < 0 || off[i + 1] < off[i] || off[i + 2] < off[i + 1] || off[i + 2] > row_idx_len)
            return fail(TLLM_ERR_ARG, "tllm_weight_create_mcsc_device: list offsets of entry %zu leave the row-index array", i / 4);
    std::vector<int32_t> ri(ri16.begin(), ri16.end());
    return tllm_weight_create_mcsc(ri.data(), off.data(), columns, inners, tile_k, scale, opts, out);
}

int tllm_weight_create_cpu_format(int kind, int group, int chunk, const int32_t* meta, const void* ri, int ri32, int64_t aux,
                                  int columns, int inners, float scale, const tllm_pack_opts* opts, tllm_weight** out) {
    if (!meta || !ri || columns <= 0 || inners <= 0) return fail(TLLM_ERR_ARG, "tllm_weight_create_cpu_format: bad argument");
    std::vector<int8_t> dense;
    const char* msg = decode_cpu_format(kind, group, chunk, meta, ri, ri32, aux, columns, inners, &dense);
    if (msg) return fail(TLLM_ERR_ARG, "%s", msg);
    return create_from_dense(dense.data(), inners, columns, scale, opts, out);
}

int tllm_weight_destroy(tllm_weight* w) {
    if (!w) return TLLM_OK;
    cudaFree(w->d_stream);
    cudaFree(w->d_meta);
    cudaFree(w->d_cta);
    cudaFree(w->d_bits);
    cudaFree(w->d_mm_partial);
    cudaFree(w->d_mm_counters);
    cudaFree(w->d_nib);
    cudaFree(w->d_nb_partial);
    cudaFree(w->d_nb_counters);
    cudaFree(w->d_nb_sched);
    cudaFree(w->d_nr_pieces);
    cudaFree(w->d_nr_row_pow);
    cudaFree(w->d_nr_partial);
    cudaFree(w->d_nr_counters);
    cudaFree(w->d_partial);
    cudaFree(w->d_counters);
    cudaFree(w->d_status);
    cudaFree(w->d_x);
    cudaFree(w->d_y);
    cudaFree(w->d_bias);
    if (w->h_status) cudaFreeHost(w->h_status);
    for (cudaEvent_t e : w->part_event)
        if (e) cudaEventDestroy(e);
    if (w->own_stream) cudaStreamDestroy(w->own_stream);
    delete w;
    if (g_handles.fetch_sub(1, std::memory_order_relaxed) == 1) ws_trim();
    return TLLM_OK;
}

int tllm_weight_get_info(const tllm_weight* w, tllm_weight_info* info) {
    if (!w || !info) return fail(TLLM_ERR_ARG, "tllm_weight_get_info: NULL");
    std::memset(info, 0, sizeof *info);
    bs_fill_info(w->lay, info);
    info->max_rows = w->max_rows;
    info->stream_bytes = (int64_t)w->stream_bytes;
    info->meta_bytes = (int64_t)w->meta_bytes;
    info->scratch_bytes = (int64_t)w->scratch_bytes;
    info->bit_tile_bytes = (int64_t)w->bits_bytes;
    info->nibble_bytes = (int64_t)w->nib_bytes;
    info->scale = w->scale;
    return TLLM_OK;
}

// ---- packed-weight files: header, column ranges, block descriptors, index stream, block tables, bit tiles ----------
namespace {
struct WeightFileHeader {
    char magic[8];                // "TLLMW003"; "TLLMW002" files hold the bit tiles in another order
    int32_t inners, columns, tile_rows, tiles, col_blocks, k_splits, tiles_per_cta, num_ctas, max_cols_per_block, max_rows, mm_n_tiles, mm_kb;
    int64_t nnz, total_vecs, units, meta_words, bits_words;
    float scale;
    int32_t reserved[7];
};
bool read_exact(FILE* f, void* p, size_t n) { return n == 0 || fread(p, 1, n, f) == n; }
bool write_exact(FILE* f, const void* p, size_t n) { return n == 0 || fwrite(p, 1, n, f) == n; }
}  // namespace

int tllm_weight_save(const tllm_weight* w, const char* path) {
    if (!w || !path) return fail(TLLM_ERR_ARG, "tllm_weight_save: NULL argument");
    const BsLayout& L = w->lay;
    WeightFileHeader h{};
    std::memcpy(h.magic, "TLLMW003", 8);
    h.inners = L.inners, h.columns = L.columns, h.tile_rows = L.tile_rows, h.tiles = L.tiles, h.col_blocks = L.col_blocks;
    h.k_splits = L.k_splits, h.tiles_per_cta = L.tiles_per_cta, h.num_ctas = L.num_ctas, h.max_cols_per_block = L.max_cols_per_block;
    h.max_rows = w->max_rows, h.mm_n_tiles = w->mm_n_tiles, h.mm_kb = w->mm_kb;
    h.nnz = L.nnz, h.total_vecs = L.total_vecs, h.units = L.units;
    h.meta_words = (int64_t)(w->meta_bytes / sizeof(uint32_t));
    h.bits_words = (int64_t)(w->bits_bytes / sizeof(uint32_t));
    h.scale = w->scale;
    std::vector<unsigned char> stream(w->stream_bytes), meta(w->meta_bytes), bits(w->bits_bytes);
    int prev = 0;
    CU_TRY(cudaGetDevice(&prev));
    CU_TRY(cudaSetDevice(w->device));
    CU_TRY(cudaMemcpy(stream.data(), w->d_stream, w->stream_bytes, cudaMemcpyDeviceToHost));
    CU_TRY(cudaMemcpy(meta.data(), w->d_meta, w->meta_bytes, cudaMemcpyDeviceToHost));
    if (w->bits_bytes) CU_TRY(cudaMemcpy(bits.data(), w->d_bits, w->bits_bytes, cudaMemcpyDeviceToHost));
    CU_TRY(cudaSetDevice(prev));
    FILE* f = fopen(path, "wb");
    if (!f) return fail(TLLM_ERR_ARG, "tllm_weight_save: cannot open %s for writing", path);
    const bool ok = write_exact(f, &h, sizeof h) && write_exact(f, L.col_start.data(), L.col_start.size() * sizeof(int32_t)) &&
                    write_exact(f, L.cta.data(), L.cta.size() * sizeof(TsCtaDesc)) && write_exact(f, stream.data(), stream.size()) &&
                    write_exact(f, meta.data(), meta.size()) && write_exact(f, bits.data(), bits.size());
    if (fclose(f) != 0 || !ok) return fail(TLLM_ERR_ARG, "tllm_weight_save: short write to %s", path);
    return TLLM_OK;
}

int tllm_weight_load(const char* path, tllm_weight** out) {
    if (!path || !out) return fail(TLLM_ERR_ARG, "tllm_weight_load: NULL argument");
    *out = nullptr;
    FILE* f = fopen(path, "rb");
    if (!f) return fail(TLLM_ERR_ARG, "tllm_weight_load: cannot open %s", path);
    WeightFileHeader h{};
    BsHostImage img;
    std::vector<uint32_t> bits;
    bool ok = read_exact(f, &h, sizeof h) && (std::memcmp(h.magic, "TLLMW003", 8) == 0 || std::memcmp(h.magic, "TLLMW002", 8) == 0);
    ok = ok && h.num_ctas > 0 && h.num_ctas <= BS_MAX_BLOCKS && h.col_blocks > 0 && h.col_blocks <= h.num_ctas && h.total_vecs >= 0 && h.meta_words >= 0 &&
         h.bits_words >= 0 && h.total_vecs < ((int64_t)1 << 32) && h.meta_words < ((int64_t)1 << 34) && h.bits_words < ((int64_t)1 << 38);
    if (ok) {
        BsLayout& L = img.lay;
        L.inners = h.inners, L.columns = h.columns, L.tile_rows = h.tile_rows, L.tiles = h.tiles, L.col_blocks = h.col_blocks;
        L.k_splits = h.k_splits, L.tiles_per_cta = h.tiles_per_cta, L.num_ctas = h.num_ctas, L.max_cols_per_block = h.max_cols_per_block;
        L.nnz = h.nnz, L.total_vecs = h.total_vecs, L.units = h.units;
        L.col_start.resize((size_t)h.col_blocks + 1);
        L.cta.resize((size_t)h.num_ctas);
        img.stream.resize((size_t)h.total_vecs * 16);
        img.meta.resize((size_t)h.meta_words);
        bits.resize((size_t)h.bits_words);
        ok = read_exact(f, L.col_start.data(), L.col_start.size() * sizeof(int32_t)) && read_exact(f, L.cta.data(), L.cta.size() * sizeof(TsCtaDesc)) &&
             read_exact(f, img.stream.data(), img.stream.size()) && read_exact(f, img.meta.data(), img.meta.size() * sizeof(uint32_t)) &&
             read_exact(f, bits.data(), bits.size() * sizeof(uint32_t));
    }
    fclose(f);
    if (!ok) return fail(TLLM_ERR_ARG, "tllm_weight_load: %s is not a packed-weight file of this library (or is truncated)", path);
    if (const char* msg = bs_validate(img)) return fail(TLLM_ERR_ARG, "tllm_weight_load: %s", msg);
    const int64_t want_bits = (int64_t)((h.columns + 127) / 128) * ((h.inners + 63) / 64) * 128 * 4;
    if (h.bits_words != 0 && (h.bits_words != want_bits || h.mm_n_tiles != (h.columns + 127) / 128 || h.mm_kb != (h.inners + 63) / 64))
        return fail(TLLM_ERR_ARG, "tllm_weight_load: bit tiles of %s do not match the matrix shape", path);
    int sms = 0;
    int rc = device_sms(&sms);
    if (rc) return rc;
    tllm_weight* w = new tllm_weight();
    g_handles.fetch_add(1, std::memory_order_relaxed);
    rc = upload(w, img, h.scale, h.max_rows > 0 && h.max_rows <= 4 ? h.max_rows : 4);
    // the four-bit planes are not stored, and older files keep the bit tiles in another order: both are rebuilt from the lists
    std::vector<int8_t> dense;
    if (rc == TLLM_OK) {
        dense.resize((size_t)h.inners * h.columns);
        bs_unpack_dense(img, dense.data());
    }
    if (rc == TLLM_OK && h.bits_words) {
        if (h.magic[7] == '3') {
            w->mm_n_tiles = h.mm_n_tiles;
            w->mm_kb = h.mm_kb;
            rc = upload_bit_tiles(w, bits, sms);
        } else rc = upload_bits(w, dense.data(), h.inners, h.columns, sms);
    }
    if (rc == TLLM_OK) rc = upload_nibbles(w, dense.data(), h.inners, h.columns, sms);
    if (rc != TLLM_OK) {
        tllm_weight_destroy(w);
        return rc;
    }
    *out = w;
    return TLLM_OK;
}

int tllm_weight_set_scale(tllm_weight* w, float scale) {
    if (!w) return fail(TLLM_ERR_ARG, "tllm_weight_set_scale: NULL");
    w->scale = scale;
    return TLLM_OK;
}

int tllm_weight_check(tllm_weight* w) {
    if (!w) return fail(TLLM_ERR_ARG, "tllm_weight_check: NULL");
    int st = 0;
    CU_TRY(cudaMemcpy(&st, w->d_status, sizeof(int), cudaMemcpyDeviceToHost));
    if (st != 0) {
        cudaMemset(w->d_status, 0, sizeof(int));
        cudaMemset(w->d_counters, 0, (size_t)w->lay.col_blocks * sizeof(unsigned int));
        if (w->d_mm_counters) cudaMemset(w->d_mm_counters, 0, (size_t)w->mm_n_tiles * MM_MAX_M_TILES * 4 * sizeof(unsigned int));
        if (w->d_nb_counters) cudaMemset(w->d_nb_counters, 0, (size_t)w->nb_tiles * 4 * sizeof(unsigned int));
        if (w->d_nr_counters) cudaMemset(w->d_nr_counters, 0, (size_t)w->nb_tiles * 4 * sizeof(unsigned int));
        return fail(TLLM_ERR_KERNEL, "a bounded wait ran out inside the kernel (code %d: %s)", st,
                    st == MM_ERR_WAIT ? "tensor-core pipeline stalled" : (st == NB_ERR_WAIT ? "decode tensor-core pipeline stalled" : "block table never arrived"));
    }
    return TLLM_OK;
}

int tllm_spmm(tllm_weight* w, const void* X, int x_dtype, int x_layout, int rows, void* Y, int y_dtype, void* stream) {
    if (!w || !X || !Y) return fail(TLLM_ERR_ARG, "tllm_spmm: NULL pointer");
    if (rows <= 0) return fail(TLLM_ERR_ARG, "tllm_spmm: rows must be positive");
    if (x_layout != TLLM_ROW_MAJOR && x_layout != TLLM_COL_MAJOR) return fail(TLLM_ERR_ARG, "tllm_spmm: bad x_layout");
    int rc = check_types(x_dtype, y_dtype, "tllm_spmm");
    if (rc) return rc;
    rc = check_device(w, "tllm_spmm");
    if (rc) return rc;
    const BsLayout& L = w->lay;
    if (rows == 1) x_layout = TLLM_ROW_MAJOR;        // the same memory
    const int x_ld = x_layout == TLLM_ROW_MAJOR ? L.inners : rows;
    return run_product(w, X, x_dtype, x_layout, x_ld, rows, Y, y_dtype, L.columns, 0, w->scale, 0.f, (cudaStream_t)stream);
}

static int spmm_host(tllm_weight* w, const void* X, int x_dtype, int x_layout, int rows, const void* bias, void* Y, int y_dtype, int y_layout, int parts,
                     void (*ready)(void*, size_t, size_t), void* arg) {
    if (!w || !X || !Y) return fail(TLLM_ERR_ARG, "tllm_spmm_host: NULL pointer");
    if (rows <= 0) return fail(TLLM_ERR_ARG, "tllm_spmm_host: rows must be positive");
    int rc = check_types(x_dtype, y_dtype, "tllm_spmm_host");
    if (rc) return rc;
    rc = check_device(w, "tllm_spmm_host");
    if (rc) return rc;
    const BsLayout& L = w->lay;
    const size_t xb = (size_t)rows * L.inners * dtype_size(x_dtype), yb = (size_t)rows * L.columns * dtype_size(y_dtype);
    if (!w->own_stream) CU_TRY(cudaStreamCreateWithFlags(&w->own_stream, cudaStreamNonBlocking));
    if (!w->h_status) CU_TRY(cudaMallocHost((void**)&w->h_status, sizeof(int)));
    int r = ensure(&w->d_x, &w->x_cap, xb, false);
    if (r) return r;
    r = ensure(&w->d_y, &w->y_cap, yb, false);
    if (r) return r;
    // With page-locked buffers the copies are still under way when something fails behind them: they end before the caller has its buffers back.
    struct Drain {
        cudaStream_t st;
        ~Drain() {
            if (st) cudaStreamSynchronize(st);
        }
    } drain{w->own_stream};
    CU_TRY(cudaMemcpyAsync(w->d_x, X, xb, cudaMemcpyHostToDevice, w->own_stream));
    if (bias) {
        r = ensure(&w->d_bias, &w->bias_cap, (size_t)L.columns * dtype_size(y_dtype), false);
        if (r) return r;
        CU_TRY(cudaMemcpyAsync(w->d_bias, bias, (size_t)L.columns * dtype_size(y_dtype), cudaMemcpyHostToDevice, w->own_stream));
    }
    // A column-major result leaves the kernels in that layout; a bias is added to rows first.
    const bool y_col = y_layout != TLLM_ROW_MAJOR && rows > 1;
    if (rows == 1) x_layout = TLLM_ROW_MAJOR;
    const int x_ld = x_layout == TLLM_ROW_MAJOR ? L.inners : rows;
    void* out = w->d_y;
    if (!bias) {
        r = run_product(w, w->d_x, x_dtype, x_layout, x_ld, rows, out, y_dtype, y_col ? rows : L.columns, 0, w->scale, 0.f, w->own_stream, y_col);
        if (r) return r;
    } else {
        r = run_product(w, w->d_x, x_dtype, x_layout, x_ld, rows, out, y_dtype, L.columns, 0, w->scale, 0.f, w->own_stream);
        if (r) return r;
        r = add_bias(out, w->d_bias, y_dtype, rows, L.columns, w->own_stream);
        if (r) return r;
    }
    Workspace ws;
    if (bias && y_col) {
        r = ws.take(w->device, yb, w->own_stream);
        if (r) return r;
        r = turn_out(out, ws.ptr, rows, L.columns, rows, (int)dtype_size(y_dtype), w->own_stream);
        if (r) return r;
        out = ws.ptr;
    }
    CU_TRY(cudaMemcpyAsync(w->h_status, w->d_status, sizeof(int), cudaMemcpyDeviceToHost, w->own_stream));
    if (!ready) CU_TRY(cudaMemcpyAsync(Y, out, yb, cudaMemcpyDeviceToHost, w->own_stream));
    else {
        const auto from = [&](int i) { return i == parts ? yb : yb / parts * i / 4096 * 4096; };
        for (int i = 0; i < parts; ++i) {
            if (!w->part_event[i]) CU_TRY(cudaEventCreateWithFlags(&w->part_event[i], cudaEventDisableTiming));
            CU_TRY(cudaMemcpyAsync((char*)Y + from(i), (const char*)out + from(i), from(i + 1) - from(i), cudaMemcpyDeviceToHost, w->own_stream));
            CU_TRY(cudaEventRecord(w->part_event[i], w->own_stream));
        }
        for (int i = 0; i < parts; ++i) {
            CU_TRY(cudaEventSynchronize(w->part_event[i]));
            ready(arg, from(i), from(i + 1));
        }
    }
    drain.st = nullptr;
    CU_TRY(cudaStreamSynchronize(w->own_stream));
    // the status word came back with the result; only a non-zero one needs the (synchronising) full check
    return *w->h_status ? tllm_weight_check(w) : TLLM_OK;
}

int tllm_spmm_host_bias(tllm_weight* w, const void* X, int x_dtype, int x_layout, int rows, const void* bias, void* Y, int y_dtype, int y_layout) {
    return spmm_host(w, X, x_dtype, x_layout, rows, bias, Y, y_dtype, y_layout, 1, nullptr, nullptr);
}

int tllm_spmm_host(tllm_weight* w, const void* X, int x_dtype, int x_layout, int rows, void* Y, int y_dtype, int y_layout) {
    return spmm_host(w, X, x_dtype, x_layout, rows, nullptr, Y, y_dtype, y_layout, 1, nullptr, nullptr);
}

int tllm_spmm_host_parts(tllm_weight* w, const void* X, int x_dtype, int x_layout, int rows, void* Y, int y_dtype, int y_layout, int parts,
                         void (*ready)(void* arg, size_t from, size_t to), void* arg) {
    if (!ready || parts < 1 || parts > TLLM_HOST_PARTS) return fail(TLLM_ERR_ARG, "tllm_spmm_host_parts: 1 to %d parts and a function", TLLM_HOST_PARTS);
    return spmm_host(w, X, x_dtype, x_layout, rows, nullptr, Y, y_dtype, y_layout, parts, ready, arg);
}

}  // extern "C"

// ------------------------------------------------------------------------------------------------------
// tllm_spmm_static_scratch: the same product as tllm_spmm, for callers that must not allocate.
//
// Some callers run where device allocation is off the table: a serving loop whose memory pool was carved up
// at start-up and is policed for late cudaMalloc calls, code that executes under a framework allocator it
// must not bypass, or a latency-critical path where an allocation (which may synchronise the device) is not
// acceptable.  tllm_spmm takes a stream-ordered workspace for some calls, and the handle it uses had its split-K scratch
// allocated with cudaMalloc when it was created.  This entry point uses neither: partial sums
// and arrival counters live in the fixed array below, which every GPU that loads this library carries until
// the process exits.  Its size is the limit on what one call may ask for.  (The 4-byte status word stays the
// handle's own -- it exists since the handle was created -- so that tllm_weight_check reports a kernel that
// gave up on a wait on this path as on every other.)
// ------------------------------------------------------------------------------------------------------
#define TLLM_STATIC_SCRATCH_CELLS (1u << 20)   // 4-byte partial sums: k_splits * rows_per_launch * columns must fit
#define TLLM_STATIC_COUNTERS 4096u
#define TLLM_STATIC_SCRATCH_BYTES (TLLM_STATIC_SCRATCH_CELLS * 4u + TLLM_STATIC_COUNTERS * 4u)

static __device__ __align__(256) unsigned char g_static_scratch[TLLM_STATIC_SCRATCH_BYTES];

namespace {
std::mutex g_static_mu;
void* g_static_ptr[64] = {};   // device address of g_static_scratch, per device ordinal

// In host code `g_static_scratch` is only a handle for the runtime, not an address a kernel could use: the
// device address has to be asked for, once per device, with that device current.
int static_scratch_address(void** out) {
    int dev = 0;
    CU_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(TLLM_ERR_ARG, "tllm_spmm_static_scratch: device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_ptr[dev]) {
        void* ptr = nullptr;
        CU_TRY(cudaGetSymbolAddress(&ptr, g_static_scratch));
        if (!ptr) return fail(TLLM_ERR_CUDA, "tllm_spmm_static_scratch: cudaGetSymbolAddress returned a null address");
        g_static_ptr[dev] = ptr;
    }
    *out = g_static_ptr[dev];
    return TLLM_OK;
}
}  // namespace

extern "C" int tllm_spmm_static_scratch(tllm_weight* w, const void* X, int x_dtype, int x_layout, int rows, void* Y, int y_dtype,
                                        void* stream) {
    if (!w || !X || !Y) return fail(TLLM_ERR_ARG, "tllm_spmm_static_scratch: NULL pointer");
    if (rows <= 0) return fail(TLLM_ERR_ARG, "tllm_spmm_static_scratch: rows must be positive");
    if (x_layout != TLLM_ROW_MAJOR && x_layout != TLLM_COL_MAJOR) return fail(TLLM_ERR_ARG, "tllm_spmm_static_scratch: bad x_layout");
    int rc = check_types(x_dtype, y_dtype, "tllm_spmm_static_scratch");
    if (rc) return rc;
    rc = check_device(w, "tllm_spmm_static_scratch");
    if (rc) return rc;
    const BsLayout& L = w->lay;
    const int per_launch = rows < w->max_rows ? rows : w->max_rows;
    const uint64_t cells = L.k_splits > 1 ? (uint64_t)L.k_splits * (uint64_t)per_launch * (uint64_t)L.columns : 0;
    if (cells > TLLM_STATIC_SCRATCH_CELLS)
        return fail(TLLM_ERR_ARG,
                    "tllm_spmm_static_scratch: %d K-splits x %d rows x %d columns = %llu partial sums exceed the built-in scratch of %u; "
                    "use tllm_spmm, fewer rows per call, or a weight packed with fewer K-splits",
                    L.k_splits, per_launch, L.columns, (unsigned long long)cells, (unsigned)TLLM_STATIC_SCRATCH_CELLS);
    if ((unsigned)L.col_blocks > TLLM_STATIC_COUNTERS) return fail(TLLM_ERR_ARG, "tllm_spmm_static_scratch: too many column blocks for the built-in counters");
    void* base = nullptr;
    rc = static_scratch_address(&base);
    if (rc) return rc;
    unsigned char* scratch = (unsigned char*)base;
    unsigned int* counters = (unsigned int*)(scratch + (size_t)TLLM_STATIC_SCRATCH_CELLS * 4u);
    cudaStream_t st = (cudaStream_t)stream;
    // The array keeps whatever the previous call left.  Partial sums are overwritten before they are read;
    // the counters must start at zero, so they are cleared here, in stream order.
    CU_TRY(cudaMemsetAsync(counters, 0, (size_t)TLLM_STATIC_COUNTERS * 4u, st));
    const int x_ld = x_layout == TLLM_ROW_MAJOR ? L.inners : rows;
    return run_gather(w, X, x_dtype, x_layout, x_ld, rows, Y, y_dtype, L.columns, 0, w->scale, 0.f, Scratch{scratch, counters}, st);
}

extern "C" {

int tllm_mlp_create(const int8_t* w_gate, const int8_t* w_up, const int8_t* w_down, int hidden, int intermediate, float s_gate,
                    float s_up, float s_down, const tllm_pack_opts* opts, tllm_mlp** out) {
    if (!w_gate || !w_up || !w_down || hidden <= 0 || intermediate <= 0 || !out) return fail(TLLM_ERR_ARG, "tllm_mlp_create: bad argument");
    *out = nullptr;
    std::vector<int8_t> gu((size_t)hidden * 2 * intermediate);
    for (int k = 0; k < hidden; ++k) {
        const int8_t* g = w_gate + (size_t)k * intermediate;
        const int8_t* u = w_up + (size_t)k * intermediate;
        int8_t* d = gu.data() + (size_t)k * 2 * intermediate;
        for (int c = 0; c < intermediate; ++c) {
            d[2 * c] = g[c];
            d[2 * c + 1] = u[c];
        }
    }
    tllm_mlp* m = new tllm_mlp();
    m->hidden = hidden;
    m->inter = intermediate;
    m->s_gate = s_gate;
    m->s_up = s_up;
    int rc = tllm_weight_create_dense(gu.data(), hidden, 2 * intermediate, 1.f, opts, &m->gate_up);
    if (rc == TLLM_OK) rc = tllm_weight_create_dense(w_down, intermediate, hidden, s_down, opts, &m->down);
    if (rc == TLLM_OK) {
        m->h_cap = (size_t)16 * intermediate * 4;
        cudaError_t e = cudaMalloc(&m->d_h, m->h_cap);
        if (e != cudaSuccess) rc = fail(TLLM_ERR_CUDA, "cudaMalloc failed: %s", cudaGetErrorString(e));
    }
    if (rc != TLLM_OK) {
        tllm_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return TLLM_OK;
}

int tllm_mlp_create_cpu_format(int kind, int group, int chunk, int ri32, const int32_t* meta_gate, const void* ri_gate,
                               const int32_t* meta_up, const void* ri_up, const int32_t* meta_down, const void* ri_down, int hidden,
                               int intermediate, const tllm_pack_opts* opts, tllm_mlp** out) {
    if (!meta_gate || !ri_gate || !meta_up || !ri_up || !meta_down || !ri_down || hidden <= 0 || intermediate <= 0 || !out)
        return fail(TLLM_ERR_ARG, "tllm_mlp_create_cpu_format: bad argument");
    if (kind < 1 || kind > 5) return fail(TLLM_ERR_ARG, "tllm_mlp_create_cpu_format: kind must be 1..5 (the single-array formats)");
    *out = nullptr;
    std::vector<int8_t> g, u, d;
    const char* msg = tllm::decode_cpu_format(kind, group, chunk, meta_gate, ri_gate, ri32, 0, intermediate, hidden, &g);
    if (!msg) msg = tllm::decode_cpu_format(kind, group, chunk, meta_up, ri_up, ri32, 0, intermediate, hidden, &u);
    if (!msg) msg = tllm::decode_cpu_format(kind, group, chunk, meta_down, ri_down, ri32, 0, hidden, intermediate, &d);
    if (msg) return fail(TLLM_ERR_ARG, "tllm_mlp_create_cpu_format: %s", msg);
    return tllm_mlp_create(g.data(), u.data(), d.data(), hidden, intermediate, 1.f, 1.f, 1.f, opts, out);
}

int tllm_mlp_destroy(tllm_mlp* m) {
    if (!m) return TLLM_OK;
    tllm_weight_destroy(m->gate_up);
    tllm_weight_destroy(m->down);
    cudaFree(m->d_h);
    cudaFree(m->d_x);
    cudaFree(m->d_y);
    cudaFree(m->d_hh);
    delete m;
    return TLLM_OK;
}

int tllm_mlp_forward(tllm_mlp* m, const void* X, int x_dtype, int rows, void* Y, void* H, void* stream) {
    return tllm_mlp_forward_ex(m, X, x_dtype, rows, Y, x_dtype, H, stream);
}

int tllm_mlp_forward_ex(tllm_mlp* m, const void* X, int x_dtype, int rows, void* Y, int y_dtype, void* H, void* stream) {
    if (!m || !X || !Y) return fail(TLLM_ERR_ARG, "tllm_mlp_forward: NULL pointer");
    if (y_dtype != TLLM_F32 && y_dtype != TLLM_F16 && y_dtype != TLLM_BF16) return fail(TLLM_ERR_ARG, "tllm_mlp_forward: unsupported y_dtype");
    if (rows <= 0) return fail(TLLM_ERR_ARG, "tllm_mlp_forward: rows must be positive");
    if (x_dtype != TLLM_F32 && x_dtype != TLLM_F16 && x_dtype != TLLM_BF16) return fail(TLLM_ERR_ARG, "tllm_mlp_forward: unsupported dtype");
    int rc = check_device(m->gate_up, "tllm_mlp_forward");
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    // the two products pick their kernel independently (gate and up share the first one: its epilogue applies SiLU and the product)
    Workspace ws;
    if (!H && x_dtype == TLLM_F32 && choose_kernel(m->gate_up, X, x_dtype, TLLM_ROW_MAJOR, m->hidden, rows) == KERNEL_MMA &&
        choose_kernel(m->down, X, x_dtype, TLLM_ROW_MAJOR, m->inter, rows) == KERNEL_MMA) {
        // the intermediate result goes from one kernel to the other as the three planes that the second one reads
        const int ld = (m->inter + 7) / 8 * 8;
        rc = ws.take(m->gate_up->device, (size_t)3 * rows * ld * 2, st);
        if (rc) return rc;
        rc = run_mm(bits_view(m->gate_up), X, x_dtype, TLLM_ROW_MAJOR, m->hidden, rows, ws.ptr, x_dtype, ld, 1, m->s_gate, m->s_up, st, false, true, (long long)rows * ld);
        if (rc) return rc;
        return run_mm_planes(bits_view(m->down), (const unsigned short*)ws.ptr, rows, (size_t)ld * 2, rows, Y, y_dtype, m->hidden, m->down->scale, st);
    }
    char* h = (char*)(H ? H : m->d_h);
    const size_t h_bytes = (size_t)rows * m->inter * dtype_size(x_dtype);
    if (!H && h_bytes > m->h_cap) {
        rc = ws.take(m->gate_up->device, h_bytes, st);
        if (rc) return rc;
        h = (char*)ws.ptr;
    }
    rc = run_product(m->gate_up, X, x_dtype, TLLM_ROW_MAJOR, m->hidden, rows, h, x_dtype, m->inter, 1, m->s_gate, m->s_up, st);
    if (rc) return rc;
    return run_product(m->down, h, x_dtype, TLLM_ROW_MAJOR, m->inter, rows, Y, y_dtype, m->hidden, 0, m->down->scale, 0.f, st);
}

// [a][b] -> [b][a] for elements of `e` bytes
static void transpose_bytes(const void* src, void* dst, size_t a, size_t b, size_t e) {
    const char* s = (const char*)src;
    char* d = (char*)dst;
    for (size_t i = 0; i < a; ++i)
        for (size_t j = 0; j < b; ++j) memcpy(d + (j * a + i) * e, s + (i * b + j) * e, e);
}

int tllm_mlp_forward_host(tllm_mlp* m, void* X, int x_dtype, int x_layout, int rows, void* H) {
    if (!m || !X) return fail(TLLM_ERR_ARG, "tllm_mlp_forward_host: NULL pointer");
    if (rows <= 0) return fail(TLLM_ERR_ARG, "tllm_mlp_forward_host: rows must be positive");
    if (x_dtype != TLLM_F32 && x_dtype != TLLM_F16 && x_dtype != TLLM_BF16) return fail(TLLM_ERR_ARG, "tllm_mlp_forward_host: unsupported dtype");
    if (x_layout != TLLM_ROW_MAJOR && x_layout != TLLM_COL_MAJOR) return fail(TLLM_ERR_ARG, "tllm_mlp_forward_host: unknown layout");
    tllm_weight* w = m->gate_up;
    int rc = check_device(w, "tllm_mlp_forward_host");
    if (rc) return rc;
    const size_t e = dtype_size(x_dtype), xb = (size_t)rows * m->hidden * e, hb = (size_t)rows * m->inter * e;
    if (!w->own_stream) CU_TRY(cudaStreamCreateWithFlags(&w->own_stream, cudaStreamNonBlocking));
    if (!w->h_status) CU_TRY(cudaMallocHost((void**)&w->h_status, sizeof(int)));
    rc = ensure(&m->d_x, &m->x_cap, xb, false);
    if (rc) return rc;
    rc = ensure(&m->d_y, &m->y_cap, xb, false);
    if (rc) return rc;
    rc = ensure(&m->d_hh, &m->hh_cap, hb, false);
    if (rc) return rc;
    // a column-major caller ([hidden][rows], rows contiguous) is turned on the host: the block itself is row-major
    const bool turn = x_layout == TLLM_COL_MAJOR && rows > 1;
    std::vector<char> tx, th;
    void* hx = X;
    if (turn) {
        tx.resize(xb);
        transpose_bytes(X, tx.data(), (size_t)m->hidden, (size_t)rows, e);
        hx = tx.data();
        if (H) th.resize(hb);
    }
    CU_TRY(cudaMemcpyAsync(m->d_x, hx, xb, cudaMemcpyHostToDevice, w->own_stream));
    rc = tllm_mlp_forward(m, m->d_x, x_dtype, rows, m->d_y, m->d_hh, w->own_stream);
    if (rc) return rc;
    CU_TRY(cudaMemcpyAsync(hx, m->d_y, xb, cudaMemcpyDeviceToHost, w->own_stream));
    if (H) CU_TRY(cudaMemcpyAsync(turn ? (void*)th.data() : H, m->d_hh, hb, cudaMemcpyDeviceToHost, w->own_stream));
    CU_TRY(cudaMemcpyAsync(w->h_status, w->d_status, sizeof(int), cudaMemcpyDeviceToHost, w->own_stream));
    CU_TRY(cudaStreamSynchronize(w->own_stream));
    if (turn) {
        transpose_bytes(tx.data(), X, (size_t)rows, (size_t)m->hidden, e);
        if (H) transpose_bytes(th.data(), H, (size_t)rows, (size_t)m->inter, e);
    }
    if (*w->h_status) return tllm_weight_check(w);
    return tllm_weight_check(m->down);
}

int tllm_mlp_get_info(const tllm_mlp* m, tllm_weight_info* gate_up, tllm_weight_info* down) {
    if (!m) return fail(TLLM_ERR_ARG, "tllm_mlp_get_info: NULL");
    if (gate_up) tllm_weight_get_info(m->gate_up, gate_up);
    if (down) tllm_weight_get_info(m->down, down);
    return TLLM_OK;
}

int tllm_add_rmsnorm(void* x, const void* delta, const void* weight, void* h, int dtype, int rows, int hidden, float eps, void* stream) {
    if (!x || !h || rows < 0 || hidden <= 0) return fail(TLLM_ERR_ARG, "tllm_add_rmsnorm: bad argument");
    if (dtype != TLLM_F32 && dtype != TLLM_F16 && dtype != TLLM_BF16) return fail(TLLM_ERR_ARG, "tllm_add_rmsnorm: unsupported dtype");
    const int vec = dtype == TLLM_F32 ? 4 : 8;
    if (hidden % vec || ((uintptr_t)x | (uintptr_t)h | (uintptr_t)delta | (uintptr_t)weight) % 16)
        return fail(TLLM_ERR_ARG, "tllm_add_rmsnorm: hidden must be a multiple of %d and the pointers 16-byte aligned", vec);
    if (rows == 0) return TLLM_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == TLLM_F32) CU_TRY((launch_add_rmsnorm<float, float>(x, delta, weight, h, rows, hidden, eps, st)));
    else if (dtype == TLLM_F16) CU_TRY((launch_add_rmsnorm<__half, __half>(x, delta, weight, h, rows, hidden, eps, st)));
    else CU_TRY((launch_add_rmsnorm<__nv_bfloat16, __nv_bfloat16>(x, delta, weight, h, rows, hidden, eps, st)));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return TLLM_OK;
}

}  // extern "C"

namespace {
// one launch of an attention kernel; `parts` blocks in x form a cluster
template <typename... P, typename... A>
int launch_attention(void (*kern)(P...), std::once_flag (&once)[64], dim3 grid, int threads, size_t smem, int parts, cudaStream_t st, A... args) {
    int dev = 0;
    CU_TRY(cudaGetDevice(&dev));
    cudaError_t err = cudaSuccess;
    std::call_once(once[dev & 63], [&] { err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); });
    CU_TRY(err);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2] = {pdl_attribute(), {}};
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)parts, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = parts > 1 ? 2 : 1;
    CU_TRY(cudaLaunchKernelEx(&cfg, kern, args...));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return TLLM_OK;
}
constexpr float LOG2E = 1.44269504f;

template <int HD>
int causal_f32(const void* qkv, void* out, int batch, int rows, int heads, int kv_heads, cudaStream_t st) {
    static std::once_flag once[64];
    return launch_attention(prompt_attention_f32_kernel<HD>, once, dim3((unsigned)((rows + AM_KEYS - 1) / AM_KEYS), (unsigned)heads, (unsigned)batch), AM_P_THREADS,
                            am_f32_smem<HD>(), 1, st, (const float*)qkv, (float*)out, rows, heads, kv_heads, (heads + 2 * kv_heads) * HD, LOG2E / sqrtf((float)HD));
}
template <typename T, int HD>
int causal_16bit(const void* qkv, void* out, int batch, int rows, int heads, int kv_heads, cudaStream_t st) {
    static std::once_flag once[64];
    return launch_attention(prompt_attention_kernel<T, HD>, once, dim3((unsigned)((rows + AM_KEYS - 1) / AM_KEYS), (unsigned)heads, (unsigned)batch), AM_P_THREADS,
                            am_prompt_smem<HD>(), 1, st, (const T*)qkv, (T*)out, rows, heads, kv_heads, (heads + 2 * kv_heads) * HD, LOG2E / sqrtf((float)HD));
}
// A cluster of up to eight blocks per key head, as many as still fit two to an SM, with 128 keys each at least.  (Twice as many blocks than
// that, in a second wave: 11 us instead of 7.5 at 16 sequences of 1024 keys, 8 key heads of 64.)
template <typename T, int HD>
int decode_16bit(const void* qkv, void* k, void* v, void* out, int rows, int heads, int kv_heads, int len, int64_t seq_step, int64_t head_step, int sms, cudaStream_t st) {
    static std::once_flag once[64];
    int parts = 1;
    while (parts < 8 && (long long)rows * kv_heads * parts <= sms && len / (2 * parts) >= 128) parts *= 2;
    return launch_attention(decode_attention_kernel<T, HD>, once, dim3((unsigned)parts, (unsigned)kv_heads, (unsigned)rows), AM_THREADS, am_decode_smem<HD>(), parts, st,
                            (const T*)qkv, (T*)k, (T*)v, (T*)out, heads, kv_heads, len, (long long)seq_step, (long long)head_step, LOG2E / sqrtf((float)HD));
}
}  // namespace

extern "C" {

int tllm_causal_attention(const void* qkv, void* out, int dtype, int batch, int rows, int heads, int kv_heads, int head_dim, void* stream) {
    if (!qkv || !out || batch <= 0 || rows <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads) return fail(TLLM_ERR_ARG, "tllm_causal_attention: bad argument");
    if (head_dim != 64 && head_dim != 128) return fail(TLLM_ERR_ARG, "tllm_causal_attention: heads of %d values (64 and 128 are built)", head_dim);
    if (batch > 65535 || heads > 65535 || ((uintptr_t)qkv | (uintptr_t)out) % 16) return fail(TLLM_ERR_ARG, "tllm_causal_attention: too many heads or unaligned pointers");
    cudaStream_t st = (cudaStream_t)stream;
    const bool narrow = head_dim == 64;
    if (dtype == TLLM_F32) return narrow ? causal_f32<64>(qkv, out, batch, rows, heads, kv_heads, st) : causal_f32<128>(qkv, out, batch, rows, heads, kv_heads, st);
    if (dtype == TLLM_F16) return narrow ? causal_16bit<__half, 64>(qkv, out, batch, rows, heads, kv_heads, st) : causal_16bit<__half, 128>(qkv, out, batch, rows, heads, kv_heads, st);
    if (dtype == TLLM_BF16)
        return narrow ? causal_16bit<__nv_bfloat16, 64>(qkv, out, batch, rows, heads, kv_heads, st) : causal_16bit<__nv_bfloat16, 128>(qkv, out, batch, rows, heads, kv_heads, st);
    return fail(TLLM_ERR_ARG, "tllm_causal_attention: unsupported dtype");
}

int tllm_decode_attention(const void* qkv, void* k_cache, void* v_cache, void* out, int dtype, int rows, int heads, int kv_heads, int head_dim, int len, int64_t seq_step,
                          int64_t head_step, void* stream) {
    if (!qkv || !k_cache || !v_cache || !out || rows <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || len < 0) return fail(TLLM_ERR_ARG, "tllm_decode_attention: bad argument");
    if ((head_dim != 64 && head_dim != 128) || heads / kv_heads > AM_MAX_GROUP || (dtype != TLLM_F16 && dtype != TLLM_BF16))
        return fail(TLLM_ERR_ARG, "tllm_decode_attention: 16-bit heads of 64 or 128 values, at most %d query heads per key head", AM_MAX_GROUP);
    if (rows > 65535 || kv_heads > 65535 || ((uintptr_t)qkv | (uintptr_t)out | (uintptr_t)k_cache | (uintptr_t)v_cache) % 16 || seq_step % 8 || head_step % 8)
        return fail(TLLM_ERR_ARG, "tllm_decode_attention: too many sequences or unaligned pointers");
    int dev = 0, sms = 0;
    CU_TRY(cudaGetDevice(&dev));
    CU_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    cudaStream_t st = (cudaStream_t)stream;
#define AM_DECODE(T) (head_dim == 64 ? decode_16bit<T, 64>(qkv, k_cache, v_cache, out, rows, heads, kv_heads, len, seq_step, head_step, sms, st) \
                                     : decode_16bit<T, 128>(qkv, k_cache, v_cache, out, rows, heads, kv_heads, len, seq_step, head_step, sms, st))
    return dtype == TLLM_F16 ? AM_DECODE(__half) : AM_DECODE(__nv_bfloat16);
#undef AM_DECODE
}

int tllm_silu_mul(void* g, const void* u, int dtype, int64_t n, void* stream) {
    if (!g || !u || n < 0) return fail(TLLM_ERR_ARG, "tllm_silu_mul: bad argument");
    if (dtype != TLLM_F32 && dtype != TLLM_F16 && dtype != TLLM_BF16) return fail(TLLM_ERR_ARG, "tllm_silu_mul: unsupported dtype");
    if (n == 0) return TLLM_OK;
    silu_mul_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(g, u, dtype, (long long)n);
    CU_TRY(cudaGetLastError());
    g_launches.fetch_add(1, std::memory_order_relaxed);
    return TLLM_OK;
}

}  // extern "C"
