// tsqr.cu -- TSQR host driver and C ABI entry points (plain precision path).
//
// Replaces the reference host driver tsqr<T> (TallShinnyQR.h:86-148).  The
// reference picks between a single persistent launch (m <= NUM_SM*BLOCK_SIZE)
// and a chunk loop + second TSQR + fix-up GEMM; here one reduction tree of
// runtime height covers every m: one factor launch per level going up, one
// apply launch per level coming down, all on the caller's stream, with no
// grid-wide spin barrier (kernelQR.h:297, :374) and no global state, so
// concurrent calls on different streams with different workspaces are safe.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "../../include/tsqr_gb300.h"
#include "internal.h"
#include "tile_f64.cuh"
#include "tsqr_kernels.cuh"

namespace tsqr {

thread_local LaunchLog* tl_log = nullptr;

// One level of 512-row tiles, 33 to 64 columns wide (panels.cu).
constexpr int kWideRows = 512;
void factor_wide_level(const FactorParams<float>& p, cudaStream_t s);
// One level of more than one wave of 512-row tiles, 17 to 32 columns wide
// (panels.cu); map: the level for boxes of 256 rows x 16 columns, or null.
void factor_panel_level(const FactorParams<float>& p, const CUtensorMap* map, cudaStream_t s);

namespace {

// cuTensorMapEncodeTiled, looked up once through the runtime (no link
// against the driver library).  Null if the driver does not offer it.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        (void)cudaGetLastError();
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}

}  // namespace

bool tensor_map_f32(CUtensorMap* map, const float* base, int64_t ld, int64_t rows, int64_t cols, int box_rows,
                    int box_cols, bool swizzle128) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc || (reinterpret_cast<uintptr_t>(base) % 16) != 0 || ld % 4 != 0 || rows < 1 || cols < 1) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)rows, (cuuint64_t)cols};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(float)};
    const cuuint32_t box[2] = {(cuuint32_t)box_rows, (cuuint32_t)box_cols};
    const cuuint32_t estr[2] = {1u, 1u};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

namespace {

// Tensor map of an FP32 level matrix (h rows x n columns) for boxes of 256
// rows x nbox columns.
bool level_tensor_map(CUtensorMap* map, const float* M, int64_t ld, int64_t h, int n, int nbox) {
    return tensor_map_f32(map, M, ld, h, n, 256, nbox, false);
}

// FP32 Q assembly of one level.  Where the level's CTAs need no third slot per
// SM, an instantiation with more registers keeps more loads in flight: at 32
// columns and 32 tiles 10.3 us against 12.3 us, while at 8192 tiles three
// CTAs per SM take 277 us and two 329 us.
template <int NMAX, int ROWS>
void apply_level_f32(const ApplyParams<float>& p, cudaStream_t s) {
    using A = ApplyF32<NMAX, ROWS>;
    constexpr int kFew = A::kResident > 2 ? 2 : 1;
    static PerDeviceOnce attr;
    attr.run([] {
        cudaFuncSetAttribute(apply_tiles_f32<NMAX, ROWS, kFew>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)A::kSmem);
        cudaFuncSetAttribute(apply_tiles_f32<NMAX, ROWS, A::kResident>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)A::kSmem);
    });
    const dim3 grid((unsigned)p.ntiles);
    if (p.ntiles <= (int64_t)device_sm_count() * kFew)
        launch_pdl(apply_tiles_f32<NMAX, ROWS, kFew>, grid, dim3(A::NT), A::kSmem, s, p);
    else
        launch_pdl(apply_tiles_f32<NMAX, ROWS, A::kResident>, grid, dim3(A::NT), A::kSmem, s, p);
}

// FP64 Q assembly of one level.  us, one CTA per tile / clusters of four: 108
// tiles of 256 x 32 at level 0 88 / 65, 1024 tiles 544 / 543; above level 0,
// where half the products are skipped, 128 tiles 69 / 79, 16 tiles 69 / 23,
// the 64-row root 57 / 20.  So: clusters for up to 4 tiles per SM at level 0,
// above it while the clusters are resident at once (2 CTAs per SM).
template <int NMAX, int ROWS>
void apply_level_f64(const ApplyParams<double>& p, cudaStream_t s) {
    constexpr int kMinB = NMAX > 8 ? 2 : 3;
    using A1 = ApplyF64<NMAX, ROWS, 1>;
    using A4 = ApplyF64<NMAX, ROWS, 4>;
    static PerDeviceOnce attr;
    attr.run([] {
        constexpr auto kMax = cudaFuncAttributeMaxDynamicSharedMemorySize;
        cudaFuncSetAttribute(apply_f64_tiles<NMAX, ROWS, 1, kMinB, false>, kMax, (int)A1::kSmem);
        cudaFuncSetAttribute(apply_f64_tiles<NMAX, ROWS, 1, kMinB, true>, kMax, (int)A1::kSmem);
        cudaFuncSetAttribute(apply_f64_tiles<NMAX, ROWS, 4, kMinB, false>, kMax, (int)A4::kSmem);
        cudaFuncSetAttribute(apply_f64_tiles<NMAX, ROWS, 4, kMinB, true>, kMax, (int)A4::kSmem);
    });
    const int64_t sms = device_sm_count();
    const bool cluster = p.stack ? 4 * p.ntiles <= 2 * sms : p.ntiles < 4 * sms;
    const dim3 grid((unsigned)(cluster ? 4 * p.ntiles : p.ntiles));
    auto go = [&](void (*kernel)(ApplyParams<double>), size_t smem) {
        launch_pdl_cluster(kernel, grid, dim3(256), smem, s, cluster ? 4 : 1, p);
    };
    if (cluster)
        go(p.stack ? apply_f64_tiles<NMAX, ROWS, 4, kMinB, true> : apply_f64_tiles<NMAX, ROWS, 4, kMinB, false>,
           A4::kSmem);
    else
        go(p.stack ? apply_f64_tiles<NMAX, ROWS, 1, kMinB, true> : apply_f64_tiles<NMAX, ROWS, 1, kMinB, false>,
           A1::kSmem);
}

template <typename T, int NMAX, int ROWS>
void apply_level(const ApplyParams<T>& p, cudaStream_t s) {
    if constexpr (std::is_same<T, float>::value)
        apply_level_f32<NMAX, ROWS>(p, s);
    else
        apply_level_f64<NMAX, ROWS>(p, s);
}

template <int NMAX, int NT, int RPT, int MINB>
struct TileCfg {
    static constexpr int kRows = NT * RPT;
    static void factor(const FactorParams<float>& p, int grid, cudaStream_t s) {
        launch_pdl(factor_tiles<NMAX, NT, RPT, MINB>, dim3(grid), dim3(NT), 0, s, p);
    }
    static void apply(const ApplyParams<float>& p, int, cudaStream_t s) { apply_level<float, NMAX, kRows>(p, s); }
};

// Factor on column-split tiles (factor_split_tiles: NMAX/CW warps per
// 32*RPT-row tile), with the same apply kernel as TileCfg.
template <typename T, int NMAX, int CW, int RPT, int MINB, bool N64 = false>
struct SplitCfg {
    static constexpr int kRows = 32 * RPT;
    static void factor(const FactorParams<T>& p, int grid, cudaStream_t s) {
        // A single-tile level (the root) of h rows takes the same kernel with
        // just enough rows per lane (32 * rpt >= h): every step issues the
        // FMAs of all RPT rows of a lane, so a 64-row root on the 512-row
        // kernel would spend 7/8 of them on zero rows.
        constexpr int W32 = 32 * (NMAX / CW);
        if constexpr (N64)
            if (p.clear) cudaMemsetAsync(p.clear, 0, sizeof(int), s);
        if constexpr (std::is_same<T, double>::value) {
            // FP64 levels above the first, us per tile of a level with one tile
            // per SM, this kernel / the column split: 256 x 32 141 / 194, 64 x 32
            // 98 / 108, 512 x 16 83 / 102, 512 x 8 36 / 51.  Level 0 has no
            // triangles to use; there the column split keeps all four warps'
            // FP64 time busier (262,144 x 32: 979 us against 1170 us).
            constexpr int CL = NMAX == 32 ? 8 : 4;
            static_assert(StackTile<NMAX, CL, 16>::kRows == kRows, "one tile height for all levels");
            if (p.stack)
                return (void)launch_pdl(factor_stack_tiles<NMAX, CL, 16>, dim3(grid), dim3(128), 0, s, p);
        }
        if constexpr (RPT > 2 && NMAX <= 64)
            if (p.ntiles == 1 && p.h <= 64)
                return (void)launch_pdl(factor_split_tiles<T, NMAX, CW, 2, 1, N64>, dim3(1), dim3(W32), 0, s, p);
        if constexpr (RPT > 4)
            if (p.ntiles == 1 && p.h <= 128)
                return (void)launch_pdl(factor_split_tiles<T, NMAX, CW, 4, 1, N64>, dim3(1), dim3(W32), 0, s, p);
        if constexpr (RPT > 8)
            if (p.ntiles == 1 && p.h <= 256)
                return (void)launch_pdl(factor_split_tiles<T, NMAX, CW, 8, 1, N64>, dim3(1), dim3(W32), 0, s, p);
        if constexpr (std::is_same<T, float>::value && RPT == 16 && NMAX == 32 && !N64) {
            // levels of more than one wave: two 16-column panels (panels.cu)
            if (p.ntiles > (int64_t)device_sm_count() * MINB) {
                CUtensorMap map;
                const bool tma = p.ntiles * kRows <= INT32_MAX && level_tensor_map(&map, p.M, p.ld, p.h, p.n, 16);
                return factor_panel_level(p, tma ? &map : nullptr, s);
            }
        }
        if constexpr (std::is_same<T, float>::value && RPT == 16 && NMAX < 32 && !N64) {
            // levels with several tiles per resident CTA: tiles staged by TMA
            // into shared memory, the next one copied while the current one
            // is factored (persistent CTAs); levels of one wave or less were
            // 2 us slower with it and keep the plain loads.
            const int64_t resident = (int64_t)device_sm_count() * MINB;
            CUtensorMap map;
            if (p.ntiles >= 2 * resident && p.ntiles * kRows <= INT32_MAX &&
                level_tensor_map(&map, p.M, p.ld, p.h, p.n, NMAX)) {
                constexpr size_t smem = tma_stage_bytes<T, NMAX, CW, RPT>();
                static PerDeviceOnce attr;
                attr.run([] {
                    cudaFuncSetAttribute(factor_split_tiles_tma<T, NMAX, CW, RPT, MINB>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                });
                const int g = (int)std::min<int64_t>(p.ntiles, resident);
                if (p.clear) cudaMemsetAsync(p.clear, 0, sizeof(int), s);
                return (void)launch_pdl(factor_split_tiles_tma<T, NMAX, CW, RPT, MINB>, dim3(g), dim3(W32), smem, s,
                                        p, map);
            }
        }
        launch_pdl(factor_split_tiles<T, NMAX, CW, RPT, MINB, N64>, dim3(grid), dim3(W32), 0, s, p);
    }
    static void apply(const ApplyParams<T>& p, int, cudaStream_t s) { apply_level<T, NMAX, kRows>(p, s); }
};

// FP32 tiles 33 to 64 columns wide, factored as two panels (panels.cu).
struct WideCfg {
    static constexpr int kRows = kWideRows;
    static void factor(const FactorParams<float>& p, int, cudaStream_t s) { factor_wide_level(p, s); }
    static void apply(const ApplyParams<float>& p, int, cudaStream_t s) { apply_level<float, 64, kRows>(p, s); }
};

template <typename T>
struct KernelSet {
    int rows = 0;  // tile height B
    void (*factor)(const FactorParams<T>&, int, cudaStream_t) = nullptr;
    void (*apply)(const ApplyParams<T>&, int, cudaStream_t) = nullptr;
};

template <typename C, typename T>
KernelSet<T> make_set() {
    KernelSet<T> k;
    k.rows = C::kRows;
    k.factor = &C::factor;
    k.apply = &C::apply;
    return k;
}

// Tile configuration per (dtype, n).  The tile height B is the tree arity
// times n; B >= 4n keeps the stacked-R levels at most a quarter of the level
// below, and the tile stays in registers (RPT rows x NMAX columns/thread).
KernelSet<float> pick(float*, int n) {
    // Level-0 factor times at 4,194,304 rows, column-split (factor_split_tiles)
    // against the earlier one-thread-per-row-slice kernel (factor_tiles):
    // n = 16: 0.20 vs 0.49 ms; n = 32: 0.72 vs 0.98 ms.  2,097,152 x 64: two
    // panels (factor_panel_tiles) 1.07 ms, column-split in one 1.64 ms.
    // n = 64 keeps 512-row tiles (256-row tiles double the stacked-R level).
    if (n <= 8) return make_set<TileCfg<8, 256, 4, 3>, float>();
    if (n <= 16) return make_set<SplitCfg<float, 16, 4, 16, 4>, float>();
    if (n <= 32) return make_set<SplitCfg<float, 32, 4, 16, 2>, float>();
    if (n <= 64) return make_set<WideCfg, float>();
    return KernelSet<float>();
}
KernelSet<double> pick(double*, int n) {
    // column split against one thread per row slice, level 0: 2,097,152 x 32
    // 7.5 against 19.0 ms; 262,144 x 16 282 against 596 us, x 8 76 against 204 us
    if (n <= 8) return make_set<SplitCfg<double, 8, 4, 16, 4>, double>();
    if (n <= 16) return make_set<SplitCfg<double, 16, 4, 16, 2>, double>();
    if (n <= 32) return make_set<SplitCfg<double, 32, 4, 8, 3>, double>();
    return KernelSet<double>();
}

template <typename T>
struct Level {
    T* M;
    int64_t ld;
    int64_t h;
    int64_t ntiles;
};

constexpr size_t kAlign = 256;

// Lays the tree out in the workspace.  With base == nullptr only the size is
// computed.  Returns the bytes used.
template <typename T>
size_t plan_levels(int64_t m, int64_t n, T* A, int64_t lda, int rows, char* base, std::vector<Level<T>>* out) {
    size_t off = 0;
    std::vector<Level<T>> lv;
    lv.push_back({A, lda, m, ceil_div(m, rows)});
    while (lv.back().ntiles > 1) {
        const int64_t h = lv.back().ntiles * n;
        const int64_t ld = round_up(h, 32);
        T* M = base ? reinterpret_cast<T*>(base + off) : nullptr;
        off += (size_t)round_up((int64_t)(ld * n * (int64_t)sizeof(T)), (int64_t)kAlign);
        lv.push_back({M, ld, h, ceil_div(h, rows)});
    }
    if (out) *out = lv;
    return off;
}

}  // namespace

// Workspace of the plain tree: a status word (256 bytes; non-zero after a
// factor kernel's bounded wait gave up, read by tsqr_workspace_check), then
// the level matrices.
template <typename T>
size_t tsqr_plain_workspace(int64_t m, int64_t n) {
    KernelSet<T> ks = pick((T*)nullptr, (int)n);
    if (!ks.factor) return 0;
    return kAlign + plan_levels<T>(m, n, nullptr, m, ks.rows, nullptr, nullptr);
}

template <typename T>
tsqr_status tsqr_plain(int64_t m, int64_t n, T* A, int64_t lda, T* R, int64_t ldr, void* work, size_t work_bytes,
                       cudaStream_t s, int phases, int* status) {
    KernelSet<T> ks = pick((T*)nullptr, (int)n);
    if (!ks.factor) return TSQR_ERR_UNSUPPORTED;
    std::vector<Level<T>> lv;
    char* wb = reinterpret_cast<char*>(work);
    size_t need = plan_levels<T>(m, n, A, lda, ks.rows, wb ? wb + kAlign : nullptr, &lv);
    if (need > 0 && (work == nullptr || work_bytes < kAlign + need)) return TSQR_ERR_WORKSPACE;
    // a single-tile problem may run without a workspace, and then without a
    // status word
    int* err = status;
    if (!err && work != nullptr && work_bytes >= kAlign) err = reinterpret_cast<int*>(work);
    const int L = (int)lv.size();
    // up-sweep
    for (int l = 0; l < L && (phases & kPhaseUp); ++l) {
        FactorParams<T> fp;
        fp.M = lv[l].M;
        fp.ld = lv[l].ld;
        fp.h = lv[l].h;
        fp.n = (int)n;
        fp.ntiles = lv[l].ntiles;
        fp.stack = l > 0;
        fp.err = err;
        fp.clear = l == 0 && !status ? err : nullptr;
        fp.tries = wait_tries().load(std::memory_order_relaxed);
        if (l == L - 1) {
            fp.Rout = R;
            fp.ldr = ldr;
        } else {
            fp.Rout = lv[l + 1].M;
            fp.ldr = lv[l + 1].ld;
        }
        ks.factor(fp, (int)std::min<int64_t>(lv[l].ntiles, 1 << 30), s);
        log_launch(kTagFactor + l, s);
    }
    // down-sweep
    for (int l = L - 1; l >= 0 && (phases & kPhaseDown); --l) {
        ApplyParams<T> ap;
        ap.M = lv[l].M;
        ap.ld = lv[l].ld;
        ap.h = lv[l].h;
        ap.n = (int)n;
        ap.ntiles = lv[l].ntiles;
        ap.stack = l > 0;
        ap.P = (l == L - 1) ? nullptr : lv[l + 1].M;
        ap.ldp = (l == L - 1) ? 0 : lv[l + 1].ld;
        constexpr int ve = 16 / sizeof(T);
        ap.vec = (lv[l].ld % ve == 0 && (reinterpret_cast<uintptr_t>(lv[l].M) % 16) == 0) ? 1 : 0;
        ks.apply(ap, (int)std::min<int64_t>(lv[l].ntiles, 1 << 30), s);
        log_launch(kTagApply + l, s);
    }
    return cudaGetLastError() == cudaSuccess ? TSQR_OK : TSQR_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// Precision form (FP32 entry points): the tile factorisation stays FP32 on
// CUDA cores; the Q assembly of a level runs on tcgen05 in TF32x3
// (tc_apply.cu) or in FP32, as precision_level_fp32 says.  With
// tsqr_opts.fp64_root the last level is converted to double and factored by
// the FP64 tree.
// Workspace: [status word (256 B) | level matrices | FP64 root copy | FP64
// root-tree workspace].
// ---------------------------------------------------------------------------
namespace {

template <typename A, typename B>
__global__ void convert_matrix(int64_t h, int n, const A* __restrict__ src, int64_t lds, B* __restrict__ dst,
                               int64_t ldd) {
    const int64_t total = h * n;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e % h, c = e / h;
        dst[r + c * ldd] = (B)src[r + c * lds];
    }
}

template <typename A, typename B>
void convert(int64_t h, int n, const A* src, int64_t lds, B* dst, int64_t ldd, cudaStream_t s) {
    const int64_t total = h * n;
    const int blocks = (int)std::min<int64_t>(ceil_div(total, 256), 1024);
    convert_matrix<A, B><<<blocks, 256, 0, s>>>(h, n, src, lds, dst, ldd);
}

struct PrecCfg {
    int nmax = 0, rows = 0;
    KernelSet<float> ks;
};

// The tile factorisation is the plain FP32 kernel; with norm64
// (tsqr_opts.fp64_scalars) its variant whose per-column norm, beta and tau
// are computed in FP64.
PrecCfg pick_precision(int n, bool norm64 = false) {
    PrecCfg c;
    if (n <= 16) {
        c.nmax = 16;
        c.ks = norm64 ? make_set<SplitCfg<float, 16, 4, 16, 4, true>, float>()
                      : make_set<SplitCfg<float, 16, 4, 16, 4>, float>();
    } else if (n <= 32) {
        c.nmax = 32;
        c.ks = norm64 ? make_set<SplitCfg<float, 32, 4, 16, 2, true>, float>()
                      : make_set<SplitCfg<float, 32, 4, 16, 2>, float>();
    } else if (n <= 64) {
        c.nmax = 64;
        c.ks = norm64 ? make_set<SplitCfg<float, 64, 8, 16, 1, true>, float>()
                      : make_set<WideCfg, float>();
    }
    c.rows = c.ks.rows;
    return c;
}

struct PrecLayout {
    size_t status = 0, levels = 0, root = 0, rootws = 0, total = 0;
};

// Root combine in FP64 (tsqr_opts.fp64_root, n <= 32): the root level
// converted to double, factored by the FP64 tree, converted back.
PrecLayout prec_layout(int64_t m, int64_t n, const PrecCfg& c, bool root64_opt = false) {
    PrecLayout L;
    L.status = 0;
    L.levels = kAlign;
    std::vector<Level<float>> lv;
    const size_t lev = plan_levels<float>(m, n, nullptr, m, c.rows, nullptr, &lv);
    L.root = L.levels + lev;
    const int64_t hroot = lv.back().h;
    const bool root64 = root64_opt && n <= 32;
    const size_t rootbytes = root64 ? (size_t)round_up(hroot * n * 8 + n * n * 8, (int64_t)kAlign) : 0;
    L.rootws = L.root + rootbytes;
    L.total = L.rootws + (root64 ? round_up((int64_t)tsqr_plain_workspace<double>(hroot, n), (int64_t)kAlign) : 0);
    return L;
}

}  // namespace

bool tc_apply_level(const ApplyParams<float>& p, int nmax, int rows, int* err, cudaStream_t s);

// Whether a level of the precision form takes the FP32 Q assembly: its CTA has
// no TMEM to allocate, no operands to split and no padded columns to multiply,
// and its error is the smaller one.  Whole calls, us with tcgen05 on every level
// over us with FP32 on every level, by rows and base and leading dimension on
// (vec) or off 16 bytes:
//   columns below the tile's width: FP32.  1.05 .. 1.48 with vec at 4 to 56
//     columns and 512 to 2,000,000 rows.  Without vec 1.00 .. 1.39, but up to 32
//     columns the level alone is the slower one where it is large and nearly as
//     wide as its tile (tcgen05 there over FP32 there 1.03 at 256 tiles of 31
//     columns, 1.00 at 391, 0.96 at 512 and 3907; 20 columns 1.05 .. 1.03, 12 and
//     24 1.03 .. 0.99): tcgen05 above 384 tiles from two thirds of the width on.
//   16 and 32 columns fill their tiles: FP32 on levels of up to 128 tiles (16
//     columns 1.05 .. 1.13 with vec, 1.01 .. 1.07 without; 32 columns 1.04 ..
//     1.09, 1.01 .. 1.04).  Above, 16 columns with vec still 1.01 .. 1.06, but
//     without 1.03 falling to 0.95 at 1,000,000 rows; 32 columns 1.05 .. 0.995
//     and 1.03 .. 0.94, equal near 300 and 150 tiles: tcgen05.
//   64 columns: FP32 above 128 tiles, for its error (200,000 x 64 backward 3.6e-7
//     against 4.5e-7; 0.99 .. 1.015 with vec, 0.96 .. 0.98 without), tcgen05 on the
//     smaller levels (0.986 .. 0.998, 0.95 .. 0.98).
static bool precision_level_fp32(int n, int nmax, int64_t ntiles, int vec) {
    if (n < nmax) return vec || nmax == 64 || ntiles <= 384 || 3 * n < 2 * nmax;
    if (n == 64) return ntiles > 128;
    return ntiles <= 128 || (n == 16 && vec);
}

size_t tsqr_precision_workspace(int64_t m, int64_t n, PrecFlags f) {
    PrecCfg c = pick_precision((int)n, f.norm64);
    if (!c.ks.factor) return 0;
    return prec_layout(m, n, c, f.root64).total;
}

tsqr_status tsqr_precision(int64_t m, int64_t n, float* A, int64_t lda, float* R, int64_t ldr, void* work,
                           size_t work_bytes, cudaStream_t s, PrecFlags f) {
    PrecCfg c = pick_precision((int)n, f.norm64);
    if (!c.ks.factor) return TSQR_ERR_UNSUPPORTED;
    if (f.root64 && n > 32) return TSQR_ERR_UNSUPPORTED;
    const PrecLayout PL = prec_layout(m, n, c, f.root64);
    if (work == nullptr || work_bytes < PL.total) return TSQR_ERR_WORKSPACE;
    char* base = reinterpret_cast<char*>(work);
    int* err = f.status ? f.status : reinterpret_cast<int*>(base + PL.status);
    std::vector<Level<float>> lv;
    plan_levels<float>(m, n, A, lda, c.rows, base + PL.levels, &lv);
    const int L = (int)lv.size();
    const bool root64 = f.root64;
    const int top = root64 ? L - 1 : L;  // levels factored in FP32 below the root
    if (!f.status && top == 0 && cudaMemsetAsync(err, 0, sizeof(int), s) != cudaSuccess) return TSQR_ERR_CUDA;
    for (int l = 0; l < top; ++l) {
        FactorParams<float> fp;
        fp.M = lv[l].M;
        fp.ld = lv[l].ld;
        fp.h = lv[l].h;
        fp.n = (int)n;
        fp.ntiles = lv[l].ntiles;
        fp.stack = l > 0;
        fp.err = err;
        fp.clear = l == 0 && !f.status ? err : nullptr;
        fp.tries = wait_tries().load(std::memory_order_relaxed);
        fp.Rout = (l == L - 1) ? R : lv[l + 1].M;
        fp.ldr = (l == L - 1) ? ldr : lv[l + 1].ld;
        c.ks.factor(fp, (int)std::min<int64_t>(lv[l].ntiles, 1 << 30), s);
        log_launch(kTagFactor + l, s);
    }
    if (root64) {
        // FP64 root combine: the last level (at most one tile of stacked R
        // factors, or A itself when m fits one tile) factored in double.
        const Level<float>& rt = lv[L - 1];
        double* Qd = reinterpret_cast<double*>(base + PL.root);
        double* Rd = Qd + rt.h * n;
        convert<float, double>(rt.h, (int)n, rt.M, rt.ld, Qd, rt.h, s);
        log_launch(kTagTc + 900, s);
        tsqr_status st = tsqr_plain<double>(rt.h, n, Qd, rt.h, Rd, n, base + PL.rootws, PL.total - PL.rootws, s);
        if (st != TSQR_OK) return st;
        convert<double, float>(rt.h, (int)n, Qd, rt.h, rt.M, rt.ld, s);
        convert<double, float>(n, (int)n, Rd, n, R, ldr, s);
        log_launch(kTagTc + 901, s);
    }
    for (int l = (root64 ? L - 2 : L - 1); l >= 0; --l) {
        ApplyParams<float> ap;
        ap.M = lv[l].M;
        ap.ld = lv[l].ld;
        ap.h = lv[l].h;
        ap.n = (int)n;
        ap.ntiles = lv[l].ntiles;
        ap.stack = l > 0;
        ap.P = (l == L - 1) ? nullptr : lv[l + 1].M;
        ap.ldp = (l == L - 1) ? 0 : lv[l + 1].ld;
        ap.vec = (lv[l].ld % 4 == 0 && (reinterpret_cast<uintptr_t>(lv[l].M) % 16) == 0) ? 1 : 0;
        if (precision_level_fp32((int)n, c.nmax, lv[l].ntiles, ap.vec)) {
            c.ks.apply(ap, (int)lv[l].ntiles, s);
        } else if (!tc_apply_level(ap, c.nmax, c.rows, err, s)) {
            return TSQR_ERR_UNSUPPORTED;
        }
        log_launch(kTagTc + l, s);
    }
    return cudaGetLastError() == cudaSuccess ? TSQR_OK : TSQR_ERR_CUDA;
}

template size_t tsqr_plain_workspace<float>(int64_t, int64_t);
template size_t tsqr_plain_workspace<double>(int64_t, int64_t);
template <typename T>
tsqr_status tsqr_plain_tree(int64_t m, int64_t n, const T* A, int64_t lda, const void* work, size_t work_bytes,
                            std::vector<TreeLevel<T>>* out) {
    KernelSet<T> ks = pick((T*)nullptr, (int)n);
    if (!ks.factor) return TSQR_ERR_UNSUPPORTED;
    std::vector<Level<T>> lv;
    char* wb = const_cast<char*>(reinterpret_cast<const char*>(work));
    size_t need = plan_levels<T>(m, n, const_cast<T*>(A), lda, ks.rows, wb ? wb + kAlign : nullptr, &lv);
    if (need > 0 && (work == nullptr || work_bytes < kAlign + need)) return TSQR_ERR_WORKSPACE;
    out->clear();
    for (const Level<T>& v : lv) out->push_back({v.M, v.ld, v.h, v.ntiles, ks.rows});
    return TSQR_OK;
}
template tsqr_status tsqr_plain_tree<float>(int64_t, int64_t, const float*, int64_t, const void*, size_t,
                                            std::vector<TreeLevel<float>>*);
template tsqr_status tsqr_plain_tree<double>(int64_t, int64_t, const double*, int64_t, const void*, size_t,
                                             std::vector<TreeLevel<double>>*);
template tsqr_status tsqr_plain<float>(int64_t, int64_t, float*, int64_t, float*, int64_t, void*, size_t,
                                       cudaStream_t, int, int*);
template tsqr_status tsqr_plain<double>(int64_t, int64_t, double*, int64_t, double*, int64_t, void*, size_t,
                                        cudaStream_t, int, int*);

// ---------------------------------------------------------------------------
// TSQR of a matrix in host memory (tsqr_s_host / tsqr_d_host).  The device
// holds a copy of A (ld rounded up to 32 rows), the n x n R and the tree.
// Level 0 is cut into chunks of whole tiles.  A library copy stream moves
// chunk c to the device while the caller's stream factors chunk c-1; after
// the upper levels, the caller's stream assembles Q chunk by chunk while the
// copy stream returns the finished chunks, so both host transfers overlap
// the level-0 kernels instead of adding to them.  The copy stream and its
// events belong to the calling host thread (one set per device), so calls
// from different threads share nothing; a problem of one chunk copies on
// the caller's stream alone.
// ---------------------------------------------------------------------------
namespace {

constexpr int kHostChunks = 8;
constexpr int64_t kHostChunkBytes = 16 << 20;

// Copy stream and events of one host thread on one device.
struct HostPipe {
    int dev = -1;
    cudaStream_t cs = nullptr;
    cudaEvent_t ev[2 * kHostChunks + 2] = {};
};

HostPipe* host_pipe() {
    thread_local HostPipe pipes[8];
    thread_local int used = 0;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    for (int i = 0; i < used; ++i)
        if (pipes[i].dev == dev) return &pipes[i];
    if (used == 8) return nullptr;
    HostPipe& p = pipes[used];
    if (cudaStreamCreateWithFlags(&p.cs, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    for (auto& e : p.ev)
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return nullptr;
    p.dev = dev;
    ++used;
    return &p;
}

template <typename T>
struct HostLayout {
    int64_t ldd = 0;
    size_t a = 0, r = 0, tree = 0, total = 0;
};

// The tree comes first, so the precision form's status word sits at the
// start of the workspace as for the device entry points.
template <typename T>
HostLayout<T> host_layout(int64_t m, int64_t n, bool prec) {
    HostLayout<T> L;
    L.ldd = round_up(m, 32);
    size_t tw = 0;
    if constexpr (sizeof(T) == 4) {
        if (prec) {
            PrecCfg c = pick_precision((int)n);
            tw = c.ks.factor ? prec_layout(m, n, c).total : 0;
        }
    }
    if (!prec) tw = tsqr_plain_workspace<T>(m, n);
    L.tree = 0;
    L.a = (size_t)round_up((int64_t)tw, (int64_t)kAlign);
    L.r = L.a + (size_t)round_up(L.ldd * n * (int64_t)sizeof(T), (int64_t)kAlign);
    const size_t end = L.r + (size_t)round_up(n * n * (int64_t)sizeof(T), (int64_t)kAlign);
    L.total = tw ? end : 0;
    return L;
}

}  // namespace

template <typename T>
size_t tsqr_host_workspace(int64_t m, int64_t n, bool prec) {
    return host_layout<T>(m, n, prec).total;
}

template <typename T>
tsqr_status tsqr_host(int64_t m, int64_t n, const T* hA, int64_t lda, T* hQ, int64_t ldq, T* hR, int64_t ldr,
                      void* work, size_t work_bytes, bool prec, cudaStream_t s) {
    const PdlOff no_pdl;  // the kernels below wait on the copy stream's events
    const HostLayout<T> HL = host_layout<T>(m, n, prec);
    if (HL.total == 0) return TSQR_ERR_UNSUPPORTED;
    if (work == nullptr || work_bytes < HL.total) return TSQR_ERR_WORKSPACE;
    char* base = reinterpret_cast<char*>(work);
    T* dA = reinterpret_cast<T*>(base + HL.a);
    T* dR = reinterpret_cast<T*>(base + HL.r);
    char* tw = base + HL.tree;

    // the tree of the chosen form
    KernelSet<T> ks;
    int nmax = 0;
    bool tc = false;
    int* err = nullptr;
    char* lvbase = tw;
    if constexpr (sizeof(T) == 4) {
        if (prec) {
            PrecCfg c = pick_precision((int)n);
            const PrecLayout PL = prec_layout(m, n, c);
            ks = c.ks;
            nmax = c.nmax;
            tc = true;
            err = reinterpret_cast<int*>(tw + PL.status);
            lvbase = tw + PL.levels;
        }
    }
    if (!prec) {
        ks = pick((T*)nullptr, (int)n);
        err = reinterpret_cast<int*>(tw);  // the plain tree's status word
        lvbase = tw + kAlign;
    }
    if (!ks.factor) return TSQR_ERR_UNSUPPORTED;
    std::vector<Level<T>> lv;
    plan_levels<T>(m, n, dA, HL.ldd, ks.rows, lvbase, &lv);
    const int L = (int)lv.size();
    const int64_t rows = ks.rows;

    auto factor = [&](int l, int64_t t0, int64_t cnt) {
        FactorParams<T> fp;
        fp.M = lv[l].M + t0 * rows;
        fp.ld = lv[l].ld;
        fp.h = std::min<int64_t>(cnt * rows, lv[l].h - t0 * rows);
        fp.n = (int)n;
        fp.ntiles = cnt;
        fp.stack = l > 0;
        fp.err = err;
        fp.tries = wait_tries().load(std::memory_order_relaxed);
        fp.Rout = (l == L - 1) ? dR : lv[l + 1].M + t0 * n;
        fp.ldr = (l == L - 1) ? n : lv[l + 1].ld;
        ks.factor(fp, (int)std::min<int64_t>(cnt, 1 << 30), s);
        log_launch(kTagFactor + l, s);
    };
    auto apply = [&](int l, int64_t t0, int64_t cnt) -> bool {
        ApplyParams<T> ap;
        ap.M = lv[l].M + t0 * rows;
        ap.ld = lv[l].ld;
        ap.h = std::min<int64_t>(cnt * rows, lv[l].h - t0 * rows);
        ap.n = (int)n;
        ap.ntiles = cnt;
        ap.stack = l > 0;
        ap.P = (l == L - 1) ? nullptr : lv[l + 1].M + t0 * n;
        ap.ldp = (l == L - 1) ? 0 : lv[l + 1].ld;
        constexpr int ve = 16 / sizeof(T);
        ap.vec = (ap.ld % ve == 0 && (reinterpret_cast<uintptr_t>(ap.M) % 16) == 0) ? 1 : 0;
        if constexpr (sizeof(T) == 4) {
            // by the whole level, as for a matrix in device memory
            if (tc && !precision_level_fp32((int)n, nmax, lv[l].ntiles, ap.vec)) {
                if (!tc_apply_level(ap, nmax, (int)rows, err, s)) return false;
                log_launch(kTagTc + l, s);
                return true;
            }
        }
        ks.apply(ap, (int)std::min<int64_t>(cnt, 1 << 30), s);
        log_launch(kTagApply + l, s);
        return true;
    };

    const int64_t nt0 = lv[0].ntiles;
    // chunks of at least kHostChunkBytes: smaller copies gain less from the
    // overlap than the extra launches and stream operations cost
    const int64_t by_size = std::max<int64_t>(1, (m * n * (int64_t)sizeof(T)) / kHostChunkBytes);
    const int nc = (int)std::min<int64_t>(std::min<int64_t>(kHostChunks, nt0), by_size);
    const int64_t per = ceil_div(nt0, nc);
    const size_t es = sizeof(T);
    tsqr_status st = TSQR_OK;
    // One chunk leaves nothing to overlap: copies on the caller's stream.
    // Otherwise the copy stream and events of this host thread (made once per
    // thread and device, reused by its later calls: a host thread issues its
    // calls one after another, and a wait captures an event's state when it
    // is enqueued, so re-recording an event cannot disturb an earlier call).
    cudaStream_t cs = s;
    cudaEvent_t* ev = nullptr;
    if (nc > 1) {
        HostPipe* hp = host_pipe();
        if (!hp) return TSQR_ERR_CUDA;
        cs = hp->cs;
        ev = hp->ev;
    }
    if (nc == 1) {
        const int64_t hr = m;
        if (cudaMemcpy2DAsync(dA, HL.ldd * es, hA, lda * es, hr * es, n, cudaMemcpyHostToDevice, s) != cudaSuccess)
            return TSQR_ERR_CUDA;
        if (err) cudaMemsetAsync(err, 0, sizeof(int), s);
        for (int l = 0; l < L; ++l) factor(l, 0, lv[l].ntiles);
        for (int l = L - 1; l >= 0; --l)
            if (!apply(l, 0, lv[l].ntiles)) return TSQR_ERR_UNSUPPORTED;
        if (cudaMemcpy2DAsync(hR, ldr * es, dR, n * es, n * es, n, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaMemcpy2DAsync(hQ, ldq * es, dA, HL.ldd * es, hr * es, n, cudaMemcpyDeviceToHost, s) != cudaSuccess)
            return TSQR_ERR_CUDA;
        return cudaGetLastError() == cudaSuccess ? TSQR_OK : TSQR_ERR_CUDA;
    }
    {
        // the copy stream starts after the caller's earlier work
        cudaEventRecord(ev[2 * kHostChunks], s);
        cudaStreamWaitEvent(cs, ev[2 * kHostChunks], 0);
        if (err) cudaMemsetAsync(err, 0, sizeof(int), s);
        // up: chunk c copied in while chunk c-1 is factored
        for (int c = 0; c < nc; ++c) {
            const int64_t t0 = c * per, cnt = std::min<int64_t>(per, nt0 - t0);
            if (cnt <= 0) break;
            const int64_t r0 = t0 * rows, hr = std::min<int64_t>(cnt * rows, m - r0);
            if (cudaMemcpy2DAsync(dA + r0, HL.ldd * es, hA + r0, lda * es, hr * es, n, cudaMemcpyHostToDevice, cs) !=
                cudaSuccess)
                st = TSQR_ERR_CUDA;
            cudaEventRecord(ev[c], cs);
            cudaStreamWaitEvent(s, ev[c], 0);
            factor(0, t0, cnt);
        }
        for (int l = 1; l < L; ++l) factor(l, 0, lv[l].ntiles);
        for (int l = L - 1; l >= 1 && st == TSQR_OK; --l)
            if (!apply(l, 0, lv[l].ntiles)) st = TSQR_ERR_UNSUPPORTED;
        if (cudaMemcpy2DAsync(hR, ldr * es, dR, n * es, n * es, n, cudaMemcpyDeviceToHost, s) != cudaSuccess)
            st = TSQR_ERR_CUDA;
        // down: chunk c of Q returned while chunk c+1 is assembled
        for (int c = 0; c < nc && st == TSQR_OK; ++c) {
            const int64_t t0 = c * per, cnt = std::min<int64_t>(per, nt0 - t0);
            if (cnt <= 0) break;
            const int64_t r0 = t0 * rows, hr = std::min<int64_t>(cnt * rows, m - r0);
            if (!apply(0, t0, cnt)) {
                st = TSQR_ERR_UNSUPPORTED;
                break;
            }
            cudaEventRecord(ev[kHostChunks + c], s);
            cudaStreamWaitEvent(cs, ev[kHostChunks + c], 0);
            if (cudaMemcpy2DAsync(hQ + r0, ldq * es, dA + r0, HL.ldd * es, hr * es, n, cudaMemcpyDeviceToHost, cs) !=
                cudaSuccess)
                st = TSQR_ERR_CUDA;
        }
        // the caller's stream completes after the last copy
        cudaEventRecord(ev[2 * kHostChunks + 1], cs);
        cudaStreamWaitEvent(s, ev[2 * kHostChunks + 1], 0);
    }
    if (st != TSQR_OK) return st;
    return cudaGetLastError() == cudaSuccess ? TSQR_OK : TSQR_ERR_CUDA;
}

template size_t tsqr_host_workspace<float>(int64_t, int64_t, bool);
template size_t tsqr_host_workspace<double>(int64_t, int64_t, bool);
template tsqr_status tsqr_host<float>(int64_t, int64_t, const float*, int64_t, float*, int64_t, float*, int64_t,
                                      void*, size_t, bool, cudaStream_t);
template tsqr_status tsqr_host<double>(int64_t, int64_t, const double*, int64_t, double*, int64_t, double*,
                                       int64_t, void*, size_t, bool, cudaStream_t);

// ---------------------------------------------------------------------------
// R <- R2 R (both upper triangular), for the reorthogonalisation pass of
// tsqr_*_ex.  One CTA: both factors are read into shared memory first, so R
// may be overwritten; thread (i, j) forms sum_{k=i}^{j} R2(i,k) R(k,j).
// ---------------------------------------------------------------------------
namespace {

template <typename T, int NMAX>
__global__ void upper_product_kernel(int n, const T* __restrict__ R2, int64_t ld2, T* R, int64_t ldr) {
    __shared__ T a[NMAX][NMAX + 1], b[NMAX][NMAX + 1];
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e % n, j = e / n;
        a[i][j] = R2[i + j * ld2];
        b[i][j] = R[i + j * ldr];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e % n, j = e / n;
        T s = T(0);
        for (int k = i; k <= j; ++k) s += a[i][k] * b[k][j];
        R[i + j * ldr] = (i <= j) ? s : T(0);
    }
}

}  // namespace

template <typename T>
tsqr_status upper_product(int n, const T* R2, int64_t ld2, T* R, int64_t ldr, cudaStream_t s) {
    constexpr int NMAX = sizeof(T) == 4 ? 64 : 32;
    if (n < 1 || n > NMAX) return TSQR_ERR_UNSUPPORTED;
    upper_product_kernel<T, NMAX><<<1, 256, 0, s>>>(n, R2, ld2, R, ldr);
    log_launch(kTagTc + 902, s);
    return cudaGetLastError() == cudaSuccess ? TSQR_OK : TSQR_ERR_CUDA;
}
template tsqr_status upper_product<float>(int, const float*, int64_t, float*, int64_t, cudaStream_t);
template tsqr_status upper_product<double>(int, const double*, int64_t, double*, int64_t, cudaStream_t);

// ---------------------------------------------------------------------------
// Per-device workspace cache for the reference-signature entry points, whose
// d_work is sized for the reference's own layout (ldwork*n elements with
// ldwork = 2*NUM_SM*BLOCK_SIZE, test_tsqr.cu:42-45).
// ---------------------------------------------------------------------------
void* cached_workspace(size_t bytes, tsqr_status* st) {
    static std::mutex mu;
    static void* buf[64] = {nullptr};
    static size_t cap[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        *st = TSQR_ERR_NO_DEVICE;
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(mu);
    if (buf[dev]) {
        // a cudaDeviceReset since the allocation invalidates it: allocate again
        cudaPointerAttributes at;
        if (cudaPointerGetAttributes(&at, buf[dev]) != cudaSuccess || at.type != cudaMemoryTypeDevice) {
            (void)cudaGetLastError();
            buf[dev] = nullptr;
            cap[dev] = 0;
        }
    }
    if (cap[dev] < bytes) {
        if (buf[dev]) {
            cudaDeviceSynchronize();
            cudaFree(buf[dev]);
            buf[dev] = nullptr;
            cap[dev] = 0;
        }
        if (cudaMalloc(&buf[dev], bytes) != cudaSuccess) {
            buf[dev] = nullptr;
            *st = TSQR_ERR_CUDA;
            return nullptr;
        }
        cap[dev] = bytes;
    }
    *st = TSQR_OK;
    return buf[dev];
}

}  // namespace tsqr
