// tsqr_kernels.cuh -- CUDA-core (plain precision) TSQR tile kernels.
//
// A "level matrix" M (h x n, column-major, leading dimension ld) is cut into
// tiles of B = NT*RPT rows.  Level 0 is the caller's A; level l+1 stacks the
// n x n R factors of level l's tiles (h_{l+1} = tiles_l * n); the level with
// a single tile is the root.  This is the reduction tree of the reference's
// persistent tsqr_kernel (kernelQR.h:341-388) and of its two-level chunk
// scheme (TallShinnyQR.h:106-127), restated as one tree with a tile height
// chosen per (dtype, n) instead of the compile-time BLOCK_SIZE=128 and
// NUM_SM=108 (kernelQR.h:3-4).
//
// factor_tiles: Householder QR of each tile (the reference's qr_kernel,
//   kernelQR.h:69-220), LAPACK larfg form: H_j = I - tau_j v_j v_j^T with
//   v_j(j) = 1 and R_jj = beta_j = -sign(alpha) ||x||, the same diagonal sign
//   rule as kernelQR.h:139-142.  Instead of forming the tile's explicit Q in
//   shared memory (kernelQR.h:224-290) it leaves the compact-WY form in place:
//   the strict lower part of the tile holds V, the upper triangle of the
//   tile's top n x n block holds T (H_0...H_{n-1} = I - V T V^T).  The tile
//   lives in registers (RPT rows x NMAX columns per thread).  Each column
//   costs two block barriers: one after the norm partials, one after the
//   dot-product partials (the warp transpose-reduction of NMAX values, then a
//   redundant per-warp finalisation instead of a third barrier).  The same
//   reduction also yields column j of V^T V, from which T is formed once per
//   tile: row i of T depends only on row i (T(i,j) = -tau_j sum_k T(i,k)
//   S(k,j)), so thread i builds it alone.  R goes to the next level's rows
//   [t*n, t*n+n), or to the caller's R at the root.
//
// apply_tiles_f32 (and apply_f64_tiles in tile_f64.cuh): down-sweep
//   (kernelQR.h:397-492 and tsgemm_tsqr, TallShinnyQR.h:11-74): given the
//   parent's n x n block B_t (the root uses B = I), the tile's final Q is
//   (I - V T V^T) [B_t; 0] = [B_t; 0] - V W, W = T (V_top^T B_t).  W needs only
//   the tile's top block, so the bulk is a reduction-free (B x n)(n x n)
//   product, in chunks of rows that pass through shared memory, 4 rows x 4 or 8
//   columns per thread; Q overwrites the tile in place.
//
// Rows of the last tile past the matrix end are treated as zero rows: they
// never change, never enter a dot product and are never stored.
#pragma once
#include <type_traits>

#include <cuda.h>  // CUtensorMap (the type only; no driver calls here)

#include "common.cuh"
#include "tc.cuh"

namespace tsqr {

template <typename T>
struct FactorParams {
    T* M;           // level matrix (tiles are factored in place)
    int64_t ld;
    int64_t h;      // rows of the level matrix
    int n;
    int64_t ntiles;
    T* Rout;        // R of tile t goes to rows [t*n, t*n+n) of Rout
    int64_t ldr;
    int stack = 0;  // 1: the level is a stack of n x n upper triangles (any level above the first)
    int* err = nullptr;  // status word: set to 1 when a bounded wait gives up (null: none)
    int tries = tc::kMbarTries;  // polls of a bounded wait before it gives up
    int* clear = nullptr;        // status word to zero first (null: none); see clear_status
};

// A call's status word is zeroed in its first kernel: a fill in front of it
// costs a launch and 2 us.  The kernels with bounded waits may set it in any
// CTA, and the FP64-norm ones would spill: their launches keep the fill.
template <typename T>
__device__ __forceinline__ void clear_status(const FactorParams<T>& p) {
    if (p.clear && blockIdx.x == 0 && threadIdx.x == 0) *p.clear = 0;
}

template <typename T>
struct ApplyParams {
    T* M;
    int64_t ld;
    int64_t h;
    int n;
    int64_t ntiles;
    const T* P;     // parent level's final Q (rows t*n.. of tile t); null = identity
    int64_t ldp;
    int vec;        // 1: ld and the level base allow 16-byte copies
    int stack = 0;  // 1: any level above the first (FactorParams::stack)
};

// Column-major V^T V of a tile: Sc[j][k] = S(k, j) = v_k . v_j for k < j,
// rows padded to a multiple of 16 bytes so a column reads as vector loads.
template <typename T, int NMAX>
struct SCols {
    static constexpr int LD = NMAX + 16 / (int)sizeof(T);
    __align__(16) T c[NMAX][LD];
};

// Shared memory of one factor_tiles CTA.
template <int NMAX, int NT>
struct FactorSmem {
    static constexpr int NW = NT / 32;
    float s_part[NW];
    float s_alpha;
    float red[NW][NMAX];
    __align__(16) float wfin[NW][NMAX];
    SCols<float, NMAX> Sc;
    float Tsh[NMAX][NMAX + 1];
    float tau_sh[NMAX];
    float rdiag[NMAX];
    // per-warp transpose scratch of the dot-product reduction
    __align__(16) float xpose[NW][32 * xpose_stride<NMAX>()];
};

// Row i of the compact-WY factor T of a tile: T(i,i) = tau_i and
// T(i,j) = -tau_j sum_{k=i}^{j-1} T(i,k) S(k,j) for i < j < n, zero
// elsewhere.  Column j of S is read with 16-byte loads that do not depend on
// the FMA chain, so their latency is paid once per column instead of once per
// product, and the chain is split into two accumulators.  T(i,k) = 0 for
// k < i, so the sum runs over every k < j without a per-thread test.
template <typename T, int NMAX>
__device__ __forceinline__ void t_factor_row(const SCols<T, NMAX>& S, const T* tau, int i, int n, T (&trow)[NMAX]) {
    constexpr int VW = 16 / (int)sizeof(T);  // elements per 16-byte load
    static_assert(NMAX % VW == 0, "T build reads whole 16-byte groups");
#pragma unroll
    for (int j = 0; j < NMAX; ++j) {
        T a0 = T(0), a1 = T(0);
#pragma unroll
        for (int k0 = 0; k0 < j; k0 += VW) {
            if constexpr (VW == 4) {
                const float4 q = *reinterpret_cast<const float4*>(&S.c[j][k0]);
                a0 += trow[k0] * q.x;
                if (k0 + 1 < j) a1 += trow[k0 + 1] * q.y;
                if (k0 + 2 < j) a0 += trow[k0 + 2] * q.z;
                if (k0 + 3 < j) a1 += trow[k0 + 3] * q.w;
            } else {
                const double2 q = *reinterpret_cast<const double2*>(&S.c[j][k0]);
                a0 += trow[k0] * q.x;
                if (k0 + 1 < j) a1 += trow[k0 + 1] * q.y;
            }
        }
        const T tj = tau[j];
        trow[j] = (j == i) ? tj : ((j > i && j < n) ? -tj * (a0 + a1) : T(0));
    }
}

// Householder QR of one tile: ht (<= NT*RPT) rows of n columns at `tile`
// (leading dimension ld), factored in place (V below the diagonal, T in the
// top block's upper triangle); its n x n R goes to Rt (leading dimension
// ldr).  Called by every thread of the CTA.
template <int NMAX, int NT, int RPT>
__device__ __forceinline__ void factor_tile(FactorSmem<NMAX, NT>& S, float* tile, int64_t ld, int ht, int n, float* Rt,
                                            int64_t ldr) {
    constexpr int NW = NT / 32;
    constexpr int U = 4;  // columns per unrolled group
    static_assert(NT >= NMAX && NT % 32 == 0 && NMAX % U == 0, "bad tile configuration");
    auto& s_part = S.s_part;
    auto& s_alpha = S.s_alpha;
    auto& red = S.red;
    auto& wfin = S.wfin;
    auto& Sc = S.Sc.c;
    auto& Tsh = S.Tsh;
    auto& tau_sh = S.tau_sh;
    auto& rdiag = S.rdiag;
    auto& xpose = S.xpose;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = (n + U - 1) / U;
    const int shift = (U * G) % NMAX;  // register position c ends up holding column (c + shift) % NMAX
    {
        // y[i][c]: row tid + NT*i.  The column loop runs in groups of U
        // columns; after each group the register row rotates left by U, so at
        // group g position c < n - U*g holds column U*g + c (positions 0..U-1
        // are the group's columns) and position NMAX - U*g + k holds the
        // finished reflector v_k.  All register indices stay compile-time
        // while the code holds U column steps instead of NMAX.
        float y[RPT][NMAX];
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = tid + NT * i;
#pragma unroll
            for (int c = 0; c < NMAX; ++c)
                y[i][c] = (r < ht && c < n) ? tile[r + c * ld] : 0.f;
        }

#pragma unroll 1
        for (int g = 0; g < G; ++g) {
            const int base = U * g;
            const int live = n - base;      // positions [0, live): columns base .. n-1
            const int past0 = NMAX - base;  // positions [past0, NMAX): v_0 .. v_{base-1}
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = base + u;
                if (j < n) {
                    // Row slots i >= 1 hold rows >= NT >= NMAX > j, so only
                    // slot 0 needs the row-versus-diagonal tests below.
                    // (a) sigma^2 = ||x(j+1:, j)||^2 and alpha = x(j, j)
                    float s = 0;
#pragma unroll
                    for (int i = 0; i < RPT; ++i) {
                        const int r = tid + NT * i;
                        if (i > 0 || r > j) s += y[i][u] * y[i][u];
                        if (i == 0 && r == j) s_alpha = y[i][u];
                    }
                    s = warp_sum(s);
                    if (lane == 0) s_part[warp] = s;
                    __syncthreads();
                    float sigma2 = 0;
#pragma unroll
                    for (int w = 0; w < NW; ++w) sigma2 += s_part[w];
                    const float alpha = s_alpha;
                    float beta, tau, scale;
                    if (sigma2 == 0.f) {
                        tau = 0;
                        beta = alpha;
                        scale = 0;
                    } else {
                        const float nrm = sqrt(alpha * alpha + sigma2);
                        beta = (alpha >= 0.f) ? -nrm : nrm;
                        // reciprocal-multiply (round-to-nearest reciprocal)
                        // keeps the slow division path off the column chain
                        tau = (beta - alpha) * recip(beta);
                        scale = recip(alpha - beta);
                    }
                    // (b) v_j below the diagonal (v_j(j) = 1 implicitly), then
                    // v_j . y[c] for every other position: trailing columns
                    // (update) and finished reflectors (column j of V^T V)
#pragma unroll
                    for (int i = 0; i < RPT; ++i) {
                        const int r = tid + NT * i;
                        if (i > 0 || r > j) y[i][u] *= scale;
                    }
                    // v of slot 0: 0 above the diagonal, 1 on it
                    const float v0 = (tid > j) ? y[0][u] : ((tid == j) ? 1.f : 0.f);
                    float pc[NMAX];
#pragma unroll
                    for (int c = 0; c < NMAX; ++c) pc[c] = (c != u) ? v0 * y[0][c] : 0.f;
#pragma unroll
                    for (int i = 1; i < RPT; ++i) {
                        const float v = y[i][u];
#pragma unroll
                        for (int c = 0; c < NMAX; ++c)
                            if (c != u) pc[c] += v * y[i][c];
                    }
                    warp_reduce_to_smem_x<NMAX>(pc, red[warp], xpose[warp], lane);
                    __syncthreads();
                    // (c) every warp sums the NW partials itself; positions
                    // that are not trailing columns get a zero coefficient, so
                    // the update below needs no per-column test
                    {
                        constexpr int K = NMAX >= 32 ? NMAX / 32 : 1;
#pragma unroll
                        for (int kk = 0; kk < K; ++kk) {
                            const int idx = (NMAX >= 32) ? lane * K + kk : lane;
                            if (idx < NMAX) {
                                float a = 0;
#pragma unroll
                                for (int w = 0; w < NW; ++w) a += red[w][idx];
                                wfin[warp][idx] = (idx > u && idx < live) ? a : 0.f;
                                if (warp == 0) {
                                    const int k = (idx >= past0) ? idx - past0 : ((idx < u) ? base + idx : -1);
                                    if (k >= 0) Sc[j][k] = a;
                                }
                            }
                        }
                        if (tid == 0) {
                            tau_sh[j] = tau;
                            rdiag[j] = beta;
                        }
                    }
                    __syncwarp();
                    // (d) trailing update x_c -= tau (v^T x_c) v (v = 0 above
                    // the diagonal, coefficient 0 off the trailing columns)
                    float wr[NMAX];
#pragma unroll
                    for (int c = 0; c < NMAX; ++c) wr[c] = wfin[warp][c];
#pragma unroll
                    for (int i = 0; i < RPT; ++i) {
                        const float tv = tau * ((i > 0) ? y[i][u] : v0);
#pragma unroll
                        for (int c = u + 1; c < NMAX; ++c) y[i][c] -= tv * wr[c];
                    }
                }
            }
            // rotate every register row left by U
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                float keep[U];
#pragma unroll
                for (int u = 0; u < U; ++u) keep[u] = y[i][u];
#pragma unroll
                for (int c = 0; c < NMAX - U; ++c) y[i][c] = y[i][c + U];
#pragma unroll
                for (int u = 0; u < U; ++u) y[i][NMAX - U + u] = keep[u];
            }
        }
        __syncthreads();  // V^T V, tau_sh, rdiag complete

        // T, one row per thread: T(i,i) = tau_i,
        // T(i,j) = -tau_j sum_{k=i}^{j-1} T(i,k) S(k,j) for j > i.
        if (tid < n) {
            const int i = tid;
            float trow[NMAX];
            t_factor_row<float, NMAX>(S.Sc, tau_sh, i, n, trow);
#pragma unroll
            for (int j = 0; j < NMAX; ++j) Tsh[i][j] = trow[j];
        }
        __syncthreads();

        // R of this tile: row r < n is held by thread r (i = 0).
        if (tid < n) {
            const int r = tid;
#pragma unroll
            for (int c = 0; c < NMAX; ++c) {
                const int k = (c + shift) % NMAX;
                if (k < n) {
                    float v = (k > r) ? y[0][c] : ((k == r) ? rdiag[r] : 0.f);
                    if (r >= ht) v = 0.f;
                    Rt[r + k * ldr] = v;
                }
            }
        }
        // V below the diagonal, T in the top block's upper triangle.
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = tid + NT * i;
            if (r < ht) {
#pragma unroll
                for (int c = 0; c < NMAX; ++c) {
                    const int k = (c + shift) % NMAX;
                    if (k < n) tile[r + k * ld] = (r > k) ? y[i][c] : Tsh[r][k];
                }
            }
        }
        __syncthreads();
    }
}

template <int NMAX, int NT, int RPT, int MINB>
__global__ void __launch_bounds__(NT, MINB) factor_tiles(FactorParams<float> p) {
    pdl_begin();
    clear_status(p);
    constexpr int B = NT * RPT;
    __shared__ FactorSmem<NMAX, NT> S;
    for (int64_t t = blockIdx.x; t < p.ntiles; t += gridDim.x) {
        const int64_t row0 = t * B;
        const int ht = (int)((p.h - row0) < B ? (p.h - row0) : B);
        factor_tile<NMAX, NT, RPT>(S, p.M + row0, p.ld, ht, p.n, p.Rout + t * p.n, p.ldr);
    }
}

// ---------------------------------------------------------------------------
// Column-split tiles (n <= NMAX <= 64, tiles of 32*RPT rows, FP32 or FP64).
// The W = NMAX/CW warps of a CTA share one tile: warp w holds columns
// [w*CW, w*CW + CW) of all 32*RPT rows (row lane + 32*i in y[i]), so a
// thread carries RPT*CW tile values instead of RPT*NMAX and more rows fit on
// an SM.  Column j is owned by warp j/CW.  At step j the owner forms v_j and
// tau_j from its column, publishes them to shared memory and passes one CTA
// barrier; then every warp applies H_j to its own columns (dot products, a
// per-warp transpose reduction, the rank-1 update) while the owner goes on to
// column j+1.  Warps whose columns are all finished only take the dot
// products that give column j of V^T V.  The critical path of a step is the
// owner's chain for one CW-column block instead of the whole tile.  v_j
// alternates between two buffers: the owner rewrites buffer b at step j+2,
// after every warp has passed the barrier of step j+1 and so has read step
// j's copy.
//
// Every warp executes the same number of barriers (one per step; a phase of
// nloc columns runs 4*ceil(nloc/4) steps, the padding steps act on zero
// columns with tau = 0).  Output format as factor_tile.

__device__ __forceinline__ float fmadd(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmadd(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float sqrt_t(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrt_t(double x) { return sqrt(x); }

// Reflector scalars on the owner's critical chain, FP32, branch-free: the
// hardware approximations refined by a Newton-Raphson step and finished with
// one residual correction each (Markstein's method for sqrt and reciprocal).  sqrt: r ~ 1/sqrt(x), r <- r (3 - x r^2) / 2,
// s = x r, s <- s + (r/2)(x - s^2) with the residual by FMA; reciprocal:
// r <- r (2 - x r), r <- r + r (1 - x r).  Both land within rounding of the
// correctly rounded results without the slow-path branches of the IEEE
// sequences.  Only used for x > 0 (the zero-column case selects other
// values).  FP64 keeps the exact operations.
__device__ __forceinline__ float refl_sqrt(float x) {
    float r = rsqrtf(x);
    r = r * fmaf(-0.5f * x * r, r, 1.5f);
    const float s = x * r;
    return fmaf(0.5f * r, fmaf(-s, s, x), s);
}
__device__ __forceinline__ double refl_sqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float refl_recip(float x) {
    float r = __fdividef(1.0f, x);
    r = r * fmaf(-x, r, 2.0f);
    return fmaf(r, fmaf(-x, r, 1.0f), r);
}
__device__ __forceinline__ double refl_recip(double x) { return 1.0 / x; }

// 16-byte vector of T.
template <typename T>
struct Vec16;
template <>
struct Vec16<float> {
    static constexpr int N = 4;
    __device__ __forceinline__ static void store(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
    __device__ __forceinline__ static void load(const float* p, float* v) {
        const float4 q = *reinterpret_cast<const float4*>(p);
        v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
    }
};
template <>
struct Vec16<double> {
    static constexpr int N = 2;
    __device__ __forceinline__ static void store(double* p, const double* v) { *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]); }
    __device__ __forceinline__ static void load(const double* p, double* v) {
        const double2 q = *reinterpret_cast<const double2*>(p);
        v[0] = q.x, v[1] = q.y;
    }
};

// Row stride (elements) of the per-warp transpose scratch.  FP32 with CW = 4
// needs no padding (lane l's 16-byte row is words 4l..4l+3, and the column
// reads of the 8 lanes per position hit 32 distinct banks); other shapes
// get 16 bytes of pad.
template <typename T, int CW>
__host__ __device__ constexpr int colsum_stride() {
    return (sizeof(T) == 4 && CW == 4) ? 4 : CW + 16 / (int)sizeof(T);
}

// Layout of the published reflector: lane-major in 16-byte chunks when RPT
// allows (KC = RPT / VN chunks per lane, a power of two up to 8), so a lane moves its
// RPT values with KC vector accesses; chunk k of lane l sits at chunk
// position k ^ ((l / (8 / KC)) & (KC - 1)) of the lane's row, which puts the
// 8 lanes of each 16-byte access phase on 8 distinct 4-bank groups.
// Otherwise, or when VEC is false, slot i of lane l is element l + 32 i
// (scalar accesses).
template <typename T, int RPT, bool VEC = true>
struct VbufLayout {
    static constexpr int VN = Vec16<T>::N;
    static constexpr int KC = RPT / VN;
    static constexpr bool kVec = VEC && (RPT % VN == 0) && KC >= 1 && KC <= 8 && (KC & (KC - 1)) == 0;
    __device__ __forceinline__ static int swz(int lane) { return kVec ? (lane / (8 / KC)) & (KC - 1) : 0; }
    template <typename F>
    __device__ __forceinline__ static void store(T* buf, int lane, int sw, F&& val) {
        if constexpr (kVec) {
#pragma unroll
            for (int k = 0; k < KC; ++k) {
                T t[VN];
#pragma unroll
                for (int e = 0; e < VN; ++e) t[e] = val(k * VN + e);
                Vec16<T>::store(buf + lane * RPT + VN * (k ^ sw), t);
            }
        } else {
#pragma unroll
            for (int i = 0; i < RPT; ++i) buf[lane + 32 * i] = val(i);
        }
    }
    __device__ __forceinline__ static void load(const T* buf, int lane, int sw, T (&v)[RPT]) {
        if constexpr (kVec) {
#pragma unroll
            for (int k = 0; k < KC; ++k) Vec16<T>::load(buf + lane * RPT + VN * (k ^ sw), &v[k * VN]);
        } else {
#pragma unroll
            for (int i = 0; i < RPT; ++i) v[i] = buf[lane + 32 * i];
        }
    }
};

template <typename T, int NMAX, int CW, int RPT>
struct SplitFactorSmem {
    static constexpr int W = NMAX / CW;
    __align__(16) T vbuf[2][32 * RPT];
    T taub[2];
    __align__(16) T xpose[W][32 * colsum_stride<T, CW>()];
    __align__(16) T coef[W][CW];
    SCols<T, NMAX> Sc;
    T tau[NMAX];
    T rdiag[NMAX];
};

// CTA barrier 1 over `count` threads; non-aligned form, since the owner and
// the other warps reach it from different code.
__device__ __forceinline__ void step_barrier(int count) {
    asm volatile("barrier.sync 1, %0;\n" ::"r"(count) : "memory");
}

// Sum CW per-lane partials over the warp through a shared-memory transpose:
// returns, in lane l, the full sum of position l % CW (32/CW lanes hold each
// sum, bitwise equal).
template <typename T, int CW>
__device__ __forceinline__ T warp_colsum(const T (&q)[CW], T* scratch, int lane) {
    constexpr int SP = colsum_stride<T, CW>();
    constexpr int VN = Vec16<T>::N;
    constexpr int LPP = 32 / CW;  // lanes per position
    constexpr int RPL = 32 / LPP;  // rows summed by one lane
    T* mine = scratch + lane * SP;
#pragma unroll
    for (int c = 0; c < CW; c += VN) Vec16<T>::store(mine + c, &q[c]);
    __syncwarp();
    const int p = lane % CW, h = lane / CW;
    T a[RPL];
#pragma unroll
    for (int r = 0; r < RPL; ++r) a[r] = scratch[(h + LPP * r) * SP + p];
#pragma unroll
    for (int w = RPL / 2; w >= 1; w >>= 1)
#pragma unroll
        for (int r = 0; r < w; ++r) a[r] += a[r + w];
    T s = a[0];
#pragma unroll
    for (int o = CW; o < 32; o <<= 1) s += __shfl_xor_sync(kFull, s, o);
    __syncwarp();  // scratch is rewritten by the next call
    return s;
}

// The column steps of a tile held in y (row lane + 32*i in slot i, columns
// warp*CW + c): on return y holds V below the diagonal and R above it, S the
// reflector scalars, R's diagonal and V^T V (complete after a barrier).
// Returns the rotation: position c holds the warp's column (c + shift) % CW.
template <typename T, int NMAX, int CW, int RPT, bool VECV, bool N64>
__device__ __forceinline__ int split_steps(SplitFactorSmem<T, NMAX, CW, RPT>& S, T (&y)[RPT][CW], int n) {
    using SC = typename std::conditional<N64, double, T>::type;  // type of the reflector scalars
    constexpr int W = NMAX / CW;
    constexpr int U = 4;
    constexpr int VN = Vec16<T>::N;
    // tau multiplies the CW coefficients (one lane each) instead of the RPT
    // row values where a multiplication costs more than the added latency
    constexpr bool kFold = sizeof(T) == 8;
    // the padding steps of a phase's last group are skipped where a step costs
    // more than the test (262,144 x 5 FP64 in the 8-column tile: 5 steps, not 8)
    constexpr bool kTrim = sizeof(T) == 8 && NMAX <= 16;
    static_assert(NMAX <= 64 && CW % U == 0 && CW % VN == 0 && NMAX % CW == 0 && W >= 2 && 32 * RPT >= NMAX &&
                      W >= NMAX / 32,
                  "bad split configuration");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col0 = warp * CW;
    const int mycols = max(0, min(CW, n - col0));
    T* scratch = S.xpose[warp];
    using VL = VbufLayout<T, RPT, VECV>;
    const int vsw = VL::swz(lane);
    // Row lane + 32*i lies strictly below diagonal element j (compile-time
    // true for every slot i >= 1 when NMAX <= 32).
    auto below = [&](int i, int j) { return (NMAX <= 32 && i > 0) || (lane + 32 * i > j); };
    // Reflector scalars: the branch-free forms shorten the owner's chain for
    // NMAX <= 32; the 64-column tile, already at its register limit, runs
    // faster with the plain operations (level-0 factor at 4,194,304 x 64:
    // 3.25 against 3.78 ms).
    auto rsq = [](SC x) {
        if constexpr (NMAX <= 32) return refl_sqrt(x);
        else return sqrt_t(x);
    };
    auto rcp = [](SC x) {
        if constexpr (NMAX <= 32) return refl_recip(x);
        else return recip(x);
    };
    // x(j, c) of position c, held by lane j % 32 in slot j / 32 (j < 64)
    auto diag_slot = [&](const T(&yy)[RPT][CW], int c, int j) {
        return (NMAX > 32 && j >= 32) ? yy[RPT > 1 ? 1 : 0][c] : yy[0][c];
    };

    int shift = 0;  // after this warp's own phase, position c holds its local column (c + shift) % CW

#pragma unroll 1
    for (int ph = 0; ph < W; ++ph) {
        const int pc0 = ph * CW;
        const int nloc = min(CW, n - pc0);
        if (nloc <= 0) break;  // same for every warp
        const int G = (nloc + U - 1) / U;
        if (warp == ph) {
            // ---- owner: reflectors of columns pc0 .. pc0+nloc-1, in groups of
            // U with the register rotation of factor_tile, and the norm of the
            // next column reduced while the current update is issued
            SC sig2, alpha;
            {
                SC s4[4] = {SC(0), SC(0), SC(0), SC(0)};
#pragma unroll
                for (int i = 0; i < RPT; ++i)
                    if (below(i, pc0)) s4[i & 3] = fmadd((SC)y[i][0], (SC)y[i][0], s4[i & 3]);
                alpha = (SC)__shfl_sync(kFull, diag_slot(y, 0, pc0), pc0 & 31);
                sig2 = warp_sum((s4[0] + s4[1]) + (s4[2] + s4[3]));
            }
#pragma unroll 1
            for (int g = 0; g < G; ++g) {
                const int base = U * g;
                const int live = nloc - base;
                const int past0 = CW - base;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (kTrim && base + u >= nloc) continue;
                    const int j = pc0 + base + u;
                    const bool zero = (sig2 == SC(0));
                    const SC nrm = rsq(fmadd(alpha, alpha, sig2));
                    const SC beta_s = zero ? alpha : ((alpha >= SC(0)) ? -nrm : nrm);
                    const T beta = (T)beta_s;
                    const T tau = zero ? T(0) : (T)((beta_s - alpha) * rcp(beta_s));
                    const T scale = zero ? T(0) : (T)rcp(alpha - beta_s);
#pragma unroll
                    for (int i = 0; i < RPT; ++i)
                        if (below(i, j)) y[i][u] *= scale;
                    // v_j of slot i (1 on the diagonal, 0 above it)
                    auto vj = [&](int i) { return below(i, j) ? y[i][u] : ((lane + 32 * i == j) ? T(1) : T(0)); };
                    const int b = j & 1;
                    VL::store(S.vbuf[b], lane, vsw, vj);
                    if (lane == 0) {
                        S.taub[b] = tau;
                        S.tau[j] = tau;
                        S.rdiag[j] = beta;
                    }
                    step_barrier(W * 32);
                    T q[CW];
#pragma unroll
                    for (int c = 0; c < CW; ++c) {
                        q[c] = (c != u) ? vj(0) * y[0][c] : T(0);
#pragma unroll
                        for (int i = 1; i < RPT; ++i)
                            if (c != u) q[c] = fmadd(vj(i), y[i][c], q[c]);
                    }
                    const T d = warp_colsum<T, CW>(q, scratch, lane);
                    if (lane < CW) {
                        S.coef[warp][lane] = (lane > u && lane < live) ? (kFold ? tau * d : d) : T(0);
                        const int k = (lane >= past0) ? lane - past0 : ((lane < u) ? base + lane : -1);
                        if (k >= 0) S.Sc.c[j][pc0 + k] = d;
                    }
                    __syncwarp();
                    T tv[RPT];
#pragma unroll
                    for (int i = 0; i < RPT; ++i) tv[i] = kFold ? vj(i) : tau * vj(i);
                    T cf[CW];
#pragma unroll
                    for (int c0 = 0; c0 < CW; c0 += VN) {
                        if (c0 + VN - 1 <= u) continue;
                        Vec16<T>::load(&S.coef[warp][c0], &cf[c0]);
                    }
                    if (u + 1 < CW) {
                        const int c = (u + 1 < CW) ? u + 1 : 0;  // keeps the index in range when u + 1 == CW
#pragma unroll
                        for (int i = 0; i < RPT; ++i) y[i][c] = fmadd(-tv[i], cf[c], y[i][c]);
                        SC s4[4] = {SC(0), SC(0), SC(0), SC(0)};  // four chains instead of one RPT-deep one
#pragma unroll
                        for (int i = 0; i < RPT; ++i)
                            if (below(i, j + 1)) s4[i & 3] = fmadd((SC)y[i][c], (SC)y[i][c], s4[i & 3]);
                        alpha = (SC)__shfl_sync(kFull, diag_slot(y, c, j + 1), (j + 1) & 31);
                        sig2 = warp_sum((s4[0] + s4[1]) + (s4[2] + s4[3]));
                    }
#pragma unroll
                    for (int c = u + 2; c < CW; ++c)
#pragma unroll
                        for (int i = 0; i < RPT; ++i) y[i][c] = fmadd(-tv[i], cf[c], y[i][c]);
                }
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    T keep[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) keep[u] = y[i][u];
#pragma unroll
                    for (int c = 0; c < CW - U; ++c) y[i][c] = y[i][c + U];
#pragma unroll
                    for (int u = 0; u < U; ++u) y[i][CW - U + u] = keep[u];
                }
            }
            shift = (U * G) % CW;
        } else {
            // ---- the other warps: apply H_j (later columns) or take column j
            // of V^T V (finished columns), one barrier per step as the owner
            const bool trailing = warp > ph;
#pragma unroll 1
            for (int st = 0; st < (kTrim ? nloc : G * U); ++st) {
                const int j = pc0 + st;
                step_barrier(W * 32);
                const int b = j & 1;
                T v[RPT];
                VL::load(S.vbuf[b], lane, vsw, v);
                const T tau = S.taub[b];
                T q[CW];
#pragma unroll
                for (int c = 0; c < CW; ++c) {
                    q[c] = v[0] * y[0][c];
#pragma unroll
                    for (int i = 1; i < RPT; ++i) q[c] = fmadd(v[i], y[i][c], q[c]);
                }
                const T d = warp_colsum<T, CW>(q, scratch, lane);
                if (trailing) {
                    if (lane < CW) S.coef[warp][lane] = kFold ? tau * d : d;
                    __syncwarp();
                    T tv[RPT];
#pragma unroll
                    for (int i = 0; i < RPT; ++i) tv[i] = kFold ? v[i] : tau * v[i];
#pragma unroll
                    for (int c0 = 0; c0 < CW; c0 += VN) {
                        T w[VN];
                        Vec16<T>::load(&S.coef[warp][c0], w);
#pragma unroll
                        for (int e = 0; e < VN; ++e)
#pragma unroll
                            for (int i = 0; i < RPT; ++i) y[i][c0 + e] = fmadd(-tv[i], w[e], y[i][c0 + e]);
                    }
                } else if (lane < CW) {
                    const int kl = (lane + shift) % CW;
                    if (kl < mycols) S.Sc.c[j][col0 + kl] = d;
                }
            }
        }
    }
    return shift;
}

// One tile: ht rows of n columns at `tile` (leading dimension ld), its R to
// Rt (leading dimension ldr).  A kernel whose registers are full keeps it in
// shared memory, from which it is read again after the column steps.
template <typename T>
struct TileDesc {
    T* tile;
    T* Rt;
    int64_t ld, ldr;
    int ht, n;
};
// VECV: publish the reflector in the 16-byte vector layout (VbufLayout).
// Off for the 64-column tile and for the batched kernels, whose registers
// leave no room for the aligned quads it needs (more spills with it).
// N64: the owner's column norm (sigma^2, accumulated and reduced), alpha and
// the reflector scalars beta, tau and 1/(alpha - beta) in FP64, rounded to
// the tile's type once computed; the tile, the dot products and the updates
// stay in T.  (The precision form's option fp64_scalars.)
// The tile comes from global memory (Hook = NoHook), or from a copy in
// shared memory staged by TMA (any other Hook; stile): 256-row boxes of
// NMAX columns, box h holding rows [256h, 256h + 256) column by column, the
// rows past the level's end and the columns past n already zero.  `loaded`
// runs once every thread holds its values.
struct NoHook {
    __device__ __forceinline__ void operator()() const {}
};
template <typename T, int NMAX, int CW, int RPT, bool VECV = (NMAX <= 32), bool N64 = false, class Hook = NoHook>
__device__ __forceinline__ void factor_split_tile(SplitFactorSmem<T, NMAX, CW, RPT>& S, const TileDesc<T>& d,
                                                  const T* stile = nullptr, Hook loaded = Hook()) {
    constexpr int W = NMAX / CW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col0 = warp * CW;

    T y[RPT][CW];
    if constexpr (!std::is_same<Hook, NoHook>::value) {
        // rows lane + 32 i of box i / 8, consecutive lanes on consecutive words
        const T* s0 = stile + col0 * 256 + lane;
#pragma unroll
        for (int c = 0; c < CW; ++c)
#pragma unroll
            for (int i = 0; i < RPT; ++i) y[i][c] = s0[((i >> 3) * NMAX + c) * 256 + 32 * (i & 7)];
    } else {
        // one column pointer stepped by ld; the row offsets 32*i are immediates
        const int ht = d.ht, mycols = max(0, min(CW, d.n - col0));
        const T* pcol = d.tile + (int64_t)col0 * d.ld + lane;
#pragma unroll
        for (int c = 0; c < CW; ++c) {
#pragma unroll
            for (int i = 0; i < RPT; ++i) y[i][c] = (lane + 32 * i < ht && c < mycols) ? pcol[32 * i] : T(0);
            pcol += d.ld;
        }
    }
    loaded();
    const int shift = split_steps<T, NMAX, CW, RPT, VECV, N64>(S, y, d.n);
    step_barrier(W * 32);  // tau, rdiag and V^T V complete
    T* const tile = d.tile;
    T* const Rt = d.Rt;
    const int64_t ld = d.ld, ldr = d.ldr;
    const int ht = d.ht, n = d.n, mycols = max(0, min(CW, n - col0));

    // R (row r < n sits in slot r / 32 of lane r % 32 in the warp holding
    // column k) and V below the diagonal, each warp for its own columns.
#pragma unroll
    for (int c = 0; c < CW; ++c) {
        const int kl = (c + shift) % CW;
        if (kl < mycols) {
            const int k = col0 + kl;
#pragma unroll
            for (int i = 0; i < (NMAX + 31) / 32; ++i) {
                const int r = lane + 32 * i;
                if (r < n) {
                    T v = (k > r) ? y[i][c] : ((k == r) ? S.rdiag[r] : T(0));
                    if (r >= ht) v = T(0);
                    Rt[r + (int64_t)k * ldr] = v;
                }
            }
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = lane + 32 * i;
                if (r < ht && r > k) tile[r + (int64_t)k * ld] = y[i][c];
            }
        }
    }
    // T in the top block's upper triangle (diagonal included), row i by
    // thread i: T(i,i) = tau_i, T(i,j) = -tau_j sum_{k=i}^{j-1} T(i,k) S(k,j).
    {
        const int i = threadIdx.x;
        if (i < n && i < ht) {
            T trow[NMAX];
            t_factor_row<T, NMAX>(S.Sc, S.tau, i, n, trow);
#pragma unroll
            for (int j = 0; j < NMAX; ++j)
                if (j >= i && j < n) tile[i + (int64_t)j * ld] = trow[j];
        }
    }
    step_barrier(W * 32);  // S is reused by the CTA's next tile
}

template <typename T, int NMAX, int CW, int RPT, int MINB, bool N64 = false>
__global__ void __launch_bounds__(32 * (NMAX / CW), MINB) factor_split_tiles(FactorParams<T> p) {
    pdl_begin();
    constexpr int B = 32 * RPT;
    __shared__ SplitFactorSmem<T, NMAX, CW, RPT> S;
    for (int64_t t = blockIdx.x; t < p.ntiles; t += gridDim.x) {
        const int64_t row0 = t * B;
        const int ht = (int)((p.h - row0) < B ? (p.h - row0) : B);
        const TileDesc<T> d{p.M + row0, p.Rout + t * p.n, p.ld, p.ldr, ht, p.n};
        factor_split_tile<T, NMAX, CW, RPT, (NMAX <= 32), N64>(S, d);
    }
    if constexpr (!N64) clear_status(p);  // in front of the loop, or with N64, it would spill
}

// Persistent form of factor_split_tiles whose tiles are staged into shared
// memory by TMA (two 256-row boxes of a 512-row tile, rows past the level's
// end filled with zeros by the copy itself): a CTA waits for its tile, every
// thread takes its values into registers, and the TMA of the CTA's next tile
// is issued while the current one is factored, so the tile load leaves the
// tile's chain.  The wait is bounded: after p.tries polls the CTA sets the
// status word, waits (with the full limit) for the copy in flight and stops.
// Dynamic shared memory of the TMA form: the tile's boxes, then the
// mbarrier that counts their bytes (both at fixed offsets, so neither
// address takes a register across the tile).
extern __shared__ __align__(128) unsigned char tma_stage[];
template <typename T, int NMAX, int CW, int RPT>
constexpr size_t tma_tile_bytes() {
    return (size_t)(RPT / 8) * NMAX * 256 * sizeof(T);
}
template <typename T, int NMAX, int CW, int RPT>
constexpr size_t tma_stage_bytes() {
    return tma_tile_bytes<T, NMAX, CW, RPT>() + 16;
}
// One thread: the copies of the tile whose first row is y, counted on the
// stage's mbarrier.
template <int BOXES, int BOX_BYTES>
__device__ __forceinline__ void tma_issue_tile(const CUtensorMap* tmap, int y) {
    const uint32_t dst = tc::smem_u32(tma_stage), mb = dst + BOXES * BOX_BYTES;
    tc::fence_smem_to_async();
    tc::mbar_arrive_expect_tx(mb, (uint32_t)(BOXES * BOX_BYTES));
#pragma unroll
    for (int h = 0; h < BOXES; ++h) tc::tma_load_2d(dst + h * BOX_BYTES, tmap, y + h * 256, 0, mb);
}
// The `loaded` hook of the TMA form: every thread holds its values, so the
// buffer is free and thread 0 (go) starts the next tile's copy.  Held by
// value: a hook that referred to the loop's locals would put them on the
// stack.
template <int BOXES, int BOX_BYTES>
struct TmaNextTile {
    const CUtensorMap* tmap;
    int y;
    bool go;
    __device__ __forceinline__ void operator()() const {
        __syncthreads();
        if (go) tma_issue_tile<BOXES, BOX_BYTES>(tmap, y);
    }
};
template <typename T, int NMAX, int CW, int RPT, int MINB>
__global__ void __launch_bounds__(32 * (NMAX / CW), MINB)
    factor_split_tiles_tma(FactorParams<T> p, const __grid_constant__ CUtensorMap tmap) {
    pdl_begin();
    static_assert(RPT % 8 == 0, "tiles of whole 256-row boxes");
    constexpr int B = 32 * RPT, BOXES = RPT / 8, BOX_BYTES = NMAX * 256 * (int)sizeof(T);
    __shared__ SplitFactorSmem<T, NMAX, CW, RPT> S;
    const T* stile = reinterpret_cast<const T*>(tma_stage);
    const uint32_t mb = tc::smem_u32(tma_stage) + BOXES * BOX_BYTES;
    if (threadIdx.x == 0) {
        tc::mbar_init(mb, 1);
        tc::fence_mbar_init();
    }
    __syncthreads();
    // Row coordinates fit 32 bits (TMA takes them signed; the host launches
    // this kernel for ntiles * B <= INT32_MAX only).  The loop carries one
    // counter k (tile
    // blockIdx.x + k gridDim.x, mbarrier phase k & 1) across the tile's
    // body, which needs every register it can get.
    const int ntiles = (int)p.ntiles;
    if (threadIdx.x == 0 && (int)blockIdx.x < ntiles)
        tma_issue_tile<BOXES, BOX_BYTES>(&tmap, (int)blockIdx.x * B);
#pragma unroll 1
    for (int k = 0;; ++k) {
        const int t = (int)blockIdx.x + k * (int)gridDim.x;
        if (t >= (int)p.ntiles) break;
        const uint32_t phase = (uint32_t)k & 1u;
        const bool ok = tc::mbar_wait(mb, phase, p.tries);
        if (__syncthreads_or(!ok)) {
            if (threadIdx.x == 0) {
                if (p.err) atomicExch(p.err, 1);
                // the copy in flight must not land after the CTA is gone:
                // this wait keeps the full limit
                (void)tc::mbar_wait(mb, phase);
            }
            break;
        }
        const int64_t row0 = (int64_t)t * B;
        const int ht = (int)((p.h - row0) < B ? (p.h - row0) : B);
        const int tn = t + (int)gridDim.x;
        const TmaNextTile<BOXES, BOX_BYTES> loaded{&tmap, tn * B, threadIdx.x == 0 && tn < (int)p.ntiles};
        const TileDesc<T> d{p.M + row0, p.Rout + t * p.n, p.ld, p.ldr, ht, p.n};
        factor_split_tile<T, NMAX, CW, RPT, (NMAX <= 32), false>(S, d, stile, loaded);
    }
}

template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// ---------------------------------------------------------------------------
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Q assembly of FP32 tiles: Q = [B; 0] - V W with W = T (V_top^T B), in place.
//
// A CTA of 256 threads walks a tile in chunks of CH rows, staged in shared
// memory by asynchronous copies in two buffers: chunk c+1 is on its way while
// chunk c is multiplied.  A thread
// owns 4 rows x TC columns of a chunk; per k it reads one 16-byte vector of V
// and TC/4 of W.  Lanes that share a column group are adjacent: a warp's
// 16-byte read of one address by adjacent lanes costs 2.1 cycles of the SM's
// shared-memory pipe, 4.0 where neighbouring lanes differ (measured), and W
// is read twice as often as V.
// W is formed once per tile from chunk 0: the strict lower part of the top
// block is V_top, its upper triangle T, so both products run over half of the
// terms and need masks in their diagonal blocks only.  B is staged row-major
// in the buffer that W takes over.
template <int NMAX, int ROWS>
struct ApplyF32 {
    static constexpr int NT = 256;
    static constexpr int TC = NMAX >= 32 ? 8 : 4;  // columns per thread
    static constexpr int CG = NMAX / TC;           // column groups
    static constexpr int LPG = 32 / CG;            // lanes of a warp that share a column group
    static constexpr int CH = 4 * (NT / CG);       // rows per chunk
    static constexpr int NCH = ROWS / CH;
    static constexpr int LDW = NMAX + 4;           // row stride of B / W / Y
    static constexpr int BK = NMAX >= 16 ? NMAX / 16 : 1;  // outputs per thread and direction in the small products
    static constexpr int NB = NMAX / BK;
    static constexpr int kBuf = NMAX * CH;
    static constexpr int kBufs = NCH > 1 ? 2 : 1;
    static constexpr size_t kSmem = sizeof(float) * (size_t)(kBufs * kBuf + 2 * NMAX * LDW);
    // resident CTAs per SM: as many as shared memory (n > 16) or 64 registers allow
    static constexpr int kResident = NMAX > 32 ? 2 : (NMAX > 16 ? (NCH > 1 ? 3 : 2) : 4);
    static_assert(ROWS % CH == 0 && CH >= NMAX, "whole chunks; the top block lies in chunk 0");
};

// One thread's asynchronous copies of chunk ch of a tile into buf ([column]
// [CH rows]); rows past the tile's end are not copied, except that the rows
// below NMAX of chunk 0 are zeroed there (the small products read them).
template <int NMAX, int ROWS>
__device__ __forceinline__ void apply_stage(float* buf, const float* tile, int64_t ld, int ch, int ht, int n, int vec) {
    using A = ApplyF32<NMAX, ROWS>;
    const int tid = threadIdx.x;
    const int r0 = ch * A::CH;
    if (vec) {
        constexpr int NV = A::CH / 4;
#pragma unroll 4
        for (int e = tid; e < n * NV; e += A::NT) {
            const int c = e / NV, r = (e % NV) * 4;
            if (r0 + r + 4 <= ht) {
                cp_async<16>(buf + c * A::CH + r, tile + r0 + r + (int64_t)c * ld);
            } else {
                for (int rr = r; rr < r + 4; ++rr) {
                    if (r0 + rr < ht)
                        cp_async<4>(buf + c * A::CH + rr, tile + r0 + rr + (int64_t)c * ld);
                    else if (r0 + rr < NMAX)
                        buf[c * A::CH + rr] = 0.f;
                }
            }
        }
    } else {
#pragma unroll 8
        for (int e = tid; e < n * A::CH; e += A::NT) {
            const int c = e / A::CH, r = e % A::CH;
            if (r0 + r < ht)
                cp_async<4>(buf + c * A::CH + r, tile + r0 + r + (int64_t)c * ld);
            else if (r0 + r < NMAX)
                buf[c * A::CH + r] = 0.f;
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// BK consecutive floats (BK = 1, 2 or 4) from an aligned shared address.
template <int BK>
__device__ __forceinline__ void load_bk(const float* p, float (&v)[BK]) {
    if constexpr (BK == 4) {
        Vec16<float>::load(p, v);
    } else if constexpr (BK == 2) {
        const float2 q = *reinterpret_cast<const float2*>(p);
        v[0] = q.x, v[1] = q.y;
    } else {
        v[0] = *p;
    }
}

// Q of one tile: ht (<= ROWS) rows of n columns at `tile` (ld), holding V and
// T, overwritten by (I - V T V^T) [B; 0], B the n x n block at Pb (ldp) or the
// identity where Pb is null.  vec: 16-byte accesses are legal (ld and tile
// aligned).  sm: ApplyF32::kSmem bytes.  Called by every thread.
template <int NMAX, int ROWS>
__device__ __forceinline__ void apply_tile_f32(float* sm, float* tile, int64_t ld, int ht, int n, const float* Pb,
                                               int64_t ldp, int vec) {
    using A = ApplyF32<NMAX, ROWS>;
    constexpr int TC = A::TC, CH = A::CH, LDW = A::LDW, BK = A::BK, NT = A::NT;
    float* D0 = sm;
    float* D1 = sm + (A::kBufs - 1) * A::kBuf;
    float* Wb = D1 + A::kBuf;
    float* Y = Wb + NMAX * LDW;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    apply_stage<NMAX, ROWS>(D0, tile, ld, 0, ht, n, vec);
    if constexpr (A::NCH > 1) apply_stage<NMAX, ROWS>(D1, tile, ld, 1, ht, n, vec);
    {
        // all global reads first, then the stores (the generic pointers may alias)
        constexpr int PER = (NMAX * NMAX + NT - 1) / NT;
        float bv[PER];
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = tid + NT * e, r = idx % NMAX, c = idx / NMAX;
            const bool ok = idx < NMAX * NMAX && r < n && c < n;
            bv[e] = Pb ? (ok ? Pb[r + (int64_t)c * ldp] : 0.f) : (ok && r == c ? 1.f : 0.f);
        }
#pragma unroll
        for (int e = 0; e < PER; ++e) {
            const int idx = tid + NT * e;
            if (idx < NMAX * NMAX) Wb[(idx % NMAX) * LDW + idx / NMAX] = bv[e];
        }
    }
    cp_async_wait_group<(A::NCH > 1 ? 1 : 0)>();
    __syncthreads();
    // Y = V_top^T B and W = T Y, a BK x BK block per thread: rows k0.., columns c0..
    const int k0 = (tid / A::NB) * BK, c0 = (tid % A::NB) * BK;
    const bool small = tid < A::NB * A::NB && k0 < n;
    if (small) {
        float a[BK][BK] = {};
        // r = k0 .. k0 + BK - 1: unit diagonal, zero above it
#pragma unroll
        for (int d = 0; d < BK; ++d) {
            float b[BK];
            load_bk<BK>(Wb + (k0 + d) * LDW + c0, b);
#pragma unroll
            for (int i = 0; i <= d; ++i) {
                const float v = i == d ? 1.f : D0[(k0 + i) * CH + k0 + d];
#pragma unroll
                for (int q = 0; q < BK; ++q) a[i][q] = fmaf(v, b[q], a[i][q]);
            }
        }
#pragma unroll 2
        for (int r = k0 + BK; r < n; r += BK) {
            float v[BK][BK];
#pragma unroll
            for (int i = 0; i < BK; ++i) load_bk<BK>(D0 + (k0 + i) * CH + r, v[i]);
#pragma unroll
            for (int d = 0; d < BK; ++d) {
                float b[BK];
                load_bk<BK>(Wb + (r + d) * LDW + c0, b);
#pragma unroll
                for (int i = 0; i < BK; ++i)
#pragma unroll
                    for (int q = 0; q < BK; ++q) a[i][q] = fmaf(v[i][d], b[q], a[i][q]);
            }
        }
#pragma unroll
        for (int i = 0; i < BK; ++i)
#pragma unroll
            for (int q = 0; q < BK; ++q) Y[(k0 + i) * LDW + c0 + q] = a[i][q];
    }
    __syncthreads();
    if (small) {
        float a[BK][BK] = {};
#pragma unroll 4
        for (int l = k0; l < n; ++l) {
            float t[BK], y[BK];
            load_bk<BK>(D0 + l * CH + k0, t);  // T(k0.., l); zero below the diagonal
            load_bk<BK>(Y + l * LDW + c0, y);
#pragma unroll
            for (int i = 0; i < BK; ++i) {
                const float x = k0 + i <= l ? t[i] : 0.f;
#pragma unroll
                for (int q = 0; q < BK; ++q) a[i][q] = fmaf(x, y[q], a[i][q]);
            }
        }
        // -W, over B
#pragma unroll
        for (int i = 0; i < BK; ++i)
#pragma unroll
            for (int q = 0; q < BK; ++q) Wb[(k0 + i) * LDW + c0 + q] = -a[i][q];
    }
    __syncthreads();
    // the top block becomes V_top itself
    for (int e = tid; e < NMAX * NMAX; e += NT) {
        const int r = e % NMAX, k = e / NMAX;
        if (r <= k) D0[k * CH + r] = r == k ? 1.f : 0.f;
    }
    __syncthreads();

    const int cg = lane / A::LPG;
    const int row = 4 * (warp * A::LPG + lane % A::LPG);  // the thread's first row in a chunk
    const float* wp = Wb + 4 * cg;
#pragma unroll 1
    for (int ch = 0; ch < A::NCH; ++ch) {
        float* D = (ch & 1) ? D1 : D0;
        if (ch * CH < ht) {
            float2 q[4][TC / 2];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int c = 0; c < TC / 2; ++c) q[i][c] = make_float2(0.f, 0.f);
#pragma unroll 4
            for (int k = 0; k < n; ++k) {
                const float4 v = *reinterpret_cast<const float4*>(D + row + k * CH);
                const float vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int c4 = 0; c4 < TC / 4; ++c4) {  // columns 4 cg .. +3 of each NMAX / (TC / 4) block
                    const float4 w = *reinterpret_cast<const float4*>(wp + k * LDW + c4 * (NMAX / 2));
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float2 vi = make_float2(vv[i], vv[i]);
                        q[i][2 * c4] = __ffma2_rn(vi, make_float2(w.x, w.y), q[i][2 * c4]);
                        q[i][2 * c4 + 1] = __ffma2_rn(vi, make_float2(w.z, w.w), q[i][2 * c4 + 1]);
                    }
                }
            }
            const int r = ch * CH + row;
            if (r < n) {  // the top block: Q = B - V W
#pragma unroll
                for (int c = 0; c < TC; ++c) {
                    const int col = (c / 4) * (NMAX / 2) + 4 * cg + (c & 3);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (r + i < n && col < n) {
                            const float b = Pb ? Pb[r + i + (int64_t)col * ldp] : (r + i == col ? 1.f : 0.f);
                            if (c & 1)
                                q[i][c / 2].y += b;
                            else
                                q[i][c / 2].x += b;
                        }
                }
            }
            float* g = tile + (int64_t)ch * CH;
            if (!vec) __syncthreads();  // every thread has read the chunk's V
#pragma unroll
            for (int c = 0; c < TC; ++c) {
                const int col = (c / 4) * (NMAX / 2) + 4 * cg + (c & 3);
                const float4 o = (c & 1) ? make_float4(q[0][c / 2].y, q[1][c / 2].y, q[2][c / 2].y, q[3][c / 2].y)
                                         : make_float4(q[0][c / 2].x, q[1][c / 2].x, q[2][c / 2].x, q[3][c / 2].x);
                if (!vec) {  // through the chunk's buffer: consecutive lanes then store consecutive rows
                    *reinterpret_cast<float4*>(D + row + col * CH) = o;
                } else if (col < n) {
                    float* gc = g + row + (int64_t)col * ld;
                    if (r + 4 <= ht) {
                        *reinterpret_cast<float4*>(gc) = o;
                    } else {
                        if (r < ht) gc[0] = o.x;
                        if (r + 1 < ht) gc[1] = o.y;
                        if (r + 2 < ht) gc[2] = o.z;
                    }
                }
            }
            if (!vec) {
                __syncthreads();
#pragma unroll 4
                for (int e = tid; e < n * CH; e += NT)
                    if (ch * CH + e % CH < ht) g[e % CH + (int64_t)(e / CH) * ld] = D[e];
            }
        }
        if (ch + 1 < A::NCH) {
            __syncthreads();  // the chunk's buffer is free
            if (ch + 2 < A::NCH) {
                apply_stage<NMAX, ROWS>(D, tile, ld, ch + 2, ht, n, vec);
                cp_async_wait_group<1>();
            } else {
                cp_async_wait_group<0>();
            }
            __syncthreads();
        }
    }
}

// One tile per CTA: the next CTA's copies run under this one's products.
// Measured against the kernel it replaced (two rows x all columns per thread,
// the tile staged whole, W by plain dot products: shared-memory reads and one
// or two CTAs per SM bound it), level 0, us: 4,194,304 x 32 440 -> 277,
// 2,097,152 x 64 1050 -> 478, 4,194,304 x 16 128 -> 106, x 8 57 -> 47; one
// tile per SM: x 32 14.6 -> 10.3, x 64 39 -> 25; with an odd ld, 1,000,003 x 32
// 123 -> 96, x 64 517 -> 287.
template <int NMAX, int ROWS, int MINB>
__global__ void __launch_bounds__(256, MINB) apply_tiles_f32(ApplyParams<float> p) {
    pdl_begin();
    extern __shared__ __align__(16) float apply_sm[];
    const int64_t t = blockIdx.x;
    const int64_t left = p.h - t * ROWS;
    apply_tile_f32<NMAX, ROWS>(apply_sm, p.M + t * ROWS, p.ld, (int)(left < ROWS ? left : ROWS), p.n,
                               p.P ? p.P + t * p.n : nullptr, p.ldp, p.vec);
}

}  // namespace tsqr
