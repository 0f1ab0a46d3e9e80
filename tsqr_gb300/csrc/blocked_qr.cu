// blocked_qr.cu -- recursive blocked QR over TSQR panels (plain precision).
//
// Replaces qr<T> (block_QR.h:72-95): recursive block classical Gram-Schmidt,
//   qr(A1);  R12 = A1^T A2;  A2 -= A1 R12;  qr(A2),
// with TSQR on panels of width <= panel (32, the reference's N_B,
// block_QR.h:5).  The reference's single naive kernel gemm_blockqr
// (block_QR.h:7-60: one thread per output, a length-m dot with stride-lda
// loads for op=T) becomes tiled SIMT kernels:
//   gemm_tn_fused (FP32): R12 = A1^T A2 in 32 x 32 output tiles, K = m split
//     across CTAs, the partial sums reduced in the same launch in a fixed
//     order (deterministic);
//   gemm_tn_partial + reduce_partials (FP64): the same product as split-K
//     partials of 64 x 64 tiles, then their sum;
//   gemm_nn: A2 = A2 - A1 R12, streamed over row blocks.
// Options the reference lacks: any split point (not only n/2 with
// (n/2) % 32 == 0, block_QR.h:78-79), a second projection (CGS2) when
// opts.reorth is set, and R21 written as zeros (the reference leaves it
// unwritten).
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "internal.h"
#include "tc.cuh"

namespace tsqr {

namespace {

constexpr int kTile = 64;    // output tile edge of gemm_nn (rows)
constexpr int kTnTile = 32;  // output tile edge of gemm_tn_partial
constexpr int kKt = 16;      // k step through shared memory
constexpr int kTnBlock = 256;  // rows that gemm_tn_partial sums on their own

// P_z (M x N, ld M) = sum over k in chunk z of A(k, i) * B(k, j);
// A is K x M, B is K x N, both column-major.
// FP64 (its only type): bound by the FP64 rate, 16 cycles of the SM per warp
// instruction, so the output tile is 32 wide and a 32-wide node computes no
// padding; the loads for 2 x 2 outputs per thread cost nothing beside it.
// 27,648 rows, us: 32 x 32 264 -> 55, the three products of a 128-column qr
// 799 -> 305, against a 64 x 64 tile with 4 x 4 outputs in chunks of at least
// 256 rows.  A chunk may be long (wide nodes fill the SMs with one each), so its
// products are summed in blocks of 256 rows: a running sum of k terms has a
// rounding error that grows with k, and one of 1100 rows cost a 1100 x 1024 qr a
// quarter of its orthogonality.
template <typename T>
__global__ void __launch_bounds__(256) gemm_tn_partial(int M, int N, int64_t K, const T* __restrict__ A,
                                                       int64_t lda, const T* __restrict__ B, int64_t ldb,
                                                       T* __restrict__ P, int64_t kchunk) {
    pdl_begin();
    __shared__ __align__(16) T As[kKt][kTnTile + 2];
    __shared__ __align__(16) T Bs[kKt][kTnTile + 2];
    constexpr int R = kTnTile / 16;             // outputs per thread and direction
    constexpr int L = kKt * kTnTile / 256;      // elements loaded per thread and operand
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int i0 = blockIdx.x * kTnTile, j0 = blockIdx.y * kTnTile;
    const int64_t kbeg = (int64_t)blockIdx.z * kchunk;
    const int64_t kend = min(K, kbeg + kchunk);
    T sum[R][R] = {};
    // the next k step's elements are loaded into registers while the current
    // one is multiplied out of shared memory
    T ra[L], rb[L];
    auto fetch = [&](int64_t k0) {
#pragma unroll
        for (int e = 0; e < L; ++e) {
            const int idx = tid + 256 * e;
            const int kk = idx % kKt, col = idx / kKt;
            const int64_t k = k0 + kk;
            ra[e] = (k < kend && i0 + col < M) ? A[k + (int64_t)(i0 + col) * lda] : T(0);
            rb[e] = (k < kend && j0 + col < N) ? B[k + (int64_t)(j0 + col) * ldb] : T(0);
        }
    };
    if (kbeg < kend) fetch(kbeg);
    for (int64_t kb = kbeg; kb < kend; kb += kTnBlock) {
        T acc[R][R] = {};
        const int64_t ke = min(kend, kb + kTnBlock);
        for (int64_t k0 = kb; k0 < ke; k0 += kKt) {
#pragma unroll
            for (int e = 0; e < L; ++e) {
                const int idx = tid + 256 * e;
                const int kk = idx % kKt, col = idx / kKt;
                As[kk][col] = ra[e];
                Bs[kk][col] = rb[e];
            }
            __syncthreads();
            if (k0 + kKt < kend) fetch(k0 + kKt);
#pragma unroll
            for (int kk = 0; kk < kKt; ++kk) {
                T a[R], b[R];
#pragma unroll
                for (int u = 0; u < R; ++u) {
                    a[u] = As[kk][ty * R + u];
                    b[u] = Bs[kk][tx * R + u];
                }
#pragma unroll
                for (int u = 0; u < R; ++u)
#pragma unroll
                    for (int v = 0; v < R; ++v) acc[u][v] += a[u] * b[v];
            }
            __syncthreads();
        }
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int v = 0; v < R; ++v) sum[u][v] += acc[u][v];
    }
    T* Pz = P + (int64_t)blockIdx.z * M * N;
#pragma unroll
    for (int u = 0; u < R; ++u)
#pragma unroll
        for (int v = 0; v < R; ++v) {
            const int i = i0 + ty * R + u, j = j0 + tx * R + v;
            if (i < M && j < N) Pz[i + (int64_t)j * M] = sum[u][v];
        }
}

// C = alpha * sum_z P_z + beta * C  (C is M x N with ldc).  A CTA of 8
// warps takes 32 consecutive elements: warp w sums the partials z = w, w+8,
// ... of its lane's element (32 independent chains per warp, loads
// coalesced), then warp 0 adds the 8 warp sums in warp order, so the result
// is deterministic.
template <typename T>
__global__ void __launch_bounds__(256) reduce_partials(int M, int N, int nz, const T* __restrict__ P, T alpha,
                                                       T beta, T* C, int64_t ldc) {
    pdl_begin();
    __shared__ T s[8][32];
    const int64_t total = (int64_t)M * N;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int64_t base = (int64_t)blockIdx.x * 32; base < total; base += (int64_t)gridDim.x * 32) {
        const int64_t e = base + lane;
        T a0 = T(0), a1 = T(0);
        if (e < total) {
            int z = w;
            for (; z + 8 < nz; z += 16) {
                a0 += P[(int64_t)z * total + e];
                a1 += P[(int64_t)(z + 8) * total + e];
            }
            if (z < nz) a0 += P[(int64_t)z * total + e];
        }
        s[w][lane] = a0 + a1;
        __syncthreads();
        if (w == 0 && e < total) {
            T t = s[0][lane];
#pragma unroll
            for (int q = 1; q < 8; ++q) t += s[q][lane];
            const int i = (int)(e % M), j = (int)(e / M);
            T* c = C + i + (int64_t)j * ldc;
            *c = (beta == T(0)) ? alpha * t : alpha * t + beta * *c;
        }
        __syncthreads();
    }
}
inline int reduce_blocks(int64_t total) { return (int)std::min<int64_t>(ceil_div(total, 32), 4096); }

// ---------------------------------------------------------------------------
// FP32 projection in one launch: C (n1 x n2, ldc) = alpha A^T B + beta C for
// A (K x n1) and B (K x n2), column-major.  The output is cut in 32 x 32
// tiles, so a 32-wide node computes no padding.  The K rows are split into S
// chunks per tile, one CTA each.  A CTA stages 64 rows of its 32 + 32
// columns per step in shared memory and reduces the step over four K slices
// of 64 threads (4 x 4 outputs per thread, 16-byte shared-memory reads).
// Its partial tile goes to global memory.  The last CTA of each group of g
// chunks to arrive (an atomic counter) sums the group's partials, and the
// last group sums the group partials into C.  Both sums run in a fixed order,
// so the result does not depend on which CTA arrives last.  No CTA waits on
// another; the last one resets the tile's counters for the next launch.
constexpr int kPT = 32;      // output tile edge
constexpr int kPRows = 64;   // rows staged per step
constexpr int kPCounters = 256 / sizeof(int);  // counter words start here in the workspace header
constexpr int kPHeader = 4096;                 // status word + counters
constexpr int kPMaxCounters = kPHeader / (int)sizeof(int) - kPCounters;

struct TnFusedPlan {
    int tiles_i = 1, ntiles = 1, S = 1, g = 1, G = 1;
    int64_t kchunk = 0;
    size_t part_bytes() const {  // chunk partials, then group partials
        return S > 1 ? (size_t)ntiles * (S + G) * kPT * kPT * sizeof(float) : 0;
    }
};

TnFusedPlan tn_fused_plan(int64_t n1, int64_t n2, int64_t K) {
    TnFusedPlan p;
    p.tiles_i = (int)ceil_div(n1, kPT);
    p.ntiles = p.tiles_i * (int)ceil_div(n2, kPT);
    // one wave of three CTAs per SM on GB300's 152 SMs (the register limit
    // of 256 threads at 75 registers), chunks of whole 64-row steps.  The
    // workspace query uses the same plan, so it takes the constant rather
    // than the device's count.
    const int64_t want = std::max<int64_t>(1, (3 * 152) / p.ntiles);
    p.kchunk = round_up(ceil_div(K, std::min<int64_t>(want, ceil_div(K, kPRows))), kPRows);
    p.S = (int)ceil_div(K, p.kchunk);
    p.g = 1;
    while ((int64_t)p.g * p.g < p.S) ++p.g;
    p.G = (int)ceil_div(p.S, p.g);
    if (p.S > 1 && (int64_t)p.ntiles * (p.G + 1) > kPMaxCounters) {  // too many counters: one chunk per tile
        p.S = 1;
        p.kchunk = round_up(std::max<int64_t>(K, 1), kPRows);
        p.g = p.G = 1;
    }
    return p;
}

struct TnFusedArgs {
    int n1, n2;
    int64_t K;
    const float* A;
    const float* B;
    int64_t ld;  // A and B share it
    float* C;
    int64_t ldc;
    float* D;  // D += the product as well (null: nothing), at ldd
    int64_t ldd;
    float alpha, beta;
    int tiles_i, S, g, G;
    int64_t kchunk;
    float* part;  // [ntiles][S][1024]
    float* gpart;  // [ntiles][G][1024]
    int* cnt;      // [ntiles][G + 1], zero between launches
    int* err;      // status word (TMA form: a bounded wait gave up)
    int tries;     // polls of a bounded wait
};

// sum over z < n of q[z * 256] (float4 elements), in order of z, read from
// L2 (other CTAs wrote them): eight loads in flight per thread, the sum
// order unchanged (a missing term adds an exact zero)
__device__ __forceinline__ float4 sum_partials(const float4* q, int n) {
    constexpr int kStride = kPT * kPT / 4;
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int z0 = 0; z0 < n; z0 += 8) {
        float4 w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e)
            w[e] = z0 + e < n ? __ldcg(q + (int64_t)(z0 + e) * kStride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int e = 0; e < 8; ++e) u.x += w[e].x, u.y += w[e].y, u.z += w[e].z, u.w += w[e].w;
    }
    return u;
}

// The CTA's partial tile t (elements 4 tid .. 4 tid + 3 of the column-major
// 32 x 32 tile, in every thread) into C: directly when the tile has one
// chunk, else through the chunk partials and the two last-arriver sums.
__device__ __forceinline__ void tn_finish(const TnFusedArgs& p, float4 t, int tile, int chunk, int i0, int j0,
                                          int& s_last) {
    const int tid = threadIdx.x;
    auto store_c = [&](float4 s) {
        const float sv[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = 4 * tid + q, i = i0 + (e & 31), j = j0 + (e >> 5);
            if (i < p.n1 && j < p.n2) {
                float* c = p.C + i + (int64_t)j * p.ldc;
                const float x = p.beta == 0.f ? p.alpha * sv[q] : p.alpha * sv[q] + p.beta * *c;
                *c = x;
                if (p.D) p.D[i + (int64_t)j * p.ldd] += x;
            }
        }
    };
    if (p.S == 1) {
        store_c(t);
        return;
    }
    constexpr int E = kPT * kPT;
    __stcg(reinterpret_cast<float4*>(p.part + ((int64_t)tile * p.S + chunk) * E) + tid, t);
    __threadfence();
    __syncthreads();
    int* cnt = p.cnt + tile * (p.G + 1);
    const int grp = chunk / p.g, g0 = grp * p.g, gn = min(p.g, p.S - g0);
    if (tid == 0) s_last = atomicAdd(cnt + grp, 1) == gn - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    float4 u = sum_partials(reinterpret_cast<const float4*>(p.part + ((int64_t)tile * p.S + g0) * E) + tid, gn);
    if (p.G > 1) {
        __stcg(reinterpret_cast<float4*>(p.gpart + ((int64_t)tile * p.G + grp) * E) + tid, u);
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(cnt + p.G, 1) == p.G - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        u = sum_partials(reinterpret_cast<const float4*>(p.gpart + (int64_t)tile * p.G * E) + tid, p.G);
    }
    store_c(u);
    if (tid <= p.G) cnt[tid] = 0;  // every CTA of the tile has counted: ready for the next launch
}

// TMA-fed form (A and B 16-byte aligned, lda a multiple of 4 floats): each
// 64-row step arrives as four 32 x 32 boxes (A rows 0-31 and 32-63, then B)
// with the 128-byte swizzle, in a ring of kPStages steps on mbarriers (the
// copies of the next three steps run under the current step's FMAs).
// Column c of a box holds 32 rows as 8 chunks of 16 bytes, chunk q at
// q ^ (c % 8).  Thread (ig, jg) of a K slice owns output rows ig + 8u and
// columns jg + 8v (u, v < 4): its eight 16-byte reads per 4 rows are free
// of bank conflicts.  Rows past the matrix end and columns past n1 / n2
// arrive as zeros; chunks are whole 64-row steps, so a CTA's last step never
// reaches into the next chunk.  The waits are bounded: after p.tries polls
// the CTA sets the status word, lets its copies in flight land and stops.
constexpr int kPStages = 4;
constexpr int kPBox = kPT * kPT * 4;                       // one 32 x 32 FP32 box
constexpr int kPStageBytes = 4 * kPBox;                    // A and B, 64 rows each
constexpr size_t kPTmaSmem = kPStages * kPStageBytes + 1024;  // + alignment of the swizzled boxes

__global__ void __launch_bounds__(256, 3)
    gemm_tn_tma(TnFusedArgs p, const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb) {
    pdl_begin();
    extern __shared__ unsigned char tn_raw[];
    __shared__ unsigned long long mbar[kPStages];
    __shared__ int s_last;
    unsigned char* base = tn_raw + ((1024 - (tc::smem_u32(tn_raw) & 1023)) & 1023);
    const uint32_t sbase = tc::smem_u32(base);
    const int tid = threadIdx.x;
    const int tile = blockIdx.x, chunk = blockIdx.y;
    const int i0 = (tile % p.tiles_i) * kPT, j0 = (tile / p.tiles_i) * kPT;
    const int64_t kbeg = (int64_t)chunk * p.kchunk;
    const int64_t kend = min(p.K, kbeg + p.kchunk);
    const int nst = (int)((kend - kbeg + kPRows - 1) / kPRows);
    if (tid == 0) {
        for (int b = 0; b < kPStages; ++b) tc::mbar_init(tc::smem_u32(&mbar[b]), 1);
        tc::fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](int s) {  // thread 0
        const int b = s % kPStages;
        const uint32_t dst = sbase + b * kPStageBytes, mb = tc::smem_u32(&mbar[b]);
        const int x = (int)(kbeg + (int64_t)s * kPRows);
        tc::fence_smem_to_async();
        tc::mbar_arrive_expect_tx(mb, kPStageBytes);
        tc::tma_load_2d(dst, &ta, x, i0, mb);
        tc::tma_load_2d(dst + kPBox, &ta, x + 32, i0, mb);
        tc::tma_load_2d(dst + 2 * kPBox, &tb, x, j0, mb);
        tc::tma_load_2d(dst + 3 * kPBox, &tb, x + 32, j0, mb);
    };
    if (tid == 0)
        for (int s = 0; s < min(kPStages, nst); ++s) issue(s);

    const int sl = tid >> 6, lt = tid & 63, ig = lt & 7, jg = lt >> 3;
    float acc[4][4] = {};
    for (int s = 0; s < nst; ++s) {
        const int b = s % kPStages;
        const bool ok = tc::mbar_wait(tc::smem_u32(&mbar[b]), (uint32_t)(s / kPStages) & 1u, p.tries);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                if (p.err) atomicExch(p.err, 1);
                // the steps issued and not consumed: s .. s + kPStages - 1
                for (int q = s; q < min(s + kPStages, nst); ++q)
                    (void)tc::mbar_wait(tc::smem_u32(&mbar[q % kPStages]), (uint32_t)(q / kPStages) & 1u);
            }
            return;
        }
        // slice sl: rows 16 sl .. 16 sl + 15 of the step = box half sl / 2,
        // 4-row groups (sl % 2) * 4 .. + 3 of it
        const unsigned char* Ab = base + b * kPStageBytes + (sl >> 1) * kPBox;
        const unsigned char* Bb = Ab + 2 * kPBox;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int k4 = (sl & 1) * 4 + q;
            float4 a[4], bv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                a[u] = *reinterpret_cast<const float4*>(Ab + (ig + 8 * u) * 128 + ((k4 ^ ig) << 4));
#pragma unroll
            for (int v = 0; v < 4; ++v)
                bv[v] = *reinterpret_cast<const float4*>(Bb + (jg + 8 * v) * 128 + ((k4 ^ jg) << 4));
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    float c = acc[u][v];
                    c = fmaf(a[u].x, bv[v].x, c);
                    c = fmaf(a[u].y, bv[v].y, c);
                    c = fmaf(a[u].z, bv[v].z, c);
                    c = fmaf(a[u].w, bv[v].w, c);
                    acc[u][v] = c;
                }
        }
        __syncthreads();  // every thread is done with buffer b
        if (tid == 0 && s + kPStages < nst) issue(s + kPStages);
    }
    // the four slices' tiles (column-major, element j * 32 + i) in the ring's
    // first 16 KB: every copy has landed, all were waited for above
    float* red = reinterpret_cast<float*>(base);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) red[sl * kPT * kPT + (jg + 8 * v) * kPT + ig + 8 * u] = acc[u][v];
    __syncthreads();
    float4 t = *reinterpret_cast<const float4*>(red + 4 * tid);
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        const float4 w = *reinterpret_cast<const float4*>(red + q * kPT * kPT + 4 * tid);
        t.x += w.x, t.y += w.y, t.z += w.z, t.w += w.w;
    }
    tn_finish(p, t, tile, chunk, i0, j0, s_last);
}

template <bool VEC>
__global__ void __launch_bounds__(256, 3) gemm_tn_fused(TnFusedArgs p) {
    pdl_begin();
    __shared__ __align__(16) float sm[2 * kPRows * kPT];  // A step | B step; later the four K slices' tiles
    __shared__ int s_last;
    float* As = sm;
    float* Bs = sm + kPRows * kPT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tile = blockIdx.x, chunk = blockIdx.y;
    const int i0 = (tile % p.tiles_i) * kPT, j0 = (tile / p.tiles_i) * kPT;
    const int64_t kbeg = (int64_t)chunk * p.kchunk;
    const int64_t kend = min(p.K, kbeg + p.kchunk);

    // Loader: slot e of a thread covers rows 4kq..4kq+3 of one column gc of
    // the step (gc < 32: A's column i0 + gc, else B's column j0 + gc - 32);
    // a warp's slot is 4 columns x 32 rows, each column one 128-byte line.
    // Row r of column c is stored at [r][((c/4) ^ (r/4 % 8)) * 4 + c % 4]:
    // the stores of a warp hit 32 distinct banks, and a 16-byte read of 4
    // consecutive columns stays contiguous.
    const int kqa = lane & 7;
    const float* src[2];
    bool colok[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int gc = 4 * (warp * 2 + h) + (lane >> 3);
        const bool isA = gc < kPT;
        const int c = isA ? i0 + gc : j0 + gc - kPT;
        colok[h] = c < (isA ? p.n1 : p.n2);
        src[h] = (isA ? p.A : p.B) + (int64_t)(colok[h] ? c : 0) * p.ld;
    }
    float4 r[4];
    auto fetch = [&](int64_t k0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int64_t row = k0 + 4 * (8 * (e & 1) + kqa);
            const float* q = src[e >> 1] + row;
            if (!colok[e >> 1]) {
                r[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            } else if (VEC && row + 3 < kend) {
                r[e] = __ldg(reinterpret_cast<const float4*>(q));
            } else {
                r[e].x = row < kend ? __ldg(q) : 0.f;
                r[e].y = row + 1 < kend ? __ldg(q + 1) : 0.f;
                r[e].z = row + 2 < kend ? __ldg(q + 2) : 0.f;
                r[e].w = row + 3 < kend ? __ldg(q + 3) : 0.f;
            }
        }
    };

    // compute: slice sl takes rows 16 sl .. 16 sl + 15 of each step; thread
    // (ig, jg) of the slice owns rows 4ig.. and columns 4jg.. of the tile
    const int sl = tid >> 6, lt = tid & 63, ig = lt >> 3, jg = lt & 7;
    float acc[4][4] = {};
    if (kbeg < kend) fetch(kbeg);
    for (int64_t k0 = kbeg; k0 < kend; k0 += kPRows) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int kq = 8 * (e & 1) + kqa;
            const int gc = 4 * (warp * 2 + (e >> 1)) + (lane >> 3);
            float* dst = (gc < kPT ? As : Bs) + ((((gc & 31) >> 2) ^ (kq & 7)) << 2) + (gc & 3);
            dst[(4 * kq + 0) * kPT] = r[e].x;
            dst[(4 * kq + 1) * kPT] = r[e].y;
            dst[(4 * kq + 2) * kPT] = r[e].z;
            dst[(4 * kq + 3) * kPT] = r[e].w;
        }
        __syncthreads();
        if (k0 + kPRows < kend) fetch(k0 + kPRows);
#pragma unroll
        for (int kk = 0; kk < 16; ++kk) {
            const int k = 16 * sl + kk, s = (k >> 2) & 7;
            const float4 a = *reinterpret_cast<const float4*>(As + k * kPT + ((ig ^ s) << 2));
            const float4 b = *reinterpret_cast<const float4*>(Bs + k * kPT + ((jg ^ s) << 2));
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(av[u], bv[v], acc[u][v]);
        }
        __syncthreads();
    }

    // the four slices' tiles, column-major (element j*32 + i), summed in
    // slice order by the thread that owns elements 4t..4t+3
#pragma unroll
    for (int v = 0; v < 4; ++v)
        *reinterpret_cast<float4*>(sm + sl * kPT * kPT + (4 * jg + v) * kPT + 4 * ig) =
            make_float4(acc[0][v], acc[1][v], acc[2][v], acc[3][v]);
    __syncthreads();
    float4 t = *reinterpret_cast<const float4*>(sm + 4 * tid);
#pragma unroll
    for (int q = 1; q < 4; ++q) {
        const float4 w = *reinterpret_cast<const float4*>(sm + q * kPT * kPT + 4 * tid);
        t.x += w.x, t.y += w.y, t.z += w.z, t.w += w.w;
    }
    tn_finish(p, t, tile, chunk, i0, j0, s_last);
}

// ---------------------------------------------------------------------------
// FP32 update on CUDA cores: A2 (m x n2) += alpha A1 (m x n1) X (n1 x n2,
// ldx), A1 and A2 sharing lda, n1 <= 256.  A CTA owns a 32-column tile of
// A2 (blockIdx.y) and walks 128-row blocks (grid-stride, one wave).  X's
// n1 x 32 tile stays in shared memory for the whole launch.  A block's A1
// rows are staged 32 columns at a time (a straight copy of the column-major
// data, 16-byte stores); the next chunk, or the next block's first chunk
// and its A2 tile, are loaded into registers while the current chunk is
// multiplied.  Each thread owns 4 rows x 4 columns of the block and reads A1
// and X as 16-byte shared-memory vectors.
constexpr int kNR = 128;    // rows per block
constexpr int kNK = 32;     // K per staged chunk
constexpr int kNXs = 36;    // row stride of the X tile in shared memory (16-byte rows, 4-way store conflicts)
constexpr int kNMaxK = 256;

struct NnFusedArgs {
    int64_t m;
    int n1, n2;
    const float* A1;
    float* A2;
    int64_t lda;
    const float* X;
    int64_t ldx;
    float alpha;
};

size_t nn_fused_smem(int n1) { return ((size_t)round_up(n1, kNK) * kNXs + (size_t)kNK * kNR) * sizeof(float); }

template <bool VEC>
__global__ void __launch_bounds__(256, 2) gemm_nn_fused(NnFusedArgs p) {
    pdl_begin();
    extern __shared__ __align__(16) float nn_smem[];
    const int n1p = (p.n1 + kNK - 1) / kNK * kNK;
    float* Xs = nn_smem;              // [n1p][kNXs]
    float* As = nn_smem + n1p * kNXs;  // [kNK][kNR]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int j0 = blockIdx.y * 32;
    for (int e = tid; e < n1p * 32; e += 256) {
        const int i = e % n1p, j = e / n1p;
        Xs[i * kNXs + j] = (i < p.n1 && j0 + j < p.n2) ? p.X[i + (int64_t)(j0 + j) * p.ldx] : 0.f;
    }
    // compute: rows 4rg..4rg+3, columns 4cg..4cg+3 of the block
    const int rg = (warp & 3) * 8 + (lane & 7), cg = (warp >> 2) * 4 + (lane >> 3);
    const int64_t nblk = (p.m + kNR - 1) / kNR;

    // A1 chunk loader: float4 slot e = rows 4(idx%32).., column idx/32 of the chunk
    float4 ra[4];
    auto fetch_a = [&](int64_t row0, int kc) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + 256 * e, kk = idx >> 5;
            const int64_t r = row0 + 4 * (idx & 31);
            const int k = kc + kk;
            const float* q = p.A1 + (int64_t)k * p.lda + r;
            if (k >= p.n1) {
                ra[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            } else if (VEC && r + 3 < p.m) {
                ra[e] = __ldg(reinterpret_cast<const float4*>(q));
            } else {
                ra[e].x = r < p.m ? __ldg(q) : 0.f;
                ra[e].y = r + 1 < p.m ? __ldg(q + 1) : 0.f;
                ra[e].z = r + 2 < p.m ? __ldg(q + 2) : 0.f;
                ra[e].w = r + 3 < p.m ? __ldg(q + 3) : 0.f;
            }
        }
    };
    // A2 tile of the thread: column 4cg + v, rows 4rg..4rg+3
    float4 rc[4];
    auto fetch_c = [&](int64_t row0) {
        const int64_t r = row0 + 4 * rg;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int j = j0 + 4 * cg + v;
            const float* q = p.A2 + (int64_t)(j < p.n2 ? j : 0) * p.lda + r;
            if (j >= p.n2) {
                rc[v] = make_float4(0.f, 0.f, 0.f, 0.f);
            } else if (VEC && r + 3 < p.m) {
                rc[v] = *reinterpret_cast<const float4*>(q);
            } else {
                rc[v].x = r < p.m ? q[0] : 0.f;
                rc[v].y = r + 1 < p.m ? q[1] : 0.f;
                rc[v].z = r + 2 < p.m ? q[2] : 0.f;
                rc[v].w = r + 3 < p.m ? q[3] : 0.f;
            }
        }
    };

    int64_t blk = blockIdx.x;
    if (blk < nblk) {
        fetch_a(blk * kNR, 0);
        fetch_c(blk * kNR);
    }
    for (; blk < nblk; blk += gridDim.x) {
        const int64_t row0 = blk * kNR;
        float4 c[4] = {rc[0], rc[1], rc[2], rc[3]};
        float acc[4][4] = {};
        for (int kc = 0; kc < p.n1; kc += kNK) {
            __syncthreads();  // the previous chunk's reads of As are done (and, first, Xs is written)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int idx = tid + 256 * e;
                *reinterpret_cast<float4*>(As + (idx >> 5) * kNR + 4 * (idx & 31)) = ra[e];
            }
            __syncthreads();
            if (kc + kNK < p.n1) {
                fetch_a(row0, kc + kNK);
            } else if (blk + gridDim.x < nblk) {
                fetch_a((blk + gridDim.x) * kNR, 0);
                fetch_c((blk + gridDim.x) * kNR);
            }
#pragma unroll 8
            for (int kk = 0; kk < kNK; ++kk) {
                const float4 a = *reinterpret_cast<const float4*>(As + kk * kNR + 4 * rg);
                const float4 x = *reinterpret_cast<const float4*>(Xs + (kc + kk) * kNXs + 4 * cg);
                const float av[4] = {a.x, a.y, a.z, a.w}, xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(av[u], xv[v], acc[u][v]);
            }
        }
        const int64_t r = row0 + 4 * rg;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const int j = j0 + 4 * cg + v;
            if (j >= p.n2) continue;
            float4 o = c[v];
            o.x = fmaf(p.alpha, acc[0][v], o.x);
            o.y = fmaf(p.alpha, acc[1][v], o.y);
            o.z = fmaf(p.alpha, acc[2][v], o.z);
            o.w = fmaf(p.alpha, acc[3][v], o.w);
            float* q = p.A2 + (int64_t)j * p.lda + r;
            if (VEC && r + 3 < p.m) {
                *reinterpret_cast<float4*>(q) = o;
            } else {
                if (r < p.m) q[0] = o.x;
                if (r + 1 < p.m) q[1] = o.y;
                if (r + 2 < p.m) q[2] = o.z;
                if (r + 3 < p.m) q[3] = o.w;
            }
        }
    }
}

// C (M x N) = alpha * A (M x K) * B (K x N) + beta * C, column-major, in tiles
// of 64 rows x NT columns.  NT = 32 for FP64, whose rate bounds it: a 32-wide
// node then computes no padding (27,648 rows, 32 x 32: 113 -> 61 us).
template <typename T, int NT>
__global__ void __launch_bounds__(256) gemm_nn(int64_t M, int N, int K, T alpha, const T* __restrict__ A,
                                               int64_t lda, const T* __restrict__ B, int64_t ldb, T beta, T* C,
                                               int64_t ldc) {
    pdl_begin();
    __shared__ T As[kKt][kTile + 1];
    __shared__ T Bs[kKt][NT + 1];
    constexpr int V = NT / 16;             // columns per thread
    constexpr int LB = kKt * NT / 256;     // elements of B loaded per thread
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int64_t i0 = (int64_t)blockIdx.x * kTile;
    const int j0 = blockIdx.y * NT;
    T acc[4][V] = {};
    // the next k step's elements are loaded into registers while the current
    // one is multiplied out of shared memory
    T ra[4], rb[LB];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + 256 * e;
            {  // A tile: kKt columns of 64 contiguous rows
                const int row = idx % kTile, kk = idx / kTile;
                const int k = k0 + kk;
                ra[e] = (k < K && i0 + row < M) ? A[i0 + row + (int64_t)k * lda] : T(0);
            }
            if (e < LB) {  // B tile: NT columns of kKt contiguous k
                const int kk = idx % kKt, col = idx / kKt;
                const int k = k0 + kk;
                rb[e < LB ? e : 0] = (k < K && j0 + col < N) ? B[k + (int64_t)(j0 + col) * ldb] : T(0);
            }
        }
    };
    if (K > 0) fetch(0);
    for (int k0 = 0; k0 < K; k0 += kKt) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + 256 * e;
            As[(idx / kTile)][idx % kTile] = ra[e];
            if (e < LB) Bs[idx % kKt][idx / kKt] = rb[e < LB ? e : 0];
        }
        __syncthreads();
        if (k0 + kKt < K) fetch(k0 + kKt);
#pragma unroll
        for (int kk = 0; kk < kKt; ++kk) {
            T a[4], b[V];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                a[u] = As[kk][ty + 16 * u];
                if (u < V) b[u < V ? u : 0] = Bs[kk][tx * V + (u < V ? u : 0)];
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < V; ++v) acc[u][v] += a[u] * b[v];
        }
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int64_t i = i0 + ty + 16 * u;
            const int j = j0 + tx * V + v;
            if (i < M && j < N) {
                T* c = C + i + (int64_t)j * ldc;
                *c = alpha * acc[u][v] + beta * *c;
            }
        }
}

template <typename T>
__global__ void axpy_block(int M, int N, const T* __restrict__ X, int64_t ldx, T* Y, int64_t ldy) {
    pdl_begin();
    const int64_t total = (int64_t)M * N;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e % M), j = (int)(e / M);
        Y[i + (int64_t)j * ldy] += X[i + (int64_t)j * ldx];
    }
}

int panel_of(const tsqr_opts& o) { return o.panel > 0 ? o.panel : 32; }

int64_t split_of(int64_t n, int nb) {
    int64_t n1 = (n / 2) / nb * nb;
    return std::max<int64_t>(n1, nb);
}

struct GemmPlan {
    int nz;
    int64_t kchunk;
};

// At most most_nz chunks (the room for partial sums).
GemmPlan tn_plan(int64_t M, int64_t N, int64_t K, int64_t most_nz = INT32_MAX) {
    // two CTAs per SM of GB300's 152 (the workspace query uses the same plan),
    // chunks of 64 rows or more
    const int64_t tiles = ceil_div(M, kTnTile) * ceil_div(N, kTnTile);
    int64_t nz = std::max<int64_t>(1, (2 * 152) / tiles);
    nz = std::min<int64_t>(nz, std::max<int64_t>(1, ceil_div(K, 64)));
    nz = std::min<int64_t>(nz, most_nz);
    int64_t kchunk = round_up(ceil_div(K, nz), kKt);
    nz = ceil_div(K, kchunk);
    return {(int)nz, kchunk};
}

// Bytes of partial sums proj_tn takes for an n1 x n2 projection over K rows.
template <typename T>
size_t proj_tn_part_bytes(int64_t n1, int64_t n2, int64_t K) {
    if (std::is_same<T, float>::value) return tn_fused_plan(n1, n2, K).part_bytes();
    return (size_t)tn_plan(n1, n2, K).nz * n1 * n2 * sizeof(T);
}

// Bytes it can do with: FP64 takes fewer and longer chunks where the room is
// short.  The least is what the query asked for with 64-wide tiles in chunks
// of 256 rows, so that a buffer of that size stays enough.
template <typename T>
size_t proj_tn_part_least(int64_t n1, int64_t n2, int64_t K) {
    const size_t want = proj_tn_part_bytes<T>(n1, n2, K);
    if (std::is_same<T, float>::value) return want;
    const int64_t nz = std::min<int64_t>(ceil_div(2 * 152, ceil_div(n1, 64) * ceil_div(n2, 64)), ceil_div(K, 256));
    return std::min(want, (size_t)(ceil_div(K, round_up(ceil_div(K, nz), kKt)) * n1 * n2) * sizeof(T));
}

// Room for partial sums in a workspace of `have` bytes that needs `least`
// with `part_least` of them: more where there is more, up to `want`.
size_t part_room(size_t have, size_t least, size_t part_least, size_t want) {
    return std::min(want, part_least + (have - least) / 256 * 256);
}

// Workspace layout: [status word | tsqr region | partial sums | reorth temp].
// The precision form (FP32, TF32X3) sizes the TSQR region for the
// precision-form TSQR and the partial sums for the tcgen05 split-K GEMM.
struct QrWs {
    size_t err_bytes = kPHeader, tsqr_bytes = 0, part_bytes = 0, part_least = 0, tmp_bytes = 0;
    size_t total() const { return err_bytes + tsqr_bytes + part_bytes + tmp_bytes; }
    size_t least() const { return total() - part_bytes + part_least; }
};

// The tensor-core forms (FP32 only): TF32X3, or BF16X3, whose GEMMs use
// BF16 hi/lo splits (the TSQR panels stay on the TF32x3 tensor-core form).
template <typename T>
bool use_tc(const tsqr_opts& o) {
    return sizeof(T) == 4 && (o.precision == TSQR_PRECISION_TF32X3 || o.precision == TSQR_PRECISION_BF16X3);
}
template <typename T>
bool use_bf16(const tsqr_opts& o) {
    return sizeof(T) == 4 && o.precision == TSQR_PRECISION_BF16X3;
}

// The projection R12 = A1^T A2 runs on the tensor cores only when both sides
// are at least 256 wide.  us at 131,072 rows, tensor cores with their sum of
// partials / CUDA cores: 256 x 256 110 / 470, 128 x 128 44 / 119.  The narrower
// one stays in FP32 for its error: a 256-column QR of 32,768 rows has 5e-8 in
// R, 2e-7 with the tensor-core product.
bool tc_projection(bool tc, int64_t n1, int64_t n2) { return tc && n1 >= 256 && n2 >= 256; }

template <typename T>
void qr_ws_walk(int64_t m, int64_t n, int nb, bool reorth, bool tc, QrWs* w) {
    if (n <= nb) {
        const size_t b = tc ? tsqr_precision_workspace(m, n) : tsqr_plain_workspace<T>(m, n);
        w->tsqr_bytes = std::max(w->tsqr_bytes, (size_t)round_up((int64_t)b, 256));
        return;
    }
    const int64_t n1 = split_of(n, nb), n2 = n - n1;
    const size_t pb = tc_projection(tc, n1, n2) ? (size_t)tc_tn_splits(n1, n2, m) * n1 * n2 * sizeof(T)
                                                : proj_tn_part_bytes<T>(n1, n2, m);
    const size_t pl = tc_projection(tc, n1, n2) ? pb : proj_tn_part_least<T>(n1, n2, m);
    w->part_bytes = std::max(w->part_bytes, (size_t)round_up((int64_t)pb, 256));
    w->part_least = std::max(w->part_least, (size_t)round_up((int64_t)pl, 256));
    if (reorth) w->tmp_bytes = std::max(w->tmp_bytes, (size_t)round_up(n1 * n2 * (int64_t)sizeof(T), 256));
    qr_ws_walk<T>(m, n1, nb, reorth, tc, w);
    qr_ws_walk<T>(m, n2, nb, reorth, tc, w);
}

// C (n1 x n2, ldc) = A1^T A2 (+ beta C) on the tensor cores (FP32 only).
template <typename T>
void proj_tn_tc(int64_t m, int64_t n1, int64_t n2, const T* A1, const T* A2, int64_t lda, T* P, T* C, int64_t ldc,
                T beta, int* err, cudaStream_t s, bool bf16) {
    if constexpr (std::is_same<T, float>::value) {
        const int nz = tc_gemm_tn((int)n1, (int)n2, m, A1, lda, A2, lda, P, err, s, bf16);
        log_launch(kTagTc + 100, s);
        launch_pdl(reduce_partials<T>, dim3(reduce_blocks(n1 * n2)), dim3(256), 0, s, (int)n1, (int)n2, nz,
                   (const T*)P, T(1), beta, C, ldc);
        log_launch(kTagReduce, s);
    }
}

// A2 (m x n2) -= A1 (m x n1) X (n1 x n2, ldx) in FP32 on CUDA cores
// (gemm_nn_fused, n1 <= 256).
void update_nn_fused(int64_t m, int64_t n1, int64_t n2, const float* A1, int64_t lda, const float* X, int64_t ldx,
                     float* A2, cudaStream_t s) {
    NnFusedArgs a;
    a.m = m;
    a.n1 = (int)n1;
    a.n2 = (int)n2;
    a.A1 = A1;
    a.A2 = A2;
    a.lda = lda;
    a.X = X;
    a.ldx = ldx;
    a.alpha = -1.f;
    const int tj = (int)ceil_div(n2, 32);
    const int64_t resident = 2 * (int64_t)device_sm_count();
    const int gx = (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(m, kNR), ceil_div(resident, tj)));
    const size_t smem = nn_fused_smem((int)n1);
    static PerDeviceOnce attr;
    attr.run([] {
        const int mx = (int)nn_fused_smem(kNMaxK);
        cudaFuncSetAttribute(gemm_nn_fused<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
        cudaFuncSetAttribute(gemm_nn_fused<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx);
    });
    const bool vec = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A1) % 16 == 0 &&
                     reinterpret_cast<uintptr_t>(A2) % 16 == 0;
    if (vec)
        launch_pdl(gemm_nn_fused<true>, dim3((unsigned)gx, (unsigned)tj), dim3(256), smem, s, a);
    else
        launch_pdl(gemm_nn_fused<false>, dim3((unsigned)gx, (unsigned)tj), dim3(256), smem, s, a);
    log_launch(kTagGemmNN, s);
}

// The tensor-core forms' updates run on the tcgen05 GEMM only when the panel
// is wider than kNnTcMin.  131,072 x 512, TF32x3, reorthogonalised, with the
// CUDA-core kernel up to 128 columns 4.531 ms, up to 64 columns 4.386 ms (both
// with a slower tcgen05 update than now).  Up to 64 columns the product stays
// in FP32.
constexpr int64_t kNnTcMin = 64;

// A2 (m x n2) -= A1 (m x n1) X (n1 x n2) in a tensor-core form (FP32 only).
template <typename T>
void update_nn_tc(int64_t m, int64_t n1, int64_t n2, const T* A1, int64_t lda, const T* X, int64_t ldx, T* A2,
                  int* err, cudaStream_t s, bool bf16) {
    if constexpr (std::is_same<T, float>::value) {
        if (n1 <= kNnTcMin) return update_nn_fused(m, n1, n2, A1, lda, X, ldx, A2, s);
        tc_gemm_nn(m, (int)n2, (int)n1, -1.f, A1, lda, X, ldx, A2, lda, err, s, bf16);
        log_launch(kTagTc + 101, s);
    }
}

// A2 (m x n2) -= A1 (m x n1) X (n1 x n2, ldx) on CUDA cores, plain form.
template <typename T>
void update_nn(int64_t m, int64_t n1, int64_t n2, const T* A1, int64_t lda, const T* X, int64_t ldx, T* A2,
               cudaStream_t s) {
    if constexpr (std::is_same<T, float>::value) {
        if (n1 <= kNMaxK) return update_nn_fused(m, n1, n2, A1, lda, X, ldx, A2, s);
    }
    constexpr int NT = sizeof(T) == 8 ? 32 : 64;
    dim3 g((unsigned)ceil_div(m, kTile), (unsigned)ceil_div(n2, NT));
    launch_pdl(gemm_nn<T, NT>, g, dim3(256), 0, s, m, (int)n2, (int)n1, T(-1), A1, lda, X, ldx, T(1), A2, lda);
    log_launch(kTagGemmNN, s);
}

// C (n1 x n2, ldc) = A1^T A2 (+ beta C) on CUDA cores.  FP32: one launch of
// gemm_tn_fused (cnt: the workspace's counter words, zero between
// launches), which adds the product to D as well if it is given; FP64: split-K
// partials (part_bytes at P), then their sum (D must be null).
template <typename T>
tsqr_status proj_tn(int64_t m, int64_t n1, int64_t n2, const T* A1, const T* A2, int64_t lda, T* P, size_t part_bytes,
                    T* C, int64_t ldc, T beta, int* cnt, int* err, cudaStream_t s, T* D = nullptr, int64_t ldd = 0) {
    if constexpr (std::is_same<T, float>::value) {
        const TnFusedPlan fp = tn_fused_plan(n1, n2, m);
        TnFusedArgs a;
        a.n1 = (int)n1;
        a.n2 = (int)n2;
        a.K = m;
        a.A = A1;
        a.B = A2;
        a.ld = lda;
        a.C = C;
        a.ldc = ldc;
        a.D = D;
        a.ldd = ldd;
        a.alpha = 1.f;
        a.beta = beta;
        a.tiles_i = fp.tiles_i;
        a.S = fp.S;
        a.g = fp.g;
        a.G = fp.G;
        a.kchunk = fp.kchunk;
        a.part = P;
        a.gpart = P + (size_t)fp.ntiles * fp.S * kPT * kPT;
        a.cnt = cnt;
        a.err = err;
        a.tries = wait_tries().load(std::memory_order_relaxed);
        const dim3 g((unsigned)fp.ntiles, (unsigned)fp.S);
        CUtensorMap ta, tb;
        if (m + kPRows <= INT32_MAX && tensor_map_f32(&ta, A1, lda, m, n1, 32, 32, true) &&
            tensor_map_f32(&tb, A2, lda, m, n2, 32, 32, true)) {
            static PerDeviceOnce attr;
            attr.run([] {
                cudaFuncSetAttribute(gemm_tn_tma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPTmaSmem);
            });
            launch_pdl(gemm_tn_tma, g, dim3(256), kPTmaSmem, s, a, ta, tb);
            log_launch(kTagGemmTN, s);
            return TSQR_OK;
        }
        const bool vec = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A1) % 16 == 0 &&
                         reinterpret_cast<uintptr_t>(A2) % 16 == 0;
        if (vec)
            launch_pdl(gemm_tn_fused<true>, g, dim3(256), 0, s, a);
        else
            launch_pdl(gemm_tn_fused<false>, g, dim3(256), 0, s, a);
        log_launch(kTagGemmTN, s);
        return TSQR_OK;
    }
    GemmPlan gp = tn_plan(n1, n2, m, (int64_t)(part_bytes / (sizeof(T) * n1 * n2)));
    dim3 g((unsigned)ceil_div(n1, kTnTile), (unsigned)ceil_div(n2, kTnTile), (unsigned)gp.nz);
    launch_pdl(gemm_tn_partial<T>, g, dim3(256), 0, s, (int)n1, (int)n2, m, A1, lda, A2, lda, P, gp.kchunk);
    log_launch(kTagGemmTN, s);
    launch_pdl(reduce_partials<T>, dim3(reduce_blocks(n1 * n2)), dim3(256), 0, s, (int)n1, (int)n2, gp.nz,
               (const T*)P, T(1), beta, C, ldc);
    log_launch(kTagReduce, s);
    return TSQR_OK;
}


// TSQR of one panel in the call's form, its bounded waits reporting to the
// call's status word.
template <typename T>
tsqr_status panel_tsqr(int64_t m, int64_t n, T* A, int64_t lda, T* R, int64_t ldr, void* work, size_t work_bytes,
                       bool tc, int* status, cudaStream_t s) {
    if constexpr (std::is_same<T, float>::value) {
        if (tc) {
            PrecFlags f;
            f.status = status;
            return tsqr_precision(m, n, A, lda, R, ldr, work, work_bytes, s, f);
        }
    }
    return tsqr_plain<T>(m, n, A, lda, R, ldr, work, work_bytes, s, kPhaseUp | kPhaseDown, status);
}

template <typename T>
tsqr_status qr_rec(int64_t m, int64_t n, T* A, int64_t lda, T* R, int64_t ldr, char* ws, const QrWs& w,
                   const tsqr_opts& o, cudaStream_t s) {
    const int nb = panel_of(o);
    const bool tc = use_tc<T>(o);
    char* tws = ws + w.err_bytes;
    int* err = reinterpret_cast<int*>(ws);
    if (n <= nb) return panel_tsqr<T>(m, n, A, lda, R, ldr, tws, w.tsqr_bytes, tc, err, s);
    const int64_t n1 = split_of(n, nb), n2 = n - n1;
    T* A1 = A;
    T* A2 = A + n1 * lda;
    T* R11 = R;
    T* R12 = R + n1 * ldr;
    T* R22 = R + n1 * ldr + n1;
    int* cnt = err + kPCounters;
    T* P = reinterpret_cast<T*>(tws + w.tsqr_bytes);
    T* tmp = reinterpret_cast<T*>(tws + w.tsqr_bytes + w.part_bytes);
    tsqr_status st = qr_rec<T>(m, n1, A1, lda, R11, ldr, ws, w, o, s);
    if (st != TSQR_OK) return st;
    const bool tcp = tc_projection(tc, n1, n2);
    if (tc) {
        if (tcp)
            proj_tn_tc<T>(m, n1, n2, A1, A2, lda, P, R12, ldr, T(0), err, s, use_bf16<T>(o));
        else
            proj_tn<T>(m, n1, n2, A1, A2, lda, P, w.part_bytes, R12, ldr, T(0), cnt, err, s);
        update_nn_tc<T>(m, n1, n2, A1, lda, R12, ldr, A2, err, s, use_bf16<T>(o));
    } else {
        proj_tn<T>(m, n1, n2, A1, A2, lda, P, w.part_bytes, R12, ldr, T(0), cnt, err, s);
        update_nn<T>(m, n1, n2, A1, lda, R12, ldr, A2, s);
    }
    if (o.reorth) {
        // R12 += tmp: by the projection's own kernel where it sums its
        // partials in one place, else by a launch of its own (3 us)
        T* D = std::is_same<T, float>::value && !tcp ? R12 : nullptr;
        if (tcp)
            proj_tn_tc<T>(m, n1, n2, A1, A2, lda, P, tmp, n1, T(0), err, s, use_bf16<T>(o));
        else
            proj_tn<T>(m, n1, n2, A1, A2, lda, P, w.part_bytes, tmp, n1, T(0), cnt, err, s, D, ldr);
        if (tc)
            update_nn_tc<T>(m, n1, n2, A1, lda, tmp, n1, A2, err, s, use_bf16<T>(o));
        else
            update_nn<T>(m, n1, n2, A1, lda, tmp, n1, A2, s);
        if (!D) {
            int blocks = (int)std::min<int64_t>(ceil_div(n1 * n2, 256), 1024);
            launch_pdl(axpy_block<T>, dim3(blocks), dim3(256), 0, s, (int)n1, (int)n2, (const T*)tmp, (int64_t)n1, R12,
                       ldr);
            log_launch(kTagAxpy, s);
        }
    }
    st = qr_rec<T>(m, n2, A2, lda, R22, ldr, ws, w, o, s);
    if (st != TSQR_OK) return st;
    return cudaGetLastError() == cudaSuccess ? TSQR_OK : TSQR_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// Blocked Householder QR (tsqr_opts.algorithm = TSQR_QR_HOUSEHOLDER): each
// b-column panel is factored by TSQR, its Householder vectors are
// reconstructed from the explicit panel Q (Ballard, Demmel, Grigori,
// Jacquelin, Knight, Nguyen, "Reconstructing Householder vectors from
// tall-skinny QR", 2015): Q_p - [S; 0] = Y U by an LU without pivoting whose
// signs S = -sign(diagonal) keep every pivot at least 1 in magnitude, and
// T = -U S Y_1^-T gives H_p = I - Y T Y^T with H_p[:, :b] = Q_p S.  The
// trailing columns get H_p^T A2 = A2 - Y (T^T (Y^T A2)) (two GEMMs), and Q is
// accumulated backwards, Q = H_1 ... H_P [I; 0], as LAPACK's orgqr does.
// Orthogonality is then independent of the condition number, unlike the
// block Gram-Schmidt recursion of the reference (block_QR.h:72-95).
// ---------------------------------------------------------------------------
constexpr int kHrMax = 32;  // panel width limit of the Householder path

// Reconstruction of one panel, one CTA.  In: the top bw x bw block of the
// panel's explicit Q (at Ap, lda) and its TSQR factor Rp (bw x bw, ldrp).
// Out: the top block rewritten as the unit lower triangular Y_1, U^-1
// (bw x bw, ld bw: its workspace block has b * b elements), T (bw x bw at Tp, ld ldt), R_h = S Rp into Rout (upper
// triangle, ldr), and M = T Y_1^T = -U S, whose diagonal is T's, transposed
// in the strict lower triangle of T's block (which no product reads).
//
// Bound by its chain of 32 pivots.  Lane r of warp w holds row r, columns
// w, w + 8, w + 16, w + 24, so each step is one division in the warp that owns
// the pivot column, one barrier, and a shuffle of the pivot row per column.
// The two triangular inverses run in two warps at once, one column per lane,
// its entries in registers, each finished entry taken out of all later ones
// (the chain is one division and one product per row instead of a sum over the
// rows before it).  32 columns, FP32: 14 us, 43 us with the columns of
// the elimination and of both inverses as serial loops over shared memory.
template <typename T>
__global__ void __launch_bounds__(256) hr_reconstruct(int bw, T* Ap, int64_t lda, const T* Rp, int ldrp, T* Uinv,
                                                      T* Tp, int64_t ldt, T* Rout, int64_t ldr) {
    pdl_begin();
    constexpr int N = kHrMax, CW = N / 8;
    __shared__ T W[N][N + 1];  // LU: U on and above, L below the diagonal
    __shared__ __align__(16) T Wt[N][N + 4];  // its transpose
    __shared__ T Li[N][N + 1];  // Y_1^-1 (unit lower)
    __shared__ T lcol[2][N], sgn[N];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    T w[CW];
#pragma unroll
    for (int c = 0; c < CW; ++c) {
        const int j = warp + 8 * c;
        // rows and columns past the panel are those of the identity
        w[c] = (lane < bw && j < bw) ? Ap[lane + (int64_t)j * lda] : T(lane == j);
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (i >= bw) break;
        if (warp == i % 8) {
            T& wi = w[i / 8];
            const T d = __shfl_sync(kFull, wi, i);
            const T s = d >= T(0) ? T(-1) : T(1);
            const T piv = d - s;
            if (lane == i) {
                wi = piv;
                sgn[i] = s;
            }
            if (lane > i) wi = wi / piv;
            lcol[i & 1][lane] = lane > i ? wi : T(0);
        }
        __syncthreads();
        const T l = lcol[i & 1][lane];
#pragma unroll
        for (int c = 0; c < CW; ++c) {
            const T u = __shfl_sync(kFull, w[c], i);
            if (warp + 8 * c > i) w[c] = fma(-l, u, w[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < CW; ++c) {
        W[lane][warp + 8 * c] = w[c];
        Wt[warp + 8 * c][lane] = w[c];
    }
    __syncthreads();
    if (warp == 0) {  // column lane of U^-1
        T x[N];
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = T(i == lane);
#pragma unroll
        for (int i = N - 1; i >= 0; --i) {
            x[i] = x[i] / Wt[i][i];
#pragma unroll
            for (int k = 0; k < i; ++k)
                if (i <= lane) x[k] = fma(-Wt[i][k], x[i], x[k]);
            if (i < bw && lane < bw) Uinv[i + lane * bw] = x[i];
        }
        return;
    }
    if (warp == 1) {  // column lane of Y_1^-1
        T x[N];
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = T(i == lane);
#pragma unroll
        for (int i = 0; i < N; ++i) {
#pragma unroll
            for (int k = i + 1; k < N; ++k)
                if (i >= lane) x[k] = fma(-Wt[i][k], x[i], x[k]);
            Li[i][lane] = x[i];
        }
    } else {
        for (int e = tid - 64; e < bw * bw; e += 192) {
            const int i = e % bw, j = e / bw;
            Ap[i + (int64_t)j * lda] = (i > j) ? W[i][j] : ((i == j) ? T(1) : T(0));
            if (i <= j) Rout[i + (int64_t)j * ldr] = sgn[i] * Rp[i + j * ldrp];
            if (i > j) Tp[i + (int64_t)j * ldt] = -W[j][i] * sgn[i];  // M(j, i)
        }
    }
    asm volatile("bar.sync 1, 224;" ::: "memory");  // warps 1 to 7
    // T = -U S Y_1^-T: sum over i <= k <= j of U(i,k) s_k Y_1^-1(j,k)
    for (int j = warp - 1; j < bw; j += 7) {
        const int i = lane;
        T t = T(0);
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (i <= k && k <= j) t -= W[i][k] * sgn[k] * Li[j][k];
        if (i <= j) Tp[i + (int64_t)j * ldt] = t;
    }
}

// Y <- Y U (kUinv: U = U^-1 of the panel, in place for the rows below a panel's top
// block) or [I; 0] - Y M (the panel's columns of Q; M as hr_reconstruct leaves
// it in T's block), U and M upper triangular, one thread per row.  The matrix
// is read as 16-byte rows of four columns for kUpperRows rows at once: 144
// shared-memory broadcasts for two rows where single values took 528 for one.
// A row is in registers before its first column is overwritten.  65,536 x 32 in
// FP32: U 7.0 us, M 8.2 us; 12 us, and 15 us with M's zeros multiplied, before.
template <typename T>
constexpr int kUpperRows = sizeof(T) == 4 ? 2 : 1;  // rows per thread

template <typename T, bool kUinv>
__global__ void __launch_bounds__(128) rows_times_upper(int64_t rows, int bw, T* Y, int64_t lda, const T* Up,
                                                        int64_t ldu) {
    pdl_begin();
    constexpr int R = kUpperRows<T>;
    __shared__ __align__(16) T U[kHrMax][kHrMax];
    const int64_t r0 = blockIdx.x * (int64_t)(128 * R) + threadIdx.x;
    T q[R][kHrMax];
#pragma unroll
    for (int h = 0; h < R; ++h)
#pragma unroll
        for (int k = 0; k < kHrMax; ++k)
            q[h][k] = (k < bw && r0 + 128 * h < rows) ? Y[r0 + 128 * h + k * lda] : T(0);
#pragma unroll
    for (int e = threadIdx.x; e < kHrMax * kHrMax; e += 128) {
        const int i = e % kHrMax, j = e / kHrMax;
        T u = T(0);
        if (i <= j && j < bw) u = kUinv ? Up[i + j * ldu] : -Up[j + i * ldu];
        U[i][j] = u;
    }
    __syncthreads();
#pragma unroll
    for (int c0 = 0; c0 < kHrMax; c0 += 4) {
        T y[R][4];
#pragma unroll
        for (int h = 0; h < R; ++h)
#pragma unroll
            for (int c = 0; c < 4; ++c) y[h][c] = T(!kUinv && r0 + 128 * h == c0 + c);
#pragma unroll
        for (int k = 0; k < c0 + 4; ++k) {
            T u[4];
            if constexpr (sizeof(T) == 4) {
                const float4 v = *reinterpret_cast<const float4*>(&U[k][c0]);
                u[0] = v.x, u[1] = v.y, u[2] = v.z, u[3] = v.w;
            } else {
                const double2 v0 = *reinterpret_cast<const double2*>(&U[k][c0]);
                const double2 v1 = *reinterpret_cast<const double2*>(&U[k][c0 + 2]);
                u[0] = v0.x, u[1] = v0.y, u[2] = v1.x, u[3] = v1.y;
            }
#pragma unroll
            for (int h = 0; h < R; ++h)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (k <= c0 + c) y[h][c] = fma(q[h][k], u[c], y[h][c]);
        }
#pragma unroll
        for (int h = 0; h < R; ++h)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (c0 + c < bw && r0 + 128 * h < rows) Y[r0 + 128 * h + (c0 + c) * lda] = y[h][c];
    }
}

// Products with an upper triangular U (ld ldu):
//   kind 0: X = alpha U^T W   (p x q; U is p x p)
//   kind 1: X = alpha U W     (p x q; U is p x p)
//   kind 2: X = alpha W U     (p x q; U is q x q)
// One CTA per 16 x 16 outputs, one output per thread; 32 rows of the inner
// dimension per step go through shared memory, the next step's loads in
// flight under the current one's products.  Small grids and few operations, so the
// time is the chain of steps.  FP32, 32 / 64 / 128 columns: 3.1 / 3.9 /
// 5.0 us; one serial loop over global memory per output 6 / 8 / 15 us (13 and
// 24 us at kind 2).
template <typename T, int KIND>
__global__ void __launch_bounds__(256) tri_mul(int p, int q, const T* U, int64_t ldu, const T* W, int64_t ldw,
                                               T alpha, T* X, int64_t ldx) {
    pdl_begin();
    constexpr int E = 16, K = 32;
    __shared__ T Ls[K][E + 1], Rs[K][E + 1];  // left(i, k) and right(k, c) by inner index
    const int tid = threadIdx.x;
    const int i0 = blockIdx.x * E, c0 = blockIdx.y * E;
    const int ti = tid % E, tc = tid / E;
    // the part of the inner dimension where the triangle is not zero
    const int kb = KIND == 1 ? i0 : 0;
    const int ke = KIND == 0 ? min(p, i0 + E) : (KIND == 1 ? p : min(q, c0 + E));
    T l[2], r[2];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            // consecutive threads on consecutive rows of a column
            const bool kfirst_l = KIND == 0;
            const int el = tid + 256 * h;
            const int lk = k0 + (kfirst_l ? el % K : el / E), li = i0 + (kfirst_l ? el / K : el % E);
            const int rk = k0 + el % K, rc = c0 + el / K;
            const bool lin = lk < ke && li < p, rin = rk < ke && rc < q;
            if (KIND == 0) l[h] = lin && lk <= li ? U[lk + (int64_t)li * ldu] : T(0);
            if (KIND == 1) l[h] = lin && lk >= li ? U[li + (int64_t)lk * ldu] : T(0);
            if (KIND == 2) l[h] = lin ? W[li + (int64_t)lk * ldw] : T(0);
            if (KIND == 2)
                r[h] = rin && rk <= rc ? U[rk + (int64_t)rc * ldu] : T(0);
            else
                r[h] = rin ? W[rk + (int64_t)rc * ldw] : T(0);
        }
    };
    T x = T(0);
    fetch(kb);
    for (int k0 = kb; k0 < ke; k0 += K) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int el = tid + 256 * h;
            Ls[KIND == 0 ? el % K : el / E][KIND == 0 ? el / K : el % E] = l[h];
            Rs[el % K][el / K] = r[h];
        }
        __syncthreads();
        if (k0 + K < ke) fetch(k0 + K);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int d = k0 + k - (KIND == 2 ? c0 + tc : i0 + ti);
            if (KIND == 1 ? d >= 0 : d <= 0) x = fma(Ls[k][ti], Rs[k][tc], x);
        }
        __syncthreads();
    }
    if (i0 + ti < p && c0 + tc < q) X[i0 + ti + (int64_t)(c0 + tc) * ldx] = alpha * x;
}

// R12 (n1 x n2) from the top rows of a block into R, zeros left in its place:
// Y of the block (leaf Y's with zeros above their unit diagonals) stays clean
// for every later product.
template <typename T>
__global__ void __launch_bounds__(256) move_block(int n1, int64_t total, T* A, int64_t lda, T* R, int64_t ldr) {
    pdl_begin();
    const int64_t e = blockIdx.x * (int64_t)256 + threadIdx.x;
    if (e >= total) return;
    const int64_t i = e % n1, j = e / n1;
    R[i + j * ldr] = A[i + j * lda];
    A[i + j * lda] = T(0);
}

// The Householder path is recursive, like the block Gram-Schmidt one: the
// left half is factored, H_1^T is applied to the right half with one GEMM
// pair of inner dimension n1, the right half's lower rows are factored, and
// the two compact-WY factors combine, T = [T1, -T1 (Y1^T Y2) T2; 0, T2].  Q
// is formed the same way backwards.  Every large product is a GEMM of inner
// dimension >= the panel width, so the tensor-core form applies to it as to
// block Gram-Schmidt.  Leaves (n <= panel) are TSQR + reconstruction.
//
// Workspace: [status word | leaf TSQR | split-K partials | Rp and U^-1 of a
// leaf | W, X (n1 x n2 each) | T of the whole matrix (n x n)].
struct HqrWs {
    size_t err = kPHeader, tsqr = 0, part = 0, part_least = 0, small = 0, wx = 0, tfull = 0;
    size_t total() const { return err + tsqr + part + small + wx + tfull; }
    size_t least() const { return total() - part + part_least; }
};

template <typename T>
void hqr_ws_walk(int64_t m, int64_t n, int b, bool tc, HqrWs* w) {
    if (n <= b) {
        const size_t tb = tc ? tsqr_precision_workspace(m, n) : tsqr_plain_workspace<T>(m, n);
        w->tsqr = std::max(w->tsqr, (size_t)round_up((int64_t)tb, 256));
        return;
    }
    const int64_t n1 = split_of(n, b), n2 = n - n1;
    for (int64_t K : {m, m - n1}) {
        const size_t pb = tc_projection(tc, n1, n2) ? (size_t)tc_tn_splits(n1, n2, K) * n1 * n2 * sizeof(T)
                                                    : proj_tn_part_bytes<T>(n1, n2, K);
        const size_t pl = tc_projection(tc, n1, n2) ? pb : proj_tn_part_least<T>(n1, n2, K);
        w->part = std::max(w->part, (size_t)round_up((int64_t)pb, 256));
        w->part_least = std::max(w->part_least, (size_t)round_up((int64_t)pl, 256));
    }
    w->wx = std::max(w->wx, 2 * (size_t)round_up(n1 * n2 * (int64_t)sizeof(T), 256));
    hqr_ws_walk<T>(m, n1, b, tc, w);
    hqr_ws_walk<T>(m - n1, n2, b, tc, w);
}

template <typename T>
HqrWs hqr_ws(int64_t m, int64_t n, int b, bool tc) {
    HqrWs w;
    hqr_ws_walk<T>(m, n, b, tc, &w);
    w.small = 2 * (size_t)round_up((int64_t)(b * b * sizeof(T)), 256);
    w.tfull = (size_t)round_up(n * n * (int64_t)sizeof(T), 256);
    return w;
}

template <typename T>
struct HqrCtx {
    int64_t lda, ldr, ldt;
    char* tws;
    size_t tsqr_bytes, part_bytes;
    T *part, *Rp, *Uinv, *W, *X;
    int* err;
    bool tc;
    bool bf16 = false;  // BF16x3 tensor-core GEMMs
    int b;
    cudaStream_t s;
};

// X = alpha times the product of an upper triangular U with W, see tri_mul
template <typename T, int KIND>
void hqr_tri(const HqrCtx<T>& c, int64_t p, int64_t q, const T* U, const T* W, T alpha, T* X, int64_t ldx) {
    launch_pdl(tri_mul<T, KIND>, dim3((unsigned)ceil_div(p, 16), (unsigned)ceil_div(q, 16)), dim3(256), 0, c.s, (int)p,
               (int)q, U, c.ldt, W, p, alpha, X, ldx);
    log_launch(kTagHouse + 2, c.s);
}

// C (n1 x n2, ld n1) = A1^T A2 over m rows (A1, A2 share lda)
template <typename T>
void hqr_tn(const HqrCtx<T>& c, int64_t m, int64_t n1, int64_t n2, const T* A1, const T* A2, T* C) {
    if (tc_projection(c.tc, n1, n2))
        proj_tn_tc<T>(m, n1, n2, A1, A2, c.lda, c.part, C, n1, T(0), c.err, c.s, c.bf16);
    else
        proj_tn<T>(m, n1, n2, A1, A2, c.lda, c.part, c.part_bytes, C, n1, T(0), c.err + kPCounters, c.err, c.s);
}

// A2 (m x n2) -= Y (m x n1) X (n1 x n2, ld n1)
template <typename T>
void hqr_nn(const HqrCtx<T>& c, int64_t m, int64_t n1, int64_t n2, const T* Y, const T* X, T* A2) {
    if (c.tc) {
        update_nn_tc<T>(m, n1, n2, Y, c.lda, X, n1, A2, c.err, c.s, c.bf16);
    } else {
        update_nn<T>(m, n1, n2, Y, c.lda, X, n1, A2, c.s);
    }
}

// Factor the m x n block A (rows and columns from its own origin): Y below
// its diagonal, R into Rb, T into Tb (ld ldt).
template <typename T>
tsqr_status hqr_factor(const HqrCtx<T>& c, int64_t m, int64_t n, T* A, T* Rb, T* Tb) {
    if (n <= c.b) {
        tsqr_status st = panel_tsqr<T>(m, n, A, c.lda, c.Rp, n, c.tws, c.tsqr_bytes, c.tc, c.err, c.s);
        if (st != TSQR_OK) return st;
        launch_pdl(hr_reconstruct<T>, dim3(1), dim3(256), 0, c.s, (int)n, A, c.lda, c.Rp, (int)n, c.Uinv, Tb, c.ldt, Rb,
                   c.ldr);
        log_launch(kTagHouse, c.s);
        if (m > n) {
            launch_pdl(rows_times_upper<T, true>, dim3((unsigned)ceil_div(m - n, 128 * kUpperRows<T>)), dim3(128), 0,
                       c.s, m - n, (int)n, A + n, c.lda, c.Uinv, n);
            log_launch(kTagHouse + 1, c.s);
        }
        return TSQR_OK;
    }
    const int64_t n1 = split_of(n, c.b), n2 = n - n1;
    T* A2 = A + n1 * c.lda;
    tsqr_status st = hqr_factor<T>(c, m, n1, A, Rb, Tb);
    if (st != TSQR_OK) return st;
    // A2 <- H_1^T A2 = A2 - Y1 (T1^T (Y1^T A2))
    hqr_tn<T>(c, m, n1, n2, A, A2, c.W);
    hqr_tri<T, 0>(c, n1, n2, Tb, c.W, T(1), c.X, n1);
    hqr_nn<T>(c, m, n1, n2, A, c.X, A2);
    launch_pdl(move_block<T>, dim3((unsigned)ceil_div(n1 * n2, 256)), dim3(256), 0, c.s, (int)n1, n1 * n2, A2, c.lda,
               Rb + n1 * c.ldr, c.ldr);
    log_launch(kTagHouse + 2, c.s);
    T* Tb2 = Tb + n1 + n1 * c.ldt;
    st = hqr_factor<T>(c, m - n1, n2, A2 + n1, Rb + n1 + n1 * c.ldr, Tb2);
    if (st != TSQR_OK) return st;
    // T12 = -T1 (Y1^T Y2) T2, Y2 living in rows n1.. of the block
    hqr_tn<T>(c, m - n1, n1, n2, A + n1, A2 + n1, c.W);
    hqr_tri<T, 2>(c, n1, n2, Tb2, c.W, T(1), c.X, n1);
    hqr_tri<T, 1>(c, n1, n2, Tb, c.X, T(-1), Tb + n1 * c.ldt, c.ldt);
    return cudaGetLastError() == cudaSuccess ? TSQR_OK : TSQR_ERR_CUDA;
}

// Q of the m x n block from its Y (in A) and T (Tb): Q = H [I; 0], in place.
template <typename T>
tsqr_status hqr_form_q(const HqrCtx<T>& c, int64_t m, int64_t n, T* A, const T* Tb) {
    if (n <= c.b) {
        launch_pdl(rows_times_upper<T, false>, dim3((unsigned)ceil_div(m, 128 * kUpperRows<T>)), dim3(128), 0, c.s, m, (int)n, A, c.lda, Tb,
                   c.ldt);
        log_launch(kTagHouse + 3, c.s);
        return cudaGetLastError() == cudaSuccess ? TSQR_OK : TSQR_ERR_CUDA;
    }
    const int64_t n1 = split_of(n, c.b), n2 = n - n1;
    T* A2 = A + n1 * c.lda;
    // right half first: Q2 = H_2 [I; 0] in rows n1.., zeros above it
    tsqr_status st = hqr_form_q<T>(c, m - n1, n2, A2 + n1, Tb + n1 + n1 * c.ldt);
    if (st != TSQR_OK) return st;
    if (cudaMemset2DAsync(A2, c.lda * sizeof(T), 0, n1 * sizeof(T), n2, c.s) != cudaSuccess) return TSQR_ERR_CUDA;
    // then H_1 applied to it: A2 - Y1 (T1 (Y1^T A2))
    hqr_tn<T>(c, m, n1, n2, A, A2, c.W);
    hqr_tri<T, 1>(c, n1, n2, Tb, c.W, T(1), c.X, n1);
    hqr_nn<T>(c, m, n1, n2, A, c.X, A2);
    // the left half last: its Y1 was needed above
    return hqr_form_q<T>(c, m, n1, A, Tb);
}

template <typename T>
tsqr_status hqr_run(int64_t m, int64_t n, T* A, int64_t lda, T* R, int64_t ldr, void* work, size_t work_bytes,
                    const tsqr_opts& o, cudaStream_t s) {
    const int b = panel_of(o);
    if (b > kHrMax) return TSQR_ERR_UNSUPPORTED;
    const bool tc = use_tc<T>(o);
    HqrWs w = hqr_ws<T>(m, n, b, tc);
    if (work == nullptr || work_bytes < w.least()) return TSQR_ERR_WORKSPACE;
    w.part = part_room(work_bytes, w.least(), w.part_least, w.part);
    char* base = static_cast<char*>(work);
    HqrCtx<T> c;
    c.lda = lda;
    c.ldr = ldr;
    c.ldt = n;
    c.err = reinterpret_cast<int*>(base);
    c.tws = base + w.err;
    c.tsqr_bytes = w.tsqr;
    c.part = reinterpret_cast<T*>(c.tws + w.tsqr);
    c.part_bytes = w.part;
    const size_t bb = (size_t)round_up((int64_t)(b * b * sizeof(T)), 256);
    char* sm = c.tws + w.tsqr + w.part;
    c.Rp = reinterpret_cast<T*>(sm);
    c.Uinv = reinterpret_cast<T*>(sm + bb);
    c.W = reinterpret_cast<T*>(sm + w.small);
    c.X = reinterpret_cast<T*>(sm + w.small + w.wx / 2);
    T* Tfull = reinterpret_cast<T*>(sm + w.small + w.wx);
    c.tc = tc;
    c.bf16 = use_bf16<T>(o);
    c.b = b;
    c.s = s;
    // status word and the projection's counters
    if (cudaMemsetAsync(c.err, 0, kPHeader, s) != cudaSuccess) return TSQR_ERR_CUDA;
    if (cudaMemset2DAsync(R, ldr * sizeof(T), 0, n * sizeof(T), n, s) != cudaSuccess) return TSQR_ERR_CUDA;
    tsqr_status st = hqr_factor<T>(c, m, n, A, R, Tfull);
    if (st != TSQR_OK) return st;
    return hqr_form_q<T>(c, m, n, A, Tfull);
}

}  // namespace

template <typename T>
size_t qr_workspace(int64_t m, int64_t n, const tsqr_opts& o) {
    if (o.algorithm == TSQR_QR_HOUSEHOLDER)
        return panel_of(o) <= kHrMax ? hqr_ws<T>(m, n, panel_of(o), use_tc<T>(o)).total() : 0;
    QrWs w;
    qr_ws_walk<T>(m, n, panel_of(o), o.reorth != 0, use_tc<T>(o), &w);
    return w.total();
}

template <typename T>
tsqr_status qr_run(int64_t m, int64_t n, T* A, int64_t lda, T* R, int64_t ldr, void* work, size_t work_bytes,
                   const tsqr_opts& o, cudaStream_t s) {
    if (o.algorithm == TSQR_QR_HOUSEHOLDER) return hqr_run<T>(m, n, A, lda, R, ldr, work, work_bytes, o, s);
    QrWs w;
    qr_ws_walk<T>(m, n, panel_of(o), o.reorth != 0, use_tc<T>(o), &w);
    if (work == nullptr || work_bytes < w.least()) return TSQR_ERR_WORKSPACE;
    w.part_bytes = part_room(work_bytes, w.least(), w.part_least, w.part_bytes);
    // status word and the projection's counters
    if (cudaMemsetAsync(work, 0, kPHeader, s) != cudaSuccess) return TSQR_ERR_CUDA;
    // zeros below R's diagonal blocks, in one fill for all nodes
    if (n > panel_of(o) && cudaMemset2DAsync(R, ldr * sizeof(T), 0, n * sizeof(T), n, s) != cudaSuccess)
        return TSQR_ERR_CUDA;
    return qr_rec<T>(m, n, A, lda, R, ldr, reinterpret_cast<char*>(work), w, o, s);
}

template size_t qr_workspace<float>(int64_t, int64_t, const tsqr_opts&);
template size_t qr_workspace<double>(int64_t, int64_t, const tsqr_opts&);
template tsqr_status qr_run<float>(int64_t, int64_t, float*, int64_t, float*, int64_t, void*, size_t,
                                   const tsqr_opts&, cudaStream_t);
template tsqr_status qr_run<double>(int64_t, int64_t, double*, int64_t, double*, int64_t, void*, size_t,
                                    const tsqr_opts&, cudaStream_t);

}  // namespace tsqr
