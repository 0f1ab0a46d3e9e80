// tc_nn.cu -- C (M x N) += alpha A (M x K) B (K x N) in TF32x3, A tall, B
// small enough to stay in shared memory as TF32 hi and lo for the whole
// launch (the blocked QR's update A2 -= A1 X, K <= 512).
//
// What bounds the update is memory: 131,072 rows, K = N = 128 read A1 and A2
// and write A2 (201 MB, 30 us), the tensor cores need 13 us for the three
// products.  So nothing but A passes through the step loop, and A is touched
// once on its way to the tensor core: a TMA ring brings it in as it lies in
// memory (32 columns of 128 rows), a thread reads its row (conflict-free, rows
// are contiguous), splits it in registers and stores hi and lo to TMEM, which
// is the A operand of the MMA.  That replaces a rewrite of A into two K-major
// shared-memory tiles and of B into two more on every step.
//
// One persistent CTA per SM, 18 warps with one task each: warps 0-3 and 4-7
// split the even and the odd steps (warp w: rows 32 (w % 4) .. +31, the TMEM
// lanes it may access), warps 8-15 add the finished blocks to C (their part
// of C loaded before they wait for the accumulator), one thread issues the
// copies, one the MMAs.  TMEM, 512 columns: two accumulators of NB, four
// steps of A (32 columns hi, 32 lo).
//
// us, 131,072 rows, this kernel / the one that rewrites A and B on every step:
// 128 x 128 45 / 97, 256 x 256 162 / 288.  At 256 the tiles are 64 wide (B of
// 128 would not stay resident), and the MMAs bound it: 12 of them with N = 64
// take 1200 cycles, the copies and splits of a step 790.
//
// Waits are bounded: a role whose wait gives up sets the status word and ends;
// the others' waits then run out as well.  The issuing threads wait (again
// with a limit) for their copies and MMAs in flight before TMEM is freed.
#include <cuda.h>
#include <cuda_runtime.h>
#include <algorithm>
#include "common.cuh"
#include "internal.h"
#include "tc.cuh"

namespace tsqr {
namespace {

constexpr int kRing = 4;                 // raw steps of A in shared memory
constexpr int kSlots = 4;                // split steps of A in TMEM
constexpr int kRawBytes = 128 * 32 * 4;  // 32 columns of 128 rows
constexpr int kResidentB = 128 * 128;    // K x NB at most: 128 KB as hi and lo
constexpr int kSplitWarps = 8, kEpiWarps = 8;
constexpr int kThreads = 32 * (kSplitWarps + kEpiWarps + 2);

// Shared memory of a launch; at least 120 KB, so that one CTA has the SM (and
// its TMEM) to itself.
size_t nn_smem(int nks, int nb) {
    return std::max<size_t>((size_t)kRing * kRawBytes + 2 * (size_t)nks * nb * 128 + 1024, 120 * 1024);
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(mbar) : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem], issued by one thread.
__device__ __forceinline__ void mma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                            bool accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

// 32 lanes x 32 bits, 8 consecutive columns per thread.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};\n" ::"r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

template <int NB>
__global__ void __launch_bounds__(kThreads, 1)
    tc_nn_kernel(int64_t M, int N, int K, float alpha, const float* __restrict__ B, int64_t ldb, float* C,
                 int64_t ldc, const __grid_constant__ CUtensorMap ta, int* err, int tries) {
    pdl_begin();
    extern __shared__ unsigned char nn_raw[];
    __shared__ unsigned long long full[kRing], empty[kRing], ready[kSlots], done[kSlots], dfull[2], dempty[2];
    __shared__ uint32_t tmem_slot;
    unsigned char* base = nn_raw + ((1024 - (tc::smem_u32(nn_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.x * NB;
    const int nks = (K + 31) / 32;
    const int nblk = (int)((M + 127) / 128);
    // this CTA's blocks: blockIdx.y, + gridDim.y, ...; steps t = (block, 32 columns of A)
    const int myblk = (nblk - 1 - (int)blockIdx.y) / (int)gridDim.y + 1;
    const int T = myblk * nks;
    unsigned char* bhi = base + kRing * kRawBytes;  // per step: NB rows of 32 K, 128-byte swizzle
    unsigned char* blo = bhi + (size_t)nks * NB * 128;
    constexpr uint32_t kACol = 2 * NB;

    auto copy = [&](int t) {
        const uint32_t mb = tc::smem_u32(&full[t % kRing]);
        tc::mbar_arrive_expect_tx(mb, kRawBytes);
        tc::tma_load_2d(tc::smem_u32(base + (t % kRing) * kRawBytes), &ta,
                        (int)(blockIdx.y + (t / nks) * gridDim.y) * 128, 32 * (t % nks), mb);
    };
    if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
    if (tid == kThreads - 64) {  // the thread of the copies
        for (int b = 0; b < kRing; ++b) {
            tc::mbar_init(tc::smem_u32(&full[b]), 1);
            tc::mbar_init(tc::smem_u32(&empty[b]), 4);
        }
        for (int b = 0; b < kSlots; ++b) {
            tc::mbar_init(tc::smem_u32(&ready[b]), 128);
            tc::mbar_init(tc::smem_u32(&done[b]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(tc::smem_u32(&dfull[b]), 1);
            tc::mbar_init(tc::smem_u32(&dempty[b]), 32 * kEpiWarps);
        }
        tc::fence_mbar_init();
        for (int t = 0; t < min(kRing, T); ++t) copy(t);
    }
    __syncwarp();
    // B: consecutive threads on consecutive k of a column, which fill one
    // 128-byte row of the swizzled tile; zeros past K and N
#pragma unroll 16
    for (int e = tid; e < nks * 32 * NB; e += kThreads) {
        const int kl = e & 31, n = (e >> 5) % NB, s = e / (32 * NB), k = 32 * s + kl;
        const float x = (k < K && n0 + n < N) ? B[k + (int64_t)(n0 + n) * ldb] : 0.f;
        const uint32_t off = (uint32_t)((s * NB + n) * 128 + (((kl >> 2) ^ (n & 7)) << 4) + (kl & 3) * 4);
        uint32_t hi, lo;
        tc::split_tf32(x, hi, lo);
        *reinterpret_cast<uint32_t*>(bhi + off) = hi;
        *reinterpret_cast<uint32_t*>(blo + off) = lo;
    }
    tc::fence_smem_to_async();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp < kSplitWarps) {
        const uint32_t row = 32 * (warp & 3) + lane, quad = (uint32_t)(32 * (warp & 3)) << 16;
        bool ok = true;
        for (int t = warp >> 2; t < T && ok; t += 2) {
            const int rb = t % kRing, sl = t % kSlots;
            ok = __all_sync(kFull, tc::mbar_wait(tc::smem_u32(&full[rb]), (uint32_t)(t / kRing) & 1u, tries));
            if (!ok) break;
            const float* src = reinterpret_cast<const float*>(base + rb * kRawBytes) + row;
            float x[32];
#pragma unroll
            for (int k = 0; k < 32; ++k) x[k] = src[128 * k];
            __syncwarp();
            if (lane == 0) mbar_arrive(tc::smem_u32(&empty[rb]));
            if (t >= kSlots) {  // the MMAs that read the slot are done
                ok = __all_sync(kFull, tc::mbar_wait(tc::smem_u32(&done[sl]), (uint32_t)(t / kSlots - 1) & 1u, tries));
                if (!ok) break;
                tc::fence_after_sync();
            }
            const uint32_t dst = tmem + quad + kACol + 64 * sl;
#pragma unroll
            for (int c = 0; c < 32; c += 8) {
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) tc::split_tf32(x[c + e], hi[e], lo[e]);
                tmem_st8(dst + c, hi);
                tmem_st8(dst + 32 + c, lo);
            }
            tmem_st_wait();
            tc::fence_before_sync();
            mbar_arrive(tc::smem_u32(&ready[sl]));
        }
        if (!ok && lane == 0 && err) atomicExch(err, 1);
    } else if (warp < kSplitWarps + kEpiWarps) {
        constexpr int HALF = NB / 2;
        const int cb = ((warp - kSplitWarps) >> 2) * HALF;
        const uint32_t src = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)cb;
        const int ncol = N - n0 - cb;  // columns of this warp inside C (may exceed HALF or be negative)
        bool ok = true;
        for (int j = 0; j < myblk; ++j) {
            const int64_t m = ((int64_t)blockIdx.y + (int64_t)j * gridDim.y) * 128 + 32 * (warp & 3) + lane;
            float* cp = C + m + (int64_t)(n0 + cb) * ldc;
            float c[HALF];
            // Column addresses step by step (all of them at once would spill),
            // rows and columns past the end clamped to the last one, so that
            // the loads are not conditional and stay in flight together.
            int64_t step = ldc;
            asm volatile("" : "+l"(step));
            {
                const float* q = C + (m < M ? m : M - 1) + (int64_t)(n0 + (ncol > 0 ? cb : 0)) * ldc;
#pragma unroll
                for (int e = 0; e < HALF; q += ++e < ncol ? step : 0) c[e] = *q;
            }
            const int b = j & 1;
            ok = __all_sync(kFull, tc::mbar_wait(tc::smem_u32(&dfull[b]), (uint32_t)(j >> 1) & 1u, tries));
            if (!ok) break;
            tc::fence_after_sync();
#pragma unroll
            for (int c8 = 0; c8 < HALF; c8 += 8) {
                float d[8];
                tc::tmem_ld8(src + b * NB + c8, d);
                tc::tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) c[c8 + e] = c[c8 + e] + alpha * d[e];
            }
            tc::fence_before_sync();
            mbar_arrive(tc::smem_u32(&dempty[b]));
            asm volatile("" : "+l"(step));
            float* q = cp;
#pragma unroll
            for (int e = 0; e < HALF; ++e, q += step)
                if (m < M && e < ncol) *q = c[e];
        }
        if (!ok && lane == 0 && err) atomicExch(err, 1);
    } else if (warp == kSplitWarps + kEpiWarps) {
        if (lane == 0) {  // copies
            int t = min(kRing, T);
            for (; t < T; ++t) {
                if (!tc::mbar_wait(tc::smem_u32(&empty[t % kRing]), (uint32_t)(t / kRing - 1) & 1u, tries)) break;
                tc::fence_smem_to_async();
                copy(t);
            }
            if (t < T && err) atomicExch(err, 1);
            for (int q = max(0, t - kRing); q < t; ++q)  // every copy has landed
                (void)tc::mbar_wait(tc::smem_u32(&full[q % kRing]), (uint32_t)(q / kRing) & 1u);
        }
    } else if (lane == 0) {  // MMAs
        constexpr uint32_t idesc = tc::idesc_tf32(128, NB);
        const uint32_t sh = tc::smem_u32(bhi), so = tc::smem_u32(blo);
        int t = 0, j = 0;
        for (int s = 0; t < T; ++t) {
            const int sl = t % kSlots, b = j & 1;
            if (s == 0 && j >= 2 &&
                !tc::mbar_wait(tc::smem_u32(&dempty[b]), (uint32_t)(j / 2 - 1) & 1u, tries))
                break;
            if (!tc::mbar_wait(tc::smem_u32(&ready[sl]), (uint32_t)(t / kSlots) & 1u, tries)) break;
            tc::fence_after_sync();
            const uint32_t d = tmem + b * NB, ah = tmem + kACol + 64 * sl, al = ah + 32;
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                const uint64_t bh = tc::smem_desc_sw128(sh + s * NB * 128 + ks * 32);
                const uint64_t bl = tc::smem_desc_sw128(so + s * NB * 128 + ks * 32);
                mma_tf32_ts(d, ah + 8 * ks, bh, idesc, s > 0 || ks > 0);
                mma_tf32_ts(d, ah + 8 * ks, bl, idesc, true);
                mma_tf32_ts(d, al + 8 * ks, bh, idesc, true);
            }
            tc::mma_commit(tc::smem_u32(&done[sl]));
            if (++s == nks) {
                tc::mma_commit(tc::smem_u32(&dfull[b]));
                s = 0;
                ++j;
            }
        }
        if (t < T && err) atomicExch(err, 1);
        for (int q = max(0, t - kSlots); q < t; ++q)  // every MMA is done
            (void)tc::mbar_wait(tc::smem_u32(&done[q % kSlots]), (uint32_t)(q / kSlots) & 1u);
        // and so is the arrival for every finished block: the warps that add
        // it to C may have given up, and it must not come after the CTA's end
        for (int q = max(0, j - 2); q < j; ++q)
            (void)tc::mbar_wait(tc::smem_u32(&dfull[q & 1]), (uint32_t)(q >> 1) & 1u);
    }
    __syncwarp();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

template <int NB>
void launch(int64_t M, int N, int K, float alpha, const CUtensorMap& ta, const float* B, int64_t ldb, float* C,
            int64_t ldc, int* err, cudaStream_t s) {
    static PerDeviceOnce attr;
    attr.run([] {
        cudaFuncSetAttribute(tc_nn_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)nn_smem(kResidentB / NB / 32, NB));
    });
    const int nks = (K + 31) / 32, ntn = (N + NB - 1) / NB;
    const int64_t nblk = (M + 127) / 128;
    const int gy = (int)std::max<int64_t>(1, std::min<int64_t>(nblk, device_sm_count() / ntn));
    launch_pdl(tc_nn_kernel<NB>, dim3((unsigned)ntn, (unsigned)gy), dim3(kThreads), nn_smem(nks, NB), s, M, N, K,
               alpha, B, ldb, C, ldc, ta, err, wait_tries().load(std::memory_order_relaxed));
}

}  // namespace

// False when A does not meet TMA's rules or B is too large to stay in shared
// memory (the caller then takes another kernel).
bool tc_nn_resident(int64_t M, int N, int K, float alpha, const float* A, int64_t lda, const float* B, int64_t ldb,
                    float* C, int64_t ldc, int* err, cudaStream_t s) {
    const int kp = (K + 31) / 32 * 32;
    CUtensorMap ta;
    if (kp > kResidentB / 32 || M + 128 > INT32_MAX || !tensor_map_f32(&ta, A, lda, M, K, 128, 32, false))
        return false;
    // the widest tile whose B stays resident: A is read and split once per tile
    int nb = N > 64 ? 128 : (N > 32 ? 64 : 32);
    while (nb * kp > kResidentB) nb /= 2;
    if (nb == 128) launch<128>(M, N, K, alpha, ta, B, ldb, C, ldc, err, s);
    if (nb == 64) launch<64>(M, N, K, alpha, ta, B, ldb, C, ldc, err, s);
    if (nb == 32) launch<32>(M, N, K, alpha, ta, B, ldb, C, ldc, err, s);
    return true;
}

}  // namespace tsqr
