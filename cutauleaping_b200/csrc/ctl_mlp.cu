// Surrogate MLP kernels for sm_100a: a tcgen05 GEMM with fused epilogues,
// the Gaussian negative-log-likelihood gradient, bias gradients and Adam.
//
// The surrogate (fitness mode, aresio/cuTauLeaping kernel.cu:365-423 computes
// fitness by full simulation; this build screens candidates first) maps
// (8 log rate constants, t) to per-species mean and log-variance:
//   9 -> 256 -> 256 -> 256 -> 256 -> 2*S_out, SiLU, BF16 weights, FP32 accumulate.
//
// GEMM: C[M][N] = A[M][K] . B[N][K]^T, A and B BF16 row-major with K
// contiguous ("K-major").  One CTA of 128 threads computes a 128 x BN tile
// (BN = N <= 256): all threads stage 128x64 / BNx64 tiles of A and B in the
// canonical no-swizzle K-major shared-memory layout (8-row x 16-byte core
// matrices), one elected thread issues tcgen05.mma (M = 128, N = BN, K = 16)
// into a TMEM accumulator and tcgen05.commit signals a per-stage mbarrier;
// two stages overlap the next tile's loads with the current MMAs.  The
// epilogue reads TMEM with tcgen05.ld (warp w owns lanes 32w..32w+31 = rows).
// Split-K over grid.z serves the weight gradients (K = batch).
// Every mbarrier wait is bounded: on timeout the kernel raises an error flag
// instead of hanging.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <cstdint>
#include <algorithm>
#include <string>

#include "ctl_internal.h"

namespace ctl {
namespace mlp {

constexpr int BM = 128, BK = 64, THREADS = 128;
constexpr uint32_t WAIT_LIMIT = 1u << 24;

struct Gemm {
    const __nv_bfloat16* A;
    const __nv_bfloat16* B;
    int lda, ldb, M, N, K, kt_per_split, epi;
    int bn;                     // columns of C per CTA (N tile, multiple of 16, <= 256)
    const float* bias;          // [N]
    const float* z_in;          // [M][ldz] pre-activations (SiLU gradient)
    int ldz;
    float* out_f32;             // [M][ldo]
    int ldo;
    __nv_bfloat16* out_bf;      // [M][ldob]
    int ldob;
    __nv_bfloat16* out_bfT;     // [N][ldobT]
    int ldobT;
    unsigned* err;
};

// ---- PTX helpers ------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: returns false (and raises *err) after `limit` polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned* err,
                                          uint32_t limit = WAIT_LIMIT) {
    for (uint32_t i = 0; i < limit; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if (i > 32) __nanosleep(64);
    }
    if (err) atomicOr(err, 1u);
    return false;
}

// Warp-uniform roles.  A warp that only issues (bulk copies, MMAs) runs its loop
// with all 32 lanes and lets one elected lane issue: the compiler then keeps
// descriptors and addresses in uniform registers, which these instructions
// read.  Under a lane test instead, every MMA waited for moves into uniform
// registers: 290 cycles per MMA with its barrier work against 180 (M = 128,
// N = 256, K = 16; 135 back to back).
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x / 32), 0); }
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
// The whole warp waits (bounded as mbar_wait); the answer is uniform.
__device__ __forceinline__ bool mbar_wait_u(uint64_t* bar, uint32_t parity, unsigned* err) {
    for (uint32_t i = 0; i < WAIT_LIMIT; i++) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        if (i > 32) __nanosleep(64);
    }
    if (err && (threadIdx.x & 31) == 0) atomicOr(err, 1u);
    return false;
}
__device__ __forceinline__ bool raised(int* flag) { return __any_sync(0xffffffffu, *(volatile int*)flag != 0) != 0; }

__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Shared-memory matrix descriptor, K-major, no swizzle: start address,
// leading byte offset (between the two 8-element K chunks of one MMA) and
// stride byte offset (between 8-row groups), all >> 4; version 1 (sm_100).
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1u << 46;  // descriptor version for tcgen05
    return d;                 // base offset 0, absolute-LBO off, swizzle none (bits 61-63 = 0)
}

// Instruction descriptor: kind::f16, A = B = BF16, D = F32, K-major A and B.
__device__ __forceinline__ uint32_t make_idesc(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

// SiLU through the logistic function written with the hardware tanh:
// sigmoid(z) = 0.5 + 0.5 tanh(z / 2), one MUFU operation per element
// (tanh.approx.f32, relative error about 2^-11, below the BF16 rounding that
// follows).  Training and screening use the same form.
__device__ __forceinline__ float tanh_hw(float x) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x));
    return t;
}
__device__ __forceinline__ float sigm(float z) { return fmaf(0.5f, tanh_hw(0.5f * z), 0.5f); }
// silu(z) = z sigmoid(z) = h tanh(h) + h with h = z / 2: one multiply, one
// MUFU and one FMA per element.
__device__ __forceinline__ float silu(float z) {
    const float h = 0.5f * z;
    return fmaf(h, tanh_hw(h), h);
}
__device__ __forceinline__ float silu_grad(float z) {
    const float s = sigm(z);
    return s * (1.0f + z * (1.0f - s));
}

// Two FP32 values -> two BF16 (round to nearest even) in one conversion.
__device__ __forceinline__ uint32_t pack_bf2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// ---- the GEMM -----------------------------------------------------------------

enum { EPI_ATOMIC_F32 = 0, EPI_BIAS_SILU = 1, EPI_BIAS = 2, EPI_SILU_GRAD = 3, EPI_F32 = 4 };

// Copy a ROWS x 64 BF16 tile (rows r0.., columns k0..k0+63) into the
// canonical layout: chunk (row, kb) of 8 elements at (kb*ROWS/8 + row/8)*128
// + (row%8)*16 bytes.  Consecutive threads take consecutive rows.
__device__ __forceinline__ void stage_tile(uint8_t* dst, const __nv_bfloat16* src, int ld, int r0,
                                           int k0, int rows) {
    const int chunks = rows * (BK / 8);
    for (int c = (int)threadIdx.x; c < chunks; c += THREADS) {
        const int row = c % rows, kb = c / rows;
        const uint4 v = *reinterpret_cast<const uint4*>(src + (size_t)(r0 + row) * ld + k0 + kb * 8);
        *reinterpret_cast<uint4*>(dst + (size_t)(kb * (rows / 8) + row / 8) * 128 + (row % 8) * 16) = v;
    }
}

// The epilogue: warp w reads TMEM lanes 32w..32w+31 (rows m0 + 32w + lane),
// 8 columns at a time, and applies the descriptor's epilogue.
__device__ __forceinline__ void gemm_epilogue(const Gemm& p, uint32_t tmem, int BN, int m0, int n0, int warp,
                                              int lane) {
    const int row = m0 + warp * 32 + lane;
    // A thread holds 8 consecutive columns of its row: it writes them as
    // 16- and 32-byte vectors (one sector per thread) when the row
    // strides allow, instead of eight 4-byte stores to 32 rows at a time.
    const bool vf = (p.ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(p.out_f32) & 15) == 0;
    const bool vb = (p.ldob & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out_bf) & 15) == 0;
    auto store_f32 = [&](int n, const float (&o)[8]) {
        float* dst = p.out_f32 + (size_t)row * p.ldo + n;
        if (vf) {
            reinterpret_cast<float4*>(dst)[0] = make_float4(o[0], o[1], o[2], o[3]);
            reinterpret_cast<float4*>(dst)[1] = make_float4(o[4], o[5], o[6], o[7]);
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) dst[j] = o[j];
        }
    };
    auto store_bf = [&](int n, const float (&o)[8]) {
        __nv_bfloat16* dst = p.out_bf + (size_t)row * p.ldob + n;
        if (vb) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf2(o[0], o[1]), pack_bf2(o[2], o[3]),
                                                        pack_bf2(o[4], o[5]), pack_bf2(o[6], o[7]));
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) dst[j] = __float2bfloat16(o[j]);
        }
        if (p.out_bfT)
#pragma unroll
            for (int j = 0; j < 8; j++) p.out_bfT[(size_t)(n + j) * p.ldobT + row] = __float2bfloat16(o[j]);
    };
    for (int c = 0; c < BN; c += 8) {
        float v[8];
        tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
        const int n = n0 + c;
        if (p.epi == EPI_ATOMIC_F32) {
#pragma unroll
            for (int j = 0; j < 8; j++) atomicAdd(p.out_f32 + (size_t)row * p.ldo + n + j, v[j]);
        } else if (p.epi == EPI_F32) {
            store_f32(n, v);
        } else if (p.epi == EPI_BIAS) {
            float o[8];
#pragma unroll
            for (int j = 0; j < 8; j++) o[j] = v[j] + p.bias[n + j];
            store_f32(n, o);
        } else if (p.epi == EPI_BIAS_SILU) {
            float z[8], h[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                z[j] = v[j] + p.bias[n + j];
                h[j] = silu(z[j]);
            }
            store_f32(n, z);
            store_bf(n, h);
        } else {  // EPI_SILU_GRAD
            float d[8];
#pragma unroll
            for (int j = 0; j < 8; j++) d[j] = v[j] * silu_grad(p.z_in[(size_t)row * p.ldz + n + j]);
            store_bf(n, d);
        }
    }
}

__global__ void __launch_bounds__(THREADS, 1) gemm_kernel(Gemm p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ uint32_t tmem_slot;
    const int BN = p.bn;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int ktiles = p.K / BK;
    const int kt0 = blockIdx.z * p.kt_per_split;
    const int kt1 = min(kt0 + p.kt_per_split, ktiles);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint8_t* sA[2] = {smem, smem + BM * BK * 2};
    uint8_t* sB[2] = {smem + 2 * BM * BK * 2, smem + 2 * BM * BK * 2 + BN * BK * 2};
    uint32_t ncols = 32;
    while ((int)ncols < BN) ncols <<= 1;

    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = make_idesc(BM, BN);
    uint32_t par[2] = {0u, 0u};
    bool ok = true;
    int last = -1;
    for (int kt = kt0; kt < kt1 && ok; kt++) {
        const int i = kt - kt0, s = i & 1;
        if (i >= 2) {  // the MMAs that read this stage two tiles ago are done
            ok = mbar_wait(&bars[s], par[s], p.err);
            par[s] ^= 1u;
            ok = __syncthreads_and(ok) != 0;  // uniform: the loop holds block barriers
            if (!ok) break;
        }
        stage_tile(sA[s], p.A, p.lda, m0, kt * BK, BM);
        stage_tile(sB[s], p.B, p.ldb, n0, kt * BK, BN);
        fence_async_smem();
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_fence_after();
            const uint32_t a = smem_u32(sA[s]), b = smem_u32(sB[s]);
#pragma unroll
            for (int kk = 0; kk < BK / 16; kk++) {
                // K chunk 2kk starts (2kk)*(rows/8)*128 bytes into the tile
                const uint64_t da = make_desc(a + kk * 2 * (BM / 8) * 128, (BM / 8) * 128, 128);
                const uint64_t db = make_desc(b + kk * 2 * (BN / 8) * 128, (BN / 8) * 128, 128);
                mma_bf16(tmem, da, db, idesc, (i > 0 || kk > 0) ? 1u : 0u);
            }
            mma_commit(&bars[s]);
        }
        last = s;
    }
    if (last >= 0 && ok) ok = mbar_wait(&bars[last], par[last], p.err);
    ok = __syncthreads_and(ok) != 0;  // tcgen05.ld below is warp-collective
    tc_fence_after();
    if (last >= 0 && ok) gemm_epilogue(p, tmem, BN, m0, n0, warp, lane);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

// ---- the GEMM with TMA tile loads -------------------------------------------------
//
// The same product, with the operand tiles brought into shared memory by
// the tensor-memory accelerator instead of through registers: thread 0
// issues, per K tile, eight 2D bulk tensor loads of A (box 8 elements x 128
// rows) and eight of B (8 x BN) -- each lands as one column of 8-row x
// 16-byte core matrices, which is exactly the canonical no-swizzle K-major
// layout -- completing on the stage's full mbarrier; the same thread issues
// that tile's MMAs once the stage is full and refills the stage when the
// MMAs reading it have completed (tcgen05.commit on its empty mbarrier).
// Four stages hold a 256-deep K slice of a 128 x 256 tile.  The tensor maps
// cover the operands in this GPU's own memory; no multicast.

constexpr int TMA_STAGES = 4;

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__global__ void __launch_bounds__(THREADS, 1)
    gemm_tma_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, Gemm p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[TMA_STAGES], empty[TMA_STAGES];
    __shared__ uint32_t tmem_slot;
    const int BN = p.bn;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int ktiles = p.K / BK;
    const int kt0 = blockIdx.z * p.kt_per_split;
    const int kt1 = min(kt0 + p.kt_per_split, ktiles);
    const int nk = kt1 > kt0 ? kt1 - kt0 : 0;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const uint32_t a_bytes = BM * BK * 2, stage_bytes = (uint32_t)(BM + BN) * BK * 2;
    uint32_t ncols = 32;
    while ((int)ncols < BN) ncols <<= 1;
    if (threadIdx.x == 0) {
        for (int s = 0; s < TMA_STAGES; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;
    if (threadIdx.x == 0 && nk > 0) {
        const uint32_t idesc = make_idesc(BM, BN);
        auto issue = [&](int i, int s) {
            uint8_t* sa = smem + (size_t)s * stage_bytes;
            uint8_t* sb = sa + a_bytes;
            const int kx = (kt0 + i) * BK;
            mbar_expect(&full[s], stage_bytes);
#pragma unroll
            for (int kb = 0; kb < BK / 8; kb++) {
                tma_load_2d(sa + kb * BM * 16, &ta, kx + kb * 8, m0, &full[s]);
                tma_load_2d(sb + kb * BN * 16, &tb, kx + kb * 8, n0, &full[s]);
            }
        };
        const int pre = nk < TMA_STAGES ? nk : TMA_STAGES;
        for (int i = 0; i < pre; i++) issue(i, i);
        for (int i = 0; i < nk && ok; i++) {
            const int s = i % TMA_STAGES;
            const uint32_t ph = (uint32_t)(i / TMA_STAGES) & 1u;
            ok = mbar_wait(&full[s], ph, p.err);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a = smem_u32(smem + (size_t)s * stage_bytes), b = a + a_bytes;
#pragma unroll
            for (int kk = 0; kk < BK / 16; kk++) {
                const uint64_t da = make_desc(a + kk * 2 * (BM / 8) * 128, (BM / 8) * 128, 128);
                const uint64_t db = make_desc(b + kk * 2 * (BN / 8) * 128, (BN / 8) * 128, 128);
                mma_bf16(tmem, da, db, idesc, (i > 0 || kk > 0) ? 1u : 0u);
            }
            mma_commit(&empty[s]);
            if (i + TMA_STAGES < nk) {  // the stage is free once these MMAs completed
                ok = mbar_wait(&empty[s], ph, p.err);
                if (ok) issue(i + TMA_STAGES, s);
            }
        }
        // every MMA has completed once the last commit arrived
        if (ok) {
            const int l = nk - 1;
            ok = mbar_wait(&empty[l % TMA_STAGES], (uint32_t)(l / TMA_STAGES) & 1u, p.err);
        }
    }
    ok = __syncthreads_and(ok) != 0;  // tcgen05.ld below is warp-collective
    tc_fence_after();
    if (nk > 0 && ok) gemm_epilogue(p, tmem, BN, m0, n0, warp, lane);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
}

// ---- small kernels ------------------------------------------------------------------

// Gaussian NLL per element: 0.5 (lv + (y - mu)^2 exp(-lv)), outputs
// y = [mu | lv | padding] (row stride ldy), targets tgt [B][S].  Writes dY
// (BF16, row stride ldd; padding columns untouched) and its transpose
// ([.][ldT], rows 0..2S-1), scaled by 1/(B*S), and accumulates the loss sum.
__global__ void nll_grad_kernel(const float* __restrict__ y, int ldy, const float* __restrict__ tgt, int B,
                                int S, __nv_bfloat16* __restrict__ dy, int ldd, __nv_bfloat16* __restrict__ dyT,
                                int ldT, float* __restrict__ loss) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.0f;
    if (i < B * S) {
        const int b = i / S, s = i % S;
        const float mu = y[(size_t)b * ldy + s];
        float lv = y[(size_t)b * ldy + S + s];
        lv = fminf(fmaxf(lv, -12.0f), 12.0f);
        const float iv = __expf(-lv);
        const float d = tgt[(size_t)b * S + s] - mu;
        l = 0.5f * (lv + d * d * iv);
        const float sc = 1.0f / ((float)B * (float)S);
        const float gmu = -d * iv * sc;
        const float glv = 0.5f * (1.0f - d * d * iv) * sc;
        const __nv_bfloat16 a = __float2bfloat16(gmu), c = __float2bfloat16(glv);
        dy[(size_t)b * ldd + s] = a;
        dy[(size_t)b * ldd + S + s] = c;
        dyT[(size_t)s * ldT + b] = a;
        dyT[(size_t)(S + s) * ldT + b] = c;
    }
    for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0 && l != 0.0f) atomicAdd(loss, l);
}

// Column sums of a BF16 [B][N] matrix into FP32 g[N] (bias gradients).
__global__ void colsum_kernel(const __nv_bfloat16* __restrict__ d, int B, int N, int ld, float* __restrict__ g) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    const int rows = (B + gridDim.y - 1) / gridDim.y;
    const int b0 = blockIdx.y * rows, b1 = min(B, b0 + rows);
    float acc = 0.0f;
    for (int b = b0; b < b1; b++) acc += __bfloat162float(d[(size_t)b * ld + n]);
    atomicAdd(g + n, acc);
}

// Adam on FP32 master weights; refreshes the BF16 copy W [rows][cols] and its
// transpose WT [cols][rows] used by the backward GEMMs.
__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m1,
                            float* __restrict__ m2, int n, int rows, int cols, float lr, float b1, float b2,
                            float eps, float c1, float c2, float wd, __nv_bfloat16* __restrict__ wb,
                            __nv_bfloat16* __restrict__ wbT) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i] + wd * w[i];
    const float a = b1 * m1[i] + (1.0f - b1) * gi;
    const float b = b2 * m2[i] + (1.0f - b2) * gi * gi;
    m1[i] = a;
    m2[i] = b;
    const float wi = w[i] - lr * (a / c1) / (sqrtf(b / c2) + eps);
    w[i] = wi;
    if (wb) {
        const __nv_bfloat16 h = __float2bfloat16(wi);
        wb[i] = h;
        if (wbT) {
            const int r = i / cols, c = i % cols;
            wbT[(size_t)c * rows + r] = h;
        }
    }
}


// ---- fused screening: input build -> 5 layers -> fitness, one kernel --------------
//
// Screening scores candidates by the surrogate's ensemble mean: rows are
// (candidate, sample instant) pairs, row = cand * ns + ti.  One persistent
// CTA per SM has two 128-row tiles under way, half a layer apart: while the
// tensor cores run one tile's layer, the other tile's warps turn its last
// accumulator into its next operand.  A tile's activations stay in shared
// memory for all five layers, so HBM sees only the candidates' parameters and
// one fitness word per candidate:
//   * warps 0-7 / 8-15 (tile 0 / 1): build the layer-0 input rows, then per
//     layer read the tile's TMEM accumulator (warp w owns rows 32(w%4).. and
//     column half (w/4)%2), add bias, SiLU, round to BF16 and write the next
//     layer's A operand in place; after the last layer sum_s |target - mean|
//     / target per row, summed over a warp's rows of one candidate and added
//     to its FP64 fitness;
//   * warp 16 (producer): streams the packed weights, 32 K-columns per stage,
//     5 stages, with bulk asynchronous copies completing on mbarriers, once
//     per tile and layer;
//   * warp 17 (MMA): one thread issues tcgen05.mma (M = 128, N = layer width,
//     K = 16), the two tiles' layers in turn.
// TMEM: 512 columns, 256 per tile.  Bounds per tile and SM: 8,192 cycles of
// MUFU tanh (16 per cycle), 7,200 of MMAs, 12,000 of shared-memory traffic
// (operands 720 KB, weights 458 KB, activations and biases 400 KB).  Both tiles
// in one step, waiting for each other's epilogues, took 34,500 cycles per tile:
// 4,600 per layer of MMAs, 5,400 of epilogue, 1,000 of hand-over, 17,000 in the
// final sums (32 lanes of a warp on one shared-memory word) and 6,000 in the
// inputs.  Now 18,600: a tile's layer is 2,600 cycles of MMAs (issue: 160 per
// MMA), 600 until the epilogue sees them, 3,600 of epilogue and 400 until the
// next MMA; what bounds it is that chain, with two tiles in TMEM to overlap.
// 100,000 candidates x 50 instants on one B200: 4,990 us before, 2,814 now (28
// and 49 % of the measured BF16 rate).
constexpr int SC_BK = 32, SC_STAGES = 5, SC_HID = 256, SC_LAYERS = 5;
constexpr int SC_EPI = 512;                       // epilogue threads (16 warps, 8 per tile)
constexpr int SC_THREADS = SC_EPI + 64;           // + producer and MMA warps
constexpr int SC_A_BYTES = 128 * SC_HID * 2;      // one tile's activations
constexpr int SC_STAGE_BYTES = SC_HID * SC_BK * 2;
constexpr int SC_CONST_BYTES = 16384;             // biases, output scaling, target (when it fits)

struct Screen {
    const float* theta;   // [n_cand][n_par]
    int n_par;
    uint32_t n_cand, ns, n_rows, n_tiles;
    const float* tvec;    // [ns]
    float t_end;
    const float* log_lo;  // [n_par]
    const float* log_hi;
    const float* y_mean;  // [S]
    const float* y_std;
    int S, out_w;
    const float* target;  // [ns][S]
    const uint8_t* wpack; // packed BF16 weights (ctl_mlp_pack)
    const float* bias;    // [4*256 + out_w]
    double* fit;          // [n_cand], zeroed by the caller
    double scale;         // 1 / (ns * S)
    unsigned* err;
};

__device__ __forceinline__ int sc_k(int l) { return l == 0 ? 64 : SC_HID; }
__device__ __forceinline__ int sc_n(const Screen& p, int l) { return l == SC_LAYERS - 1 ? p.out_w : SC_HID; }

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// One arrival for a warp's 32 lanes, each with its shared-memory writes fenced:
// 512 arrivals on one barrier took longer than the MMAs they announced.
__device__ __forceinline__ void mbar_arrive_warp(uint64_t* bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// 32 columns of the accumulator into registers; tmem_wait() makes them
// valid, so a second load can be in flight while the first is processed.
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
// One lane waits for its warp.  The shuffle hands over the answer but orders no
// memory: the barrier does, between that lane's acquire and the accumulator and
// shared memory that the other lanes go on to.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, unsigned* err) {
    bool ok = true;
    if ((threadIdx.x & 31) == 0) ok = mbar_wait(bar, parity, err);
    ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
    __syncwarp();
    return ok;
}

// Byte offset of (row, k) in a K-major no-swizzle tile with `rows` rows.
__device__ __forceinline__ uint32_t canon(int row, int k, int rows) {
    return (uint32_t)(((k >> 3) * (rows >> 3) + (row >> 3)) * 128 + (row & 7) * 16 + (k & 7) * 2);
}


// A tile row's candidate, instant and first eight parameters, loaded while the
// tile before it is still in its last layer.
struct ScRow {
    uint32_t cand, ti;
    bool live;
    float t, th[8];
};
__device__ __forceinline__ void sc_load_row(const Screen& p, uint32_t row, int h, ScRow& x) {
    x.live = row < p.n_rows;
    x.cand = x.live ? row / p.ns : 0u;
    x.ti = x.live ? row - x.cand * p.ns : 0u;
    x.t = p.tvec[x.ti];
    const float* th = p.theta + (size_t)x.cand * p.n_par;
#pragma unroll
    for (int q = 0; q < 8; q++) x.th[q] = h == 0 && q < p.n_par ? th[q] : 0.0f;
}

// Layer-0 input columns [32 h, 32 h + 32) of row r of the tile: scaled log
// parameters in [-1, 1], scaled time, zeros (the same FP32 operations as
// surrogate.make_inputs).  lo, hi: the prior box in shared memory.
__device__ __forceinline__ void sc_build_input(const Screen& p, const float* lo, const float* hi, uint8_t* A, int r, int h,
                                               const ScRow& row) {
    const float* th = p.theta + (size_t)row.cand * p.n_par;
    const float tsc = (2.0f * row.t) / p.t_end - 1.0f;
#pragma unroll
    for (int kb = 0; kb < 4; kb++) {
        const int c = 32 * h + kb * 8;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (c <= p.n_par && row.live) {
            float x[8];
#pragma unroll
            for (int q = 0; q < 8; q++) x[q] = kb == 0 && h == 0 ? row.th[q] : c + q < p.n_par ? th[c + q] : 0.0f;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int j = c + q;
                if (j < p.n_par) x[q] = (2.0f * (x[q] - lo[j])) / (hi[j] - lo[j]) - 1.0f;
                else if (j == p.n_par) x[q] = tsc;
            }
            v = make_uint4(pack_bf2(x[0], x[1]), pack_bf2(x[2], x[3]), pack_bf2(x[4], x[5]), pack_bf2(x[6], x[7]));
        }
        *reinterpret_cast<uint4*>(A + canon(r, c, 128)) = v;
    }
}

// Tiles of this CTA: blockIdx.x + i * gridDim.x for i < my_tiles; tile i
// runs in slot i % 2.
__device__ __forceinline__ uint32_t sc_my_tiles(const Screen& p) {
    return blockIdx.x < p.n_tiles ? (p.n_tiles - 1u - blockIdx.x) / gridDim.x + 1u : 0u;
}

__global__ void __launch_bounds__(SC_THREADS, 1) screen_kernel(const __grid_constant__ Screen p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[SC_STAGES], empty[SC_STAGES], acc_full[2], a_ready[2], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    uint8_t* stage = smem + 2 * SC_A_BYTES;
    // per-CTA constants in shared memory: biases [4*256 + out_w], y_mean [S],
    // y_std [S], the prior box [2][n_par], and the target [ns][S] when it fits,
    // in rows of odd length (neighbouring lanes read neighbouring instants)
    float* c_bias = reinterpret_cast<float*>(stage + SC_STAGES * SC_STAGE_BYTES);
    float* c_ym = c_bias + 4 * SC_HID + p.out_w;
    float* c_ys = c_ym + p.S;
    float* c_lo = c_ys + p.S;
    float* c_hi = c_lo + p.n_par;
    float* c_tg = c_hi + p.n_par;
    const uint32_t trow = (uint32_t)p.S | 1u;
    const bool tg_smem =
        (size_t)(4 * SC_HID + p.out_w + 2 * p.S + 2 * p.n_par) * 4 + (size_t)p.ns * trow * 4 <= (size_t)SC_CONST_BYTES;
    const float* tgt = tg_smem ? c_tg : p.target;
    const uint32_t tstride = tg_smem ? trow : (uint32_t)p.S;
    for (int i = threadIdx.x; i < 4 * SC_HID + p.out_w; i += SC_THREADS) c_bias[i] = p.bias[i];
    for (int i = threadIdx.x; i < p.S; i += SC_THREADS) {
        c_ym[i] = p.y_mean[i];
        c_ys[i] = p.y_std[i];
    }
    for (int i = threadIdx.x; i < p.n_par; i += SC_THREADS) {
        c_lo[i] = p.log_lo[i];
        c_hi[i] = p.log_hi[i];
    }
    if (tg_smem)
        for (int i = threadIdx.x; i < (int)(p.ns * p.S); i += SC_THREADS)
            c_tg[(uint32_t)(i / p.S) * trow + i % p.S] = p.target[i];
    const int warp = warp_index(), lane = threadIdx.x % 32;
    const uint32_t my = sc_my_tiles(p);
    if (threadIdx.x == 0) {
        for (int i = 0; i < SC_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&a_ready[i], SC_EPI / 64);
        }
        mbar_init(&drain, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_slot)), "r"(2 * SC_HID));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp == 16) {
        // ---- producer: the weight stream, once per tile and layer ----
        uint32_t sl = 0, par = 1u, issued = 0;  // stage, parity of its empty barrier (the first round passes), copies
        bool ok = true;
        for (uint32_t i0 = 0; i0 < my && ok; i0 += 2) {
            size_t base = 0;
            for (int l = 0; l < SC_LAYERS && ok; l++) {
                const uint32_t bytes = (uint32_t)(sc_n(p, l) * SC_BK * 2);
                const int ns = sc_k(l) / SC_BK;
                for (uint32_t e = 0; e < (i0 + 1 < my ? 2u : 1u) && ok; e++) {
                    if (raised(&abort_flag)) { ok = false; break; }
                    for (int ks = 0; ks < ns; ks++) {
                        if (!mbar_wait_u(&empty[sl], par, p.err)) { ok = false; break; }
                        if (elect_one()) {
                            mbar_expect_tx(&full[sl], bytes);
                            bulk_g2s(stage + sl * SC_STAGE_BYTES, p.wpack + base + (size_t)ks * bytes, bytes, &full[sl]);
                        }
                        issued++;
                        if (++sl == SC_STAGES) {
                            sl = 0;
                            par ^= 1u;
                        }
                    }
                }
                base += (size_t)ns * bytes;
            }
        }
        if (!ok) {
            if (lane == 0) atomicExch(&abort_flag, 1);
            // let the copies in flight land before the CTA exits
            for (uint32_t i = issued > SC_STAGES ? issued - SC_STAGES : 0u; i < issued; i++)
                mbar_wait_u(&full[i % SC_STAGES], (i / SC_STAGES) & 1u, nullptr);
        }
    } else if (warp == 17) {
        // ---- MMA issuer: the tiles' layers in turn ----
        uint32_t sl = 0, par = 0u, jobs = 0;
        bool ok = true;
        const uint32_t s0 = smem_u32(stage);
        for (uint32_t i0 = 0; i0 < my && ok; i0 += 2) {
            for (int l = 0; l < SC_LAYERS && ok; l++, jobs++) {
                const int N = sc_n(p, l);
                const uint32_t idesc = make_idesc(128, N);
                const uint32_t kstep = (uint32_t)(2 * (N / 8) * 128), lbo = (uint32_t)((N / 8) * 128);
                for (uint32_t e = 0; e < (i0 + 1 < my ? 2u : 1u); e++) {
                    if (!mbar_wait_u(&a_ready[e], jobs & 1u, p.err) || raised(&abort_flag)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a = smem_u32(smem + e * SC_A_BYTES), d = tmem + e * SC_HID;
#pragma unroll 4
                    for (int ks = 0; ks < sc_k(l) / SC_BK; ks++) {
                        if (!mbar_wait_u(&full[sl], par, p.err)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t b = s0 + sl * SC_STAGE_BYTES;
                        if (elect_one()) {
#pragma unroll
                            for (int kk = 0; kk < SC_BK / 16; kk++)  // K offset in the activation tile: 32 ks + 16 kk
                                mma_bf16(d, make_desc(a + (uint32_t)(ks * 4 + kk * 2) * 16u * 128u, 16u * 128u, 128u),
                                         make_desc(b + (uint32_t)kk * kstep, lbo, 128u), idesc,
                                         (ks > 0 || kk > 0) ? 1u : 0u);
                            mma_commit(&empty[sl]);
                        }
                        if (++sl == SC_STAGES) {
                            sl = 0;
                            par ^= 1u;
                        }
                    }
                    if (!ok) break;
                    if (elect_one()) mma_commit(&acc_full[e]);
                }
            }
        }
        if (!ok && lane == 0) atomicExch(&abort_flag, 1);
        if (elect_one()) mma_commit(&drain);  // every MMA this warp issued has completed once drain flips
        mbar_wait_u(&drain, 0u, nullptr);
    } else {
        // ---- epilogue: warps 8e..8e+7 serve tile e; warp w owns rows 32(w%4)..
        // (its TMEM lane quadrant) and column half h = (w/4)%2 ----
        const uint32_t e = (uint32_t)warp >> 3;
        const int q = warp & 3, h = (warp >> 2) & 1;
        const int r = q * 32 + lane;
        uint8_t* A = smem + e * SC_A_BYTES;
        const uint32_t tbase = tmem + e * SC_HID + ((uint32_t)(q * 32) << 16);
        uint32_t nacc = 0;
        bool ok = true;
        ScRow next;
        if (e < my) sc_load_row(p, (blockIdx.x + e * gridDim.x) * 128u + (uint32_t)r, h, next);
        for (uint32_t i = e; i < my && ok; i += 2) {
            const bool live = next.live;
            const uint32_t cand = live ? next.cand : 0xffffffffu, ti = next.ti;  // (rows past the end: no candidate's)
            sc_build_input(p, c_lo, c_hi, A, r, h, next);
            fence_async_smem();
            tc_fence_before();
            mbar_arrive_warp(&a_ready[e]);
            for (int l = 0; l < SC_LAYERS - 1; l++) {
                ok = mbar_wait_warp(&acc_full[e], nacc & 1u, p.err) && !__any_sync(0xffffffffu, *(volatile int*)&abort_flag);
                nacc++;
                if (!ok) break;
                tc_fence_after();
                const float* b = c_bias + l * SC_HID;
                const int c0 = 128 * h;
                uint32_t ra[32], rb[32];
                tmem_ld32_issue(tbase + (uint32_t)c0, ra);
#pragma unroll
                for (int j = 0; j < 4; j++) {  // four 32-column chunks, the next load in flight
                    tmem_wait();
                    uint32_t(&cur)[32] = (j & 1) ? rb : ra;
                    if (j < 3) tmem_ld32_issue(tbase + (uint32_t)(c0 + 32 * (j + 1)), (j & 1) ? ra : rb);
                    const int c = c0 + 32 * j;
                    const float4* b4 = reinterpret_cast<const float4*>(b + c);
#pragma unroll
                    for (int k = 0; k < 4; k++) {  // 8 columns -> one 16-byte store
                        const float4 ba = b4[2 * k], bb = b4[2 * k + 1];
                        const uint32_t* u = cur + 8 * k;
                        uint4 o;
                        o.x = pack_bf2(silu(__uint_as_float(u[0]) + ba.x), silu(__uint_as_float(u[1]) + ba.y));
                        o.y = pack_bf2(silu(__uint_as_float(u[2]) + ba.z), silu(__uint_as_float(u[3]) + ba.w));
                        o.z = pack_bf2(silu(__uint_as_float(u[4]) + bb.x), silu(__uint_as_float(u[5]) + bb.y));
                        o.w = pack_bf2(silu(__uint_as_float(u[6]) + bb.z), silu(__uint_as_float(u[7]) + bb.w));
                        *reinterpret_cast<uint4*>(A + canon(r, c + 8 * k, 128)) = o;
                    }
                }
                fence_async_smem();
                tc_fence_before();
                mbar_arrive_warp(&a_ready[e]);
            }
            if (!ok) break;
            if (i + 2 < my) sc_load_row(p, (blockIdx.x + (i + 2) * gridDim.x) * 128u + (uint32_t)r, h, next);
            ok = mbar_wait_warp(&acc_full[e], nacc & 1u, p.err) && !__any_sync(0xffffffffu, *(volatile int*)&abort_flag);
            nacc++;
            if (!ok) break;
            tc_fence_after();
            // fitness terms of this row: sum_s |target - mean| (/ target when
            // nonzero), 16-column chunks alternating between the column halves
            const float* b = c_bias + (SC_LAYERS - 1) * SC_HID;
            const float* tr = tgt + (size_t)ti * tstride;
            float acc = 0.0f;
            for (int c = 16 * h; c < p.S; c += 32) {
                float v[16];
                tmem_ld16(tbase + (uint32_t)c, v);
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const int s_ = c + j;
                    if (s_ < p.S) {
                        const float mean = (v[j] + b[s_]) * c_ys[s_] + c_ym[s_];
                        const float tg = tr[s_];
                        const float d = fabsf(tg - mean), dq = d / (tg != 0.0f ? tg : 1.0f);
                        acc += live ? dq : 0.0f;
                    }
                }
            }
            tc_fence_before();
            // the warp's rows of one candidate are neighbouring lanes: a
            // segmented sum leaves each candidate's share in its last lane
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, acc, o);
                const uint32_t cu = __shfl_up_sync(0xffffffffu, cand, o);
                if (lane >= o && cu == cand) acc += up;
            }
            const uint32_t cn = __shfl_down_sync(0xffffffffu, cand, 1);
            if (live && (lane == 31 || cn != cand)) atomicAdd(&p.fit[cand], (double)acc * p.scale);
        }
        if (!ok) atomicExch(&abort_flag, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * SC_HID));
}

// Packs a BF16 weight matrix W [N][K] (K contiguous, row stride ldw) into
// K-stages of 32 columns, each stage N x 32 in the canonical K-major layout,
// stages consecutive: the screening kernel copies one stage per bulk copy.
__global__ void pack_kernel(const __nv_bfloat16* __restrict__ W, int N, int K, int ldw,
                            __nv_bfloat16* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N * K) return;
    const int n = i / K, k = i % K;
    const int ks = k / SC_BK, kin = k % SC_BK;
    const size_t o = (size_t)ks * N * SC_BK + canon(n, kin, N) / 2;
    out[o] = W[(size_t)n * ldw + k];
}

}  // namespace mlp
}  // namespace ctl

#include "ctl_train.cuh"

using namespace ctl;

static ctl_status mlp_cuda(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return CTL_OK;
    set_error(std::string(what) + ": " + cudaGetErrorString(e));
    return CTL_ERR_CUDA;
}

namespace ctl {
namespace mlp {

// A 2D tensor map over a row-major BF16 operand [rows][ld] (K contiguous)
// with boxes of 8 K-elements x box_rows rows, for gemm_tma_kernel.  False
// when the driver offers no encoder or the operand breaks its rules.
static bool tensor_map(CUtensorMap& map, const void* base, int K, int rows, int ld, int box_rows) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static bool tried = false;
    if (!tried) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
        else
            cudaGetLastError();
        tried = true;
    }
    if (!encode || (reinterpret_cast<uintptr_t>(base) & 15) || ((size_t)ld * 2) % 16 || box_rows > 256) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {8u, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1u, 1u};
    return encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One warp waits, through the same bounded wait as the GEMM and screening
// kernels, on an mbarrier that nothing arrives on; no MMA or bulk copy is in
// flight.  The wait gives up after `limit` polls, raises bit 0 of *err and
// the kernel returns.
__global__ void wait_check_kernel(unsigned* err, uint32_t limit) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (threadIdx.x == 0 && !mbar_wait(&bar, 0u, err, limit)) atomicOr(err, 2u);
}

}  // namespace mlp
}  // namespace ctl

extern "C" ctl_status ctl_mlp_wait_check(unsigned* d_err, uint32_t limit, void* stream) {
    if (!d_err || limit == 0 || limit > mlp::WAIT_LIMIT) {
        set_error("ctl_mlp_wait_check: a device error word and 1 <= limit <= 2^24");
        return CTL_ERR_ARG;
    }
    mlp::wait_check_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(d_err, limit);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error(std::string("ctl_mlp_wait_check: ") + cudaGetErrorString(e));
        return CTL_ERR_CUDA;
    }
    return CTL_OK;
}

extern "C" ctl_status ctl_mlp_gemm(const ctl_gemm_desc* d, void* stream) {
    if (!d || !d->A || !d->B) return CTL_ERR_ARG;
    if (d->M % 128 || d->K % 64 || d->N % 16 || d->N <= 0 || (d->N > 256 && d->N % 256)) {
        set_error("ctl_mlp_gemm: M % 128, K % 64, N % 16 (and N % 256 above 256) must be 0");
        return CTL_ERR_SHAPE;
    }
    if (d->lda % 8 || d->ldb % 8) {
        set_error("ctl_mlp_gemm: leading dimensions must be multiples of 8 elements");
        return CTL_ERR_SHAPE;
    }
    mlp::Gemm p;
    p.A = static_cast<const __nv_bfloat16*>(d->A);
    p.B = static_cast<const __nv_bfloat16*>(d->B);
    p.lda = d->lda; p.ldb = d->ldb; p.M = d->M; p.N = d->N; p.K = d->K;
    p.epi = d->epilogue;
    p.bias = d->bias; p.z_in = d->z_in; p.ldz = d->ldz;
    p.out_f32 = d->out_f32; p.ldo = d->ldo;
    p.out_bf = static_cast<__nv_bfloat16*>(d->out_bf); p.ldob = d->ldob;
    p.out_bfT = static_cast<__nv_bfloat16*>(d->out_bfT); p.ldobT = d->ldobT;
    p.err = d->err;
    const int ktiles = d->K / 64;
    const int splits = d->splits > 0 ? (d->splits < ktiles ? d->splits : ktiles) : 1;
    p.kt_per_split = (ktiles + splits - 1) / splits;
    const int BN = d->N < 256 ? d->N : 256;
    p.bn = BN;
    const size_t smem = (size_t)2 * mlp::BM * mlp::BK * 2 + (size_t)2 * BN * mlp::BK * 2;
    static bool attr_set = false;
    if (!attr_set) {
        ctl_status st = mlp_cuda(cudaFuncSetAttribute(mlp::gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                      2 * mlp::BM * mlp::BK * 2 + 2 * 256 * mlp::BK * 2),
                                 "cudaFuncSetAttribute(gemm)");
        if (st != CTL_OK) return st;
        attr_set = true;
    }
    dim3 grid((unsigned)(d->M / 128), (unsigned)((d->N + BN - 1) / BN), (unsigned)splits);
    // TMA tile loads when the driver's tensor-map encoder is available and
    // the operands meet its rules (16-byte aligned bases and row strides);
    // register staging otherwise.
    CUtensorMap ta, tb;
    if (mlp::tensor_map(ta, d->A, d->K, d->M, d->lda, 128) && mlp::tensor_map(tb, d->B, d->K, d->N, d->ldb, BN)) {
        const size_t tsmem = (size_t)mlp::TMA_STAGES * (size_t)(mlp::BM + BN) * mlp::BK * 2;
        static bool tattr_set = false;
        if (!tattr_set) {
            ctl_status st = mlp_cuda(cudaFuncSetAttribute(mlp::gemm_tma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                          mlp::TMA_STAGES * (mlp::BM + 256) * mlp::BK * 2),
                                     "cudaFuncSetAttribute(gemm_tma)");
            if (st != CTL_OK) return st;
            tattr_set = true;
        }
        mlp::gemm_tma_kernel<<<grid, mlp::THREADS, tsmem, static_cast<cudaStream_t>(stream)>>>(ta, tb, p);
        return mlp_cuda(cudaGetLastError(), "gemm_tma_kernel launch");
    }
    mlp::gemm_kernel<<<grid, mlp::THREADS, smem, static_cast<cudaStream_t>(stream)>>>(p);
    return mlp_cuda(cudaGetLastError(), "gemm_kernel launch");
}

extern "C" ctl_status ctl_mlp_nll_grad(const float* y, int32_t ldy, const float* tgt, int32_t B, int32_t S,
                                       void* dy, int32_t ldd, void* dyT, int32_t ldT, float* loss, void* stream) {
    if (!y || !tgt || !dy || !dyT || !loss || B <= 0 || S <= 0 || 2 * S > 128 || ldT < B || ldy < 2 * S ||
        ldd < 2 * S)
        return CTL_ERR_ARG;
    const int n = B * S;
    mlp::nll_grad_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        y, ldy, tgt, B, S, static_cast<__nv_bfloat16*>(dy), ldd, static_cast<__nv_bfloat16*>(dyT), ldT, loss);
    return mlp_cuda(cudaGetLastError(), "nll_grad_kernel launch");
}

extern "C" ctl_status ctl_mlp_colsum(const void* d, int32_t B, int32_t N, int32_t ld, float* g, void* stream) {
    if (!d || !g || B <= 0 || N <= 0) return CTL_ERR_ARG;
    dim3 grid((unsigned)((N + 127) / 128), (unsigned)(B > 64 * 1024 ? 128 : (B + 511) / 512));
    mlp::colsum_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(d), B, N, ld, g);
    return mlp_cuda(cudaGetLastError(), "colsum_kernel launch");
}

extern "C" ctl_status ctl_mlp_adam(float* w, const float* g, float* m1, float* m2, int32_t rows, int32_t cols,
                                   float lr, float beta1, float beta2, float eps, int32_t step, float wd,
                                   void* wb, void* wbT, void* stream) {
    if (!w || !g || !m1 || !m2 || rows <= 0 || cols <= 0 || step <= 0) return CTL_ERR_ARG;
    const int n = rows * cols;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    mlp::adam_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        w, g, m1, m2, n, rows, cols, lr, beta1, beta2, eps, c1, c2, wd, static_cast<__nv_bfloat16*>(wb),
        static_cast<__nv_bfloat16*>(wbT));
    return mlp_cuda(cudaGetLastError(), "adam_kernel launch");
}

extern "C" size_t ctl_mlp_pack_bytes(int32_t out_w) {
    return (size_t)2 * (256 * 64 + 3 * 256 * 256 + (size_t)out_w * 256);
}

extern "C" ctl_status ctl_mlp_pack(const void* const* W, const int32_t* ldw, int32_t out_w, void* wpack,
                                   void* stream) {
    if (!W || !ldw || !wpack || out_w <= 0 || out_w % 16 || out_w > 256) return CTL_ERR_ARG;
    if (reinterpret_cast<uintptr_t>(wpack) % 16) {
        set_error("ctl_mlp_pack: output must be 16-byte aligned");
        return CTL_ERR_ARG;
    }
    auto* out = static_cast<__nv_bfloat16*>(wpack);
    size_t off = 0;
    for (int l = 0; l < mlp::SC_LAYERS; l++) {
        const int N = l == mlp::SC_LAYERS - 1 ? out_w : mlp::SC_HID, K = l == 0 ? 64 : mlp::SC_HID;
        if (!W[l] || ldw[l] < K) return CTL_ERR_ARG;
        mlp::pack_kernel<<<(N * K + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
            static_cast<const __nv_bfloat16*>(W[l]), N, K, ldw[l], out + off);
        ctl_status st = mlp_cuda(cudaGetLastError(), "pack_kernel launch");
        if (st != CTL_OK) return st;
        off += (size_t)N * K;
    }
    return CTL_OK;
}

extern "C" ctl_status ctl_mlp_screen(const ctl_screen_desc* d, void* stream) {
    if (!d || !d->theta || !d->tvec || !d->log_lo || !d->log_hi || !d->y_mean || !d->y_std || !d->target ||
        !d->wpack || !d->bias || !d->fitness)
        return CTL_ERR_ARG;
    if (d->n_par < 1 || d->n_par > 63 || d->ns == 0 || d->S < 1 || 2 * d->S > d->out_w || d->out_w % 16 ||
        d->out_w > 256 || !(d->t_end > 0.0f)) {
        set_error("ctl_mlp_screen: need 1 <= n_par <= 63, ns >= 1, 2*S <= out_w <= 256, out_w % 16 == 0, t_end > 0");
        return CTL_ERR_SHAPE;
    }
    if (reinterpret_cast<uintptr_t>(d->wpack) % 16 || reinterpret_cast<uintptr_t>(d->bias) % 16) {
        set_error("ctl_mlp_screen: packed weights and biases must be 16-byte aligned");
        return CTL_ERR_ARG;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    ctl_status st = mlp_cuda(cudaMemsetAsync(d->fitness, 0, sizeof(double) * d->n_cand, s), "memset fitness");
    if (st != CTL_OK || d->n_cand == 0) return st;
    const uint64_t rows = (uint64_t)d->n_cand * d->ns;
    if (rows > 0xffffff00ull) {
        set_error("ctl_mlp_screen: n_cand * ns must fit in 32 bits");
        return CTL_ERR_SHAPE;
    }
    mlp::Screen p;
    p.theta = d->theta; p.n_par = d->n_par; p.n_cand = d->n_cand; p.ns = d->ns;
    p.n_rows = (uint32_t)rows; p.n_tiles = (uint32_t)((rows + 127) / 128);
    p.tvec = d->tvec; p.t_end = d->t_end; p.log_lo = d->log_lo; p.log_hi = d->log_hi;
    p.y_mean = d->y_mean; p.y_std = d->y_std; p.S = d->S; p.out_w = d->out_w; p.target = d->target;
    p.wpack = static_cast<const uint8_t*>(d->wpack); p.bias = d->bias; p.fit = d->fitness; p.err = d->err;
    const size_t smem = (size_t)2 * mlp::SC_A_BYTES + (size_t)mlp::SC_STAGES * mlp::SC_STAGE_BYTES +
                        (size_t)mlp::SC_CONST_BYTES;
    static int sms[16];
    int dev = 0;
    if ((st = mlp_cuda(cudaGetDevice(&dev), "cudaGetDevice")) != CTL_OK) return st;
    if (dev < 0 || dev >= 16) return CTL_ERR_ARG;
    if (!sms[dev]) {
        if ((st = mlp_cuda(cudaFuncSetAttribute(mlp::screen_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)smem), "cudaFuncSetAttribute(screen)")) != CTL_OK)
            return st;
        int n = 0;
        if ((st = mlp_cuda(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev), "sm count")) != CTL_OK)
            return st;
        sms[dev] = n;
    }
    const uint32_t grid = std::min<uint32_t>(p.n_tiles, (uint32_t)sms[dev]);  // one CTA per SM
    p.scale = 1.0 / ((double)d->ns * (double)d->S);
    mlp::screen_kernel<<<grid, mlp::SC_THREADS, smem, s>>>(p);
    return mlp_cuda(cudaGetLastError(), "screen_kernel launch");
}

// ---- one training step ------------------------------------------------------------

namespace {

bool aligned(const void* p, size_t n) { return p && reinterpret_cast<uintptr_t>(p) % n == 0; }

ctl_status check_step(const ctl_mlp_step_desc* d, const char* who) {
    if (!d) return CTL_ERR_ARG;
    if (d->B <= 0 || d->B % 128 || (d->out_w != 64 && d->out_w != 128)) {
        set_error(std::string(who) + ": the batch is a positive multiple of 128 rows and out_w 64 or 128");
        return CTL_ERR_SHAPE;
    }
    return CTL_OK;
}

// SM count of the current device, after raising the kernels' shared-memory
// ceilings there once.
ctl_status step_device(int& sms) {
    static int known[16];
    int dev = 0;
    ctl_status st = mlp_cuda(cudaGetDevice(&dev), "cudaGetDevice");
    if (st != CTL_OK) return st;
    if (dev < 0 || dev >= 16) return CTL_ERR_ARG;
    if (!known[dev]) {
        const struct {
            const void* k;
            int bytes;
        } ks[] = {{reinterpret_cast<const void*>(mlp::train_forward_kernel), mlp::TR_SMEM},
                  {reinterpret_cast<const void*>(mlp::train_backward_kernel), mlp::TR_SMEM},
                  {reinterpret_cast<const void*>(mlp::train_wgrad_kernel), mlp::WG_SMEM}};
        for (const auto& k : ks)
            if ((st = mlp_cuda(cudaFuncSetAttribute(k.k, cudaFuncAttributeMaxDynamicSharedMemorySize, k.bytes),
                               "cudaFuncSetAttribute(training step)")) != CTL_OK)
                return st;
        int n = 0;
        if ((st = mlp_cuda(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev), "sm count")) != CTL_OK)
            return st;
        known[dev] = n;
    }
    sms = known[dev];
    return CTL_OK;
}

ctl_status pack_matrices(const void* const* w, const int* n, const int* k, int count, void* out, cudaStream_t s) {
    mlp::Pack p = {};
    size_t off = 0;
    int most = 0;
    for (int l = 0; l < count; l++) {
        if (!aligned(w[l], 16)) return CTL_ERR_ARG;
        p.w[l] = static_cast<const __nv_bfloat16*>(w[l]);
        p.ld[l] = p.k[l] = k[l];
        p.n[l] = n[l];
        p.off[l] = off;
        off += (size_t)n[l] * k[l] * 2;
        most = std::max(most, n[l] * k[l] / 8);
    }
    p.out = static_cast<uint8_t*>(out);
    mlp::train_pack_kernel<<<dim3((unsigned)((most + 255) / 256), (unsigned)count), 256, 0, s>>>(p);
    return mlp_cuda(cudaGetLastError(), "train_pack_kernel launch");
}

}  // namespace

extern "C" ctl_status ctl_mlp_forward(const ctl_mlp_step_desc* d, void* stream) {
    ctl_status st = check_step(d, "ctl_mlp_forward");
    if (st != CTL_OK) return st;
    bool ok = aligned(d->X, 16) && aligned(d->wpack, 16) && aligned(d->y, 32);
    for (int l = 0; l < mlp::TR_L; l++) ok = ok && d->bias[l] && (d->hp[l] == nullptr || aligned(d->hp[l], 16));
    for (int l = 0; l < 4; l++) ok = ok && aligned(d->z[l], 32);
    if (!ok) {
        set_error("ctl_mlp_forward: a buffer is missing or not aligned");
        return CTL_ERR_ARG;
    }
    int sms = 0;
    if ((st = step_device(sms)) != CTL_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int n[5] = {256, 256, 256, 256, d->out_w}, k[5] = {64, 256, 256, 256, 256};
    if ((st = pack_matrices(d->W, n, k, 5, d->wpack, s)) != CTL_OK) return st;
    mlp::Train p = {};
    p.X = static_cast<const __nv_bfloat16*>(d->X);
    p.wpack = static_cast<const uint8_t*>(d->wpack);
    for (int l = 0; l < mlp::TR_L; l++) {
        p.bias[l] = d->bias[l];
        p.hp[l] = static_cast<uint8_t*>(d->hp[l]);
    }
    for (int l = 0; l < 4; l++) p.z[l] = d->z[l];
    p.y = d->y;
    p.B = d->B;
    p.out_w = d->out_w;
    p.err = d->err;
    mlp::train_forward_kernel<<<d->B / 128, mlp::TR_THREADS, mlp::TR_SMEM, s>>>(p);
    return mlp_cuda(cudaGetLastError(), "train_forward_kernel launch");
}

extern "C" ctl_status ctl_mlp_backward(const ctl_mlp_step_desc* d, void* stream) {
    ctl_status st = check_step(d, "ctl_mlp_backward");
    if (st != CTL_OK) return st;
    bool ok = aligned(d->wpack, 16) && aligned(d->y, 32) && d->target && d->loss && d->S > 0 && 2 * d->S <= d->out_w;
    for (int l = 0; l < mlp::TR_L; l++)
        ok = ok && aligned(d->hp[l], 16) && aligned(d->dp[l], 16) && aligned(d->dW[l], 16) && d->db[l];
    for (int l = 0; l < 4; l++) ok = ok && aligned(d->z[l], 32);
    if (!ok) {
        set_error("ctl_mlp_backward: a buffer is missing or not aligned, or 2 S > out_w");
        return CTL_ERR_ARG;
    }
    int sms = 0;
    if ((st = step_device(sms)) != CTL_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const void* w[4] = {d->WT[4], d->WT[3], d->WT[2], d->WT[1]};
    const int n[4] = {256, 256, 256, 256}, k[4] = {d->out_w, 256, 256, 256};
    if ((st = pack_matrices(w, n, k, 4, d->wpack, s)) != CTL_OK) return st;
    mlp::Train p = {};
    p.wtpack = static_cast<const uint8_t*>(d->wpack);
    for (int l = 0; l < mlp::TR_L; l++) {
        p.hp[l] = static_cast<uint8_t*>(d->hp[l]);
        p.dp[l] = static_cast<uint8_t*>(d->dp[l]);
        p.dW[l] = d->dW[l];
        p.db[l] = d->db[l];
    }
    for (int l = 0; l < 4; l++) p.z[l] = d->z[l];
    p.y = d->y;
    p.target = d->target;
    p.loss = d->loss;
    p.B = d->B;
    p.S = d->S;
    p.out_w = d->out_w;
    p.err = d->err;
    mlp::train_backward_kernel<<<d->B / 128, mlp::TR_THREADS, mlp::TR_SMEM, s>>>(p);
    if ((st = mlp_cuda(cudaGetLastError(), "train_backward_kernel launch")) != CTL_OK) return st;
    mlp::WgPlan plan;
    plan.first[0] = 0;
    for (int l = 0; l < mlp::TR_L; l++) plan.first[l + 1] = plan.first[l] + mlp::wg_ctas(l, d->B / 128, sms);
    mlp::train_wgrad_kernel<<<plan.first[mlp::TR_L], mlp::TR_THREADS, mlp::WG_SMEM, s>>>(p, plan);
    return mlp_cuda(cudaGetLastError(), "train_wgrad_kernel launch");
}

extern "C" ctl_status ctl_mlp_adam_step(const ctl_mlp_adam_desc* d, void* stream) {
    if (!d || d->step <= 0 || (d->out_w != 64 && d->out_w != 128)) return CTL_ERR_ARG;
    mlp::AdamAll p = {};
    for (int l = 0; l < mlp::TR_L; l++) {
        if (!d->w[l] || !d->g[l] || !d->m[l] || !d->v[l] || !d->b[l] || !d->gb[l] || !d->mb[l] || !d->vb[l] || !d->wb[l] ||
            !d->wbT[l])
            return CTL_ERR_ARG;
        const int rows = l == 4 ? d->out_w : 256, cols = l == 0 ? 64 : 256;
        p.w[l] = d->w[l]; p.m1[l] = d->m[l]; p.m2[l] = d->v[l]; p.g[l] = d->g[l];
        p.w[5 + l] = d->b[l]; p.m1[5 + l] = d->mb[l]; p.m2[5 + l] = d->vb[l]; p.g[5 + l] = d->gb[l];
        p.wb[l] = static_cast<__nv_bfloat16*>(d->wb[l]);
        p.wbT[l] = static_cast<__nv_bfloat16*>(d->wbT[l]);
        p.rows[l] = rows; p.cols[l] = cols;
        p.rows[5 + l] = 1; p.cols[5 + l] = rows;
    }
    p.lr = d->lr; p.b1 = d->beta1; p.b2 = d->beta2; p.eps = d->eps; p.wd = d->weight_decay;
    p.c1 = 1.0f - powf(d->beta1, (float)d->step);
    p.c2 = 1.0f - powf(d->beta2, (float)d->step);
    mlp::train_adam_kernel<<<dim3(64, 2 * mlp::TR_L), 256, 0, static_cast<cudaStream_t>(stream)>>>(p);
    return mlp_cuda(cudaGetLastError(), "train_adam_kernel launch");
}
