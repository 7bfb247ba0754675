// One optimiser step of the surrogate MLP in four kernels (included by
// ctl_mlp.cu after its GEMM helpers): the forward pass of all five layers, the
// loss gradient with the data gradients of all layers, the weight gradients of
// all layers, and Adam on every parameter.
//
// The batch is cut into tiles of 128 rows.  A CTA of the forward or backward
// kernel keeps its tile's activations (or gradients) in shared memory from
// layer to layer as the next layer's A operand, so that HBM and L2 see only
// what the backward pass needs: the FP32 pre-activations and, transposed, the
// BF16 activations and gradients.  Those are written in the order in which the
// weight-gradient kernel's MMAs read them ("packed": per 128-row tile, chunks
// of 8 batch rows by 8 features as the 8-row x 16-byte core matrices of the
// canonical no-swizzle K-major layout), so that its loads are plain contiguous
// bulk copies.  Every mbarrier wait is bounded and raises the error word.
//
// One B200, batch 16,384, 32 species: a step of forward, backward and Adam took
// 874 us as 40 launches (a GEMM per product with transposes written 2 bytes at
// a time, a serial column sum of 108 us per layer, Adam per tensor); here 124
// us as 7 (140 before the pre-activations lay in the order of the lanes that
// store and load them, and y and the target were read by whole lines).  Bound:
// the 280 MB that pre-activations, activations and gradients make between the
// kernels (43 us at the copy rate; 140 MB live, a little more than L2), then
// the chain of a tile's five layers.
#pragma once

#include "ctl_train_plan.h"

namespace ctl {
namespace mlp {

constexpr int IN_W = 64;                          // input width
constexpr int TR_EPI = 256, TR_THREADS = TR_EPI + 64;
constexpr int TR_STAGES = 5;                      // weight stages of 32 K-columns
constexpr int TR_A_BYTES = 128 * SC_HID * 2;
constexpr int TR_SMEM = TR_A_BYTES + TR_STAGES * SC_STAGE_BYTES + (4 * SC_HID + 128) * 4;

struct Train {
    const __nv_bfloat16* X;      // [B][64]
    const uint8_t* wpack;        // forward weights, stages of 32 K-columns
    const uint8_t* wtpack;       // backward weights (W^T of layers 4, 3, 2, 1)
    const float* bias[TR_L];
    float* z[4];                 // [B][256] pre-activations, in the order of z_at
    float* y;                    // [B][out_w]
    uint8_t* hp[TR_L];           // packed transposed inputs of each layer: [0] X, [l] the activations of layer l - 1; or null
    uint8_t* dp[TR_L];           // packed transposed gradients of each layer's output ([4]: 128 rows)
    const float* target;         // [B][S]
    float* loss;                 // [1]
    float* dW[TR_L];             // [N][K], accumulated
    float* db[TR_L];
    int B, S, out_w;
    unsigned* err;
};

__device__ __forceinline__ void st8(float* p, const float (&v)[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
                 "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}
__device__ __forceinline__ void ld8(const float* p, float (&v)[8]) {
    asm volatile("ld.global.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void tr_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ bool tr_all(bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred a, b;\n\t"
        "setp.ne.u32 a, %1, 0;\n\t"
        "bar.red.and.pred b, 1, 256, a;\n\t"
        "selp.u32 %0, 1, 0, b;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v)
        : "memory");
    return r != 0;
}

// A tile's columns [0, cols) as packed transposed rows, and their column sums
// added to `sums` (or null): the 8 epilogue warps take 8 columns each in turn.
// ldmatrix with transposition reads four 8 x 8 core matrices' worth of rows,
// chosen so that a lane receives 8 consecutive rows of one column: one 16-byte
// store, eight neighbouring lanes 128 contiguous bytes.
__device__ __forceinline__ void tile_transpose(uint32_t a, int cols, int prows, uint8_t* out, float* sums, int warp,
                                               int lane) {
    const int i = lane >> 3, k = lane & 7;
    for (int kb = warp; kb < cols / 8; kb += 8) {
        float s = 0.0f;
#pragma unroll
        for (int rb = 0; rb < 4; rb++) {
            const int row = rb * 32 + 8 * (k >> 1) + 2 * i + (k & 1);
            uint32_t r[4];
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                         : "r"(a + canon(row, kb * 8, 128))
                         : "memory");
            // column kb * 8 + lane / 4, rows rb * 32 + 8 (lane % 4) ..
            const int n = kb * 8 + (lane >> 2), b8 = rb * 4 + (lane & 3);
            if (out) *reinterpret_cast<uint4*>(out + (size_t)(b8 * (prows >> 3) + (n >> 3)) * 128 + (n & 7) * 16) =
                make_uint4(r[0], r[1], r[2], r[3]);
            if (sums)
#pragma unroll
                for (int q = 0; q < 4; q++)
                    s += __uint_as_float(r[q] << 16) + __uint_as_float(r[q] & 0xffff0000u);
        }
        if (sums) {
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if ((lane & 3) == 0) atomicAdd(sums + kb * 8 + (lane >> 2), s);
        }
    }
}

// Where a lane of an epilogue warp keeps its part of a tile's pre-activations:
// 16 groups of 8 columns of its row, each group next to its neighbour lanes'
// (a warp's 32-byte stores then fill 8 lines, where rows 1 KB apart touched 32).
__device__ __forceinline__ size_t z_at(int warp, int lane) {
    return ((size_t)(blockIdx.x * 8 + warp) * 16 * 32 + lane) * 8;
}

// Barriers and TMEM of a forward or backward CTA.
struct TrShared {
    uint64_t full[TR_STAGES], empty[TR_STAGES], acc, ready, drain;
    uint32_t tmem;
    int abort;
};

__device__ __forceinline__ void tr_init(TrShared& sh, int warp) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < TR_STAGES; i++) {
            mbar_init(&sh.full[i], 1);
            mbar_init(&sh.empty[i], 1);
        }
        mbar_init(&sh.acc, 1);
        mbar_init(&sh.ready, TR_EPI / 32);
        mbar_init(&sh.drain, 1);
        sh.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)),
                     "r"(SC_HID));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
}

// The weight stream and the MMAs of a chain of products: product i has N
// columns and K(i) / 32 stages.  Warp 8 copies the stages, warp 9 issues the
// MMAs of product i once the epilogue has announced its A operand.
template <class NF, class KF>
__device__ __forceinline__ void tr_produce(TrShared& sh, uint8_t* stage, const uint8_t* w, int products, NF&& N, KF&& K,
                                           unsigned* err) {
    uint32_t idx = 0, issued = 0;
    bool ok = true;
    size_t off = 0;
    for (int l = 0; l < products && ok; l++) {
        const uint32_t bytes = (uint32_t)(N(l) * SC_BK * 2);
        for (int ks = 0; ks < K(l) / SC_BK; ks++, idx++) {
            const uint32_t sl = idx % TR_STAGES, round = idx / TR_STAGES;
            if (round > 0 && !mbar_wait_u(&sh.empty[sl], (round - 1) & 1u, err)) { ok = false; break; }
            if (raised(&sh.abort)) { ok = false; break; }
            if (elect_one()) {
                mbar_expect_tx(&sh.full[sl], bytes);
                bulk_g2s(stage + sl * SC_STAGE_BYTES, w + off, bytes, &sh.full[sl]);
            }
            issued = idx + 1;
            off += bytes;
        }
    }
    if (!ok) {
        if (elect_one()) atomicExch(&sh.abort, 1);
        // let the copies in flight land before the CTA exits
        for (uint32_t i = issued > TR_STAGES ? issued - TR_STAGES : 0u; i < issued; i++)
            mbar_wait_u(&sh.full[i % TR_STAGES], (i / TR_STAGES) & 1u, nullptr);
    }
}

template <class NF, class KF>
__device__ __forceinline__ void tr_mma(TrShared& sh, uint32_t stage, uint32_t a, uint32_t tmem, int products, NF&& N,
                                       KF&& K, unsigned* err) {
    uint32_t idx = 0;
    bool ok = true;
    for (int l = 0; l < products && ok; l++) {
        if (!mbar_wait_u(&sh.ready, (uint32_t)l & 1u, err) || raised(&sh.abort)) { ok = false; break; }
        tc_fence_after();
        const int n = N(l);
        const uint32_t idesc = make_idesc(128, n);
        const uint32_t kstep = (uint32_t)(2 * (n / 8) * 128), lbo = (uint32_t)((n / 8) * 128);
        for (int ks = 0; ks < K(l) / SC_BK; ks++, idx++) {
            const uint32_t sl = idx % TR_STAGES, round = idx / TR_STAGES;
            if (!mbar_wait_u(&sh.full[sl], round & 1u, err)) { ok = false; break; }
            tc_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < SC_BK / 16; kk++)
                    mma_bf16(tmem, make_desc(a + (uint32_t)(ks * 4 + kk * 2) * 16u * 128u, 16u * 128u, 128u),
                             make_desc(stage + sl * SC_STAGE_BYTES + (uint32_t)kk * kstep, lbo, 128u), idesc,
                             (ks > 0 || kk > 0) ? 1u : 0u);
                mma_commit(&sh.empty[sl]);
            }
        }
        if (ok && elect_one()) mma_commit(&sh.acc);
    }
    if (!ok && elect_one()) atomicExch(&sh.abort, 1);
    if (elect_one()) mma_commit(&sh.drain);  // every MMA this warp issued has completed once drain flips
    mbar_wait_u(&sh.drain, 0u, nullptr);
}

__device__ __forceinline__ void tr_finish(uint32_t tmem, int warp) {
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(SC_HID));
}

// Forward: X -> four hidden layers -> y, one CTA per 128 rows.  Per layer the
// 8 epilogue warps (rows 32 (warp % 4).., column half warp / 4) add the bias,
// store the FP32 pre-activation (32-byte stores), round SiLU to BF16 into the
// next layer's A operand, and, while that layer's MMAs run, write its packed
// transpose.
__global__ void __launch_bounds__(TR_THREADS, 1) train_forward_kernel(const __grid_constant__ Train p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) TrShared sh;
    uint8_t* A = smem;
    uint8_t* stage = smem + TR_A_BYTES;
    float* c_bias = reinterpret_cast<float*>(stage + TR_STAGES * SC_STAGE_BYTES);
    const int warp = warp_index(), lane = threadIdx.x % 32;
    for (int i = threadIdx.x; i < 4 * SC_HID + p.out_w; i += TR_THREADS)
        c_bias[i] = p.bias[i / SC_HID < 4 ? i / SC_HID : 4][i < 4 * SC_HID ? i % SC_HID : i - 4 * SC_HID];
    tr_init(sh, warp);
    const uint32_t tmem = sh.tmem;
    const int out_w = p.out_w;
    auto N = [&](int l) { return l == TR_L - 1 ? out_w : SC_HID; };
    auto K = [](int l) { return l == 0 ? IN_W : SC_HID; };
    if (warp == 8) {
        tr_produce(sh, stage, p.wpack, TR_L, N, K, p.err);
    } else if (warp == 9) {
        tr_mma(sh, smem_u32(stage), smem_u32(A), tmem, TR_L, N, K, p.err);
    } else {
        const int q = warp & 3, h = warp >> 2, r = q * 32 + lane;
        const size_t row = (size_t)blockIdx.x * 128 + r;
        const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16);
#pragma unroll
        for (int i = 0; i < 4; i++) {  // eight lanes a row: whole lines
            const int xr = 32 * i + (int)threadIdx.x / 8, xc = 8 * ((int)threadIdx.x % 8);
            *reinterpret_cast<uint4*>(A + canon(xr, xc, 128)) =
                *reinterpret_cast<const uint4*>(p.X + ((size_t)blockIdx.x * 128 + xr) * IN_W + xc);
        }
        fence_async_smem();
        mbar_arrive_warp(&sh.ready);
        if (p.hp[0]) {
            tr_sync();
            tile_transpose(smem_u32(A), IN_W, IN_W, p.hp[0] + (size_t)blockIdx.x * 128 * IN_W * 2, nullptr, warp, lane);
        }
        for (int l = 0; l < TR_L; l++) {
            bool got = mbar_wait(&sh.acc, (uint32_t)l & 1u, p.err);
            if (!tr_all(got && !*(volatile int*)&sh.abort)) {
                atomicExch(&sh.abort, 1);
                break;
            }
            tc_fence_after();
            const float* b = c_bias + l * SC_HID;
            const int width = N(l), c0 = h * (width / 2), nc = width / 64;  // 32-column chunks of this half
            float* zout = l < TR_L - 1 ? p.z[l] + z_at(warp, lane) : p.y + row * width + c0;
            const int zstep = l < TR_L - 1 ? 256 : 8;
            uint32_t ra[32], rb[32];
            tmem_ld32_issue(tbase + (uint32_t)c0, ra);
#pragma unroll 1
            for (int j = 0; j < nc; j += 2) {
#pragma unroll
                for (int u = 0; u < 2; u++) {  // two chunks per trip, the next load in flight
                    if (j + u >= nc) break;
                    tmem_wait();
                    uint32_t(&cur)[32] = u ? rb : ra;
                    if (j + u + 1 < nc) tmem_ld32_issue(tbase + (uint32_t)(c0 + 32 * (j + u + 1)), u ? ra : rb);
                    const int c = c0 + 32 * (j + u);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float4 ba = *reinterpret_cast<const float4*>(b + c + 8 * k);
                        const float4 bb = *reinterpret_cast<const float4*>(b + c + 8 * k + 4);
                        const float bias[8] = {ba.x, ba.y, ba.z, ba.w, bb.x, bb.y, bb.z, bb.w};
                        float z[8];
#pragma unroll
                        for (int e = 0; e < 8; e++) z[e] = __uint_as_float(cur[8 * k + e]) + bias[e];
                        st8(zout + (4 * (j + u) + k) * zstep, z);
                        if (l < TR_L - 1) {
                            uint4 o;
                            o.x = pack_bf2(silu(z[0]), silu(z[1]));
                            o.y = pack_bf2(silu(z[2]), silu(z[3]));
                            o.z = pack_bf2(silu(z[4]), silu(z[5]));
                            o.w = pack_bf2(silu(z[6]), silu(z[7]));
                            *reinterpret_cast<uint4*>(A + canon(r, c + 8 * k, 128)) = o;
                        }
                    }
                }
            }
            if (l < TR_L - 1) {
                fence_async_smem();
                tc_fence_before();
                mbar_arrive_warp(&sh.ready);
                if (p.hp[l + 1]) {
                    tr_sync();
                    tile_transpose(smem_u32(A), SC_HID, SC_HID, p.hp[l + 1] + (size_t)blockIdx.x * TR_A_BYTES, nullptr,
                                   warp, lane);
                }
            }
        }
    }
    tr_finish(tmem, warp);
}

// Backward: the loss gradient of the tile's rows (Gaussian negative
// log-likelihood, as nll_grad_kernel), then layer by layer
// dz[l] = (dz[l + 1] W[l + 1]) * silu'(z[l]); every gradient leaves as its
// packed transpose with its column sums (the bias gradients) taken on the way.
__global__ void __launch_bounds__(TR_THREADS, 1) train_backward_kernel(const __grid_constant__ Train p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) TrShared sh;
    uint8_t* A = smem;
    uint8_t* stage = smem + TR_A_BYTES;
    const int warp = warp_index(), lane = threadIdx.x % 32;
    tr_init(sh, warp);
    const uint32_t tmem = sh.tmem;
    const int out_w = p.out_w;
    auto N = [](int) { return SC_HID; };
    auto K = [&](int i) { return i == 0 ? out_w : SC_HID; };
    if (warp == 8) {
        tr_produce(sh, stage, p.wtpack, 4, N, K, p.err);
    } else if (warp == 9) {
        tr_mma(sh, smem_u32(stage), smem_u32(A), tmem, 4, N, K, p.err);
    } else {
        const int q = warp & 3, h = warp >> 2, r = q * 32 + lane;
        const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16);
        {
            // a warp's lanes take a row's species side by side (whole lines of y
            // and target; a lane per row touched 32 lines with each load)
            const int S = p.S;
            const float sc = 1.0f / ((float)p.B * (float)S);
            float l = 0.0f;
            auto put = [&](int rr, int c, float v) {
                *reinterpret_cast<__nv_bfloat16*>(A + canon(rr, c, 128)) = __float2bfloat16(v);
            };
#pragma unroll 4
            for (int rr = warp; rr < 128; rr += 8) {
                const float* y = p.y + ((size_t)blockIdx.x * 128 + rr) * out_w;
                const float* tg = p.target + ((size_t)blockIdx.x * 128 + rr) * S;
                for (int k = lane; k < S; k += 32) {
                    const float mu = y[k];
                    float lv = y[S + k];
                    lv = fminf(fmaxf(lv, -12.0f), 12.0f);
                    const float iv = __expf(-lv);
                    const float d = tg[k] - mu;
                    l += 0.5f * (lv + d * d * iv);
                    put(rr, k, -d * iv * sc);
                    put(rr, S + k, 0.5f * (1.0f - d * d * iv) * sc);
                }
                for (int k = 2 * S + lane; k < out_w; k += 32) put(rr, k, 0.0f);
            }
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (lane == 0 && l != 0.0f) atomicAdd(p.loss, l);
        }
        fence_async_smem();
        mbar_arrive_warp(&sh.ready);
        tr_sync();
        tile_transpose(smem_u32(A), out_w, 128, p.dp[4] + (size_t)blockIdx.x * 128 * 128 * 2, p.db[4], warp, lane);
        for (int i = 0; i < 4; i++) {
            const int l = 3 - i;
            const float* zin = p.z[l] + z_at(warp, lane);
            float z[2][4][8];  // a chunk's pre-activations, loaded a chunk ahead
#pragma unroll
            for (int k = 0; k < 4; k++) ld8(zin + k * 256, z[0][k]);
            bool got = mbar_wait(&sh.acc, (uint32_t)i & 1u, p.err);
            if (!tr_all(got && !*(volatile int*)&sh.abort)) {
                atomicExch(&sh.abort, 1);
                break;
            }
            tc_fence_after();
            const int c0 = 128 * h;
            uint32_t ra[32], rb[32];
            tmem_ld32_issue(tbase + (uint32_t)c0, ra);
#pragma unroll 1
            for (int j = 0; j < 4; j += 2) {
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int c = c0 + 32 * (j + u);
                    if (j + u + 1 < 4)
#pragma unroll
                        for (int k = 0; k < 4; k++) ld8(zin + (4 * (j + u + 1) + k) * 256, z[u ^ 1][k]);
                    tmem_wait();
                    uint32_t(&cur)[32] = u ? rb : ra;
                    if (j + u + 1 < 4) tmem_ld32_issue(tbase + (uint32_t)(c + 32), u ? ra : rb);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        float d[8];
#pragma unroll
                        for (int e = 0; e < 8; e++) d[e] = __uint_as_float(cur[8 * k + e]) * silu_grad(z[u][k][e]);
                        *reinterpret_cast<uint4*>(A + canon(r, c + 8 * k, 128)) = make_uint4(
                            pack_bf2(d[0], d[1]), pack_bf2(d[2], d[3]), pack_bf2(d[4], d[5]), pack_bf2(d[6], d[7]));
                    }
                }
            }
            fence_async_smem();
            tc_fence_before();
            if (l > 0) mbar_arrive_warp(&sh.ready);
            tr_sync();
            tile_transpose(smem_u32(A), SC_HID, SC_HID, p.dp[l] + (size_t)blockIdx.x * TR_A_BYTES, p.db[l], warp, lane);
        }
    }
    tr_finish(tmem, warp);
}

// Weight gradients of all layers: dW[l] += dz[l]^T h[l - 1], the batch as the
// contraction.  A CTA takes a share of one layer's 128-row tiles and holds the
// whole [256][K] product in TMEM (two M = 128 halves); per stage it copies 32
// batch rows of both packed operands.  Shares are sized by the layers' MMAs
// (layer 0 has K = 64, the last one half the rows).  A chain of MMA
// accumulations rounds towards zero at each step, so a share's tiles are cut
// into as many chains as accumulators fit into TMEM (four of layer 0, two of
// the last), which the epilogue adds up; ctl_train_plan.h bounds their length.
// The sums meet in L2 by vector reductions.
constexpr int WG_STAGES = 6;
constexpr int WG_STAGE_BYTES = 2 * 32 * SC_HID * 2;
constexpr int WG_SMEM = WG_STAGES * WG_STAGE_BYTES;
struct WgPlan {
    int first[TR_L + 1];  // CTAs of layer l: [first[l], first[l + 1])
};

__global__ void __launch_bounds__(TR_THREADS, 1) train_wgrad_kernel(const __grid_constant__ Train p, WgPlan plan) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[WG_STAGES], empty[WG_STAGES], done;
    __shared__ uint32_t tmem_slot;
    const int warp = warp_index(), lane = threadIdx.x % 32;
    int l = 0;
    while ((int)blockIdx.x >= plan.first[l + 1]) l++;
    const int part = (int)blockIdx.x - plan.first[l], parts = plan.first[l + 1] - plan.first[l];
    const int tiles = p.B / 128;
    const int t0 = (int)((int64_t)tiles * part / parts), t1 = (int)((int64_t)tiles * (part + 1) / parts);
    const int arows = l == 4 ? 128 : SC_HID;         // packed rows of dz
    const int mrows = l == 4 ? p.out_w : SC_HID;     // of them in dW
    const int N = l == 0 ? IN_W : SC_HID;            // columns of dW
    const int halves = arows / 128;
    const uint32_t abytes = (uint32_t)(32 * arows * 2), bbytes = (uint32_t)(32 * N * 2);
    const int steps = (t1 - t0) * 4, chains = min(wg_chains(l), t1 - t0);
    const uint32_t acols = l == 0 ? IN_W : SC_HID;   // TMEM columns between a half's accumulators
    if (threadIdx.x == 0) {
        for (int i = 0; i < WG_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(2 * SC_HID));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = true;
    if (warp == 8) {
        int issued = 0;
        for (int i = 0; i < steps && ok; i++) {
            const int s = i % WG_STAGES, round = i / WG_STAGES;
            if (round > 0) ok = mbar_wait_u(&empty[s], (uint32_t)(round - 1) & 1u, p.err);
            if (!ok) break;
            uint8_t* dst = smem + (size_t)s * WG_STAGE_BYTES;
            const size_t tile = (size_t)(t0 + i / 4), sub = (size_t)(i & 3);
            if (elect_one()) {
                mbar_expect_tx(&full[s], abytes + bbytes);
                bulk_g2s(dst, p.dp[l] + tile * 4 * abytes + sub * abytes, abytes, &full[s]);
                bulk_g2s(dst + WG_STAGE_BYTES / 2, p.hp[l] + tile * 4 * bbytes + sub * bbytes, bbytes, &full[s]);
            }
            issued = i + 1;
        }
        if (!ok)  // the copies in flight land before the CTA exits
            for (int i = issued > WG_STAGES ? issued - WG_STAGES : 0; i < issued; i++)
                mbar_wait_u(&full[i % WG_STAGES], (uint32_t)(i / WG_STAGES) & 1u, nullptr);
    } else if (warp == 9) {
        const uint32_t idesc = make_idesc(128, N);
        int chain = -1;
        for (int i = 0; i < steps && ok; i++) {
            const int s = i % WG_STAGES, round = i / WG_STAGES, c = i / 4 * chains / (t1 - t0);
            const bool add = c == chain;  // else the chain's first product
            chain = c;
            ok = mbar_wait_u(&full[s], (uint32_t)round & 1u, p.err);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a = smem_u32(smem + (size_t)s * WG_STAGE_BYTES), b = a + WG_STAGE_BYTES / 2;
            if (elect_one()) {
#pragma unroll
                for (int kk = 0; kk < 2; kk++) {
                    const uint64_t db = make_desc(b + (uint32_t)(kk * 2 * (N / 8) * 128), (uint32_t)((N / 8) * 128), 128u);
                    for (int m = 0; m < halves; m++)
                        mma_bf16(tmem + (uint32_t)(m * SC_HID) + (uint32_t)c * acols,
                                 make_desc(a + (uint32_t)(kk * 2 * (arows / 8) * 128 + m * 16 * 128),
                                           (uint32_t)((arows / 8) * 128), 128u),
                                 db, idesc, (add || kk > 0) ? 1u : 0u);
                }
                mma_commit(&empty[s]);
            }
        }
        if (elect_one()) mma_commit(&done);
    }
    // (on a timeout the products are not used; the MMAs issued still end first)
    ok = mbar_wait(&done, 0u, p.err) && ok;
    ok = __syncthreads_and(ok) != 0;
    tc_fence_after();
    if (ok && warp < 8 && steps > 0) {
        const int q = warp & 3;
        for (int m = 0; m < halves; m++) {
            const int n = m * 128 + q * 32 + lane;  // row of dW
            for (int c = (warp >> 2) * 32; c < N; c += 64) {
                float v[32];
                const uint32_t at = tmem + (uint32_t)(m * SC_HID) + ((uint32_t)(q * 32) << 16) + (uint32_t)c;
                tmem_ld32(at, v);
                for (int a = 1; a < chains; a++) {
                    float u[32];
                    tmem_ld32(at + (uint32_t)a * acols, u);
#pragma unroll
                    for (int k = 0; k < 32; k++) v[k] += u[k];
                }
                if (n < mrows)
#pragma unroll
                    for (int k = 0; k < 32; k += 4)
                        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p.dW[l] + (size_t)n * N + c + k),
                                     "f"(v[k]), "f"(v[k + 1]), "f"(v[k + 2]), "f"(v[k + 3])
                                     : "memory");
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * SC_HID));
}

// Weight matrices W [N][K] into K-stages of 32 columns in the canonical
// layout, several matrices in one launch (grid.y), 16 bytes per thread.
struct Pack {
    const __nv_bfloat16* w[TR_L];
    int ld[TR_L], n[TR_L], k[TR_L];
    size_t off[TR_L];  // bytes
    uint8_t* out;
};
__global__ void train_pack_kernel(const __grid_constant__ Pack p) {
    const int l = blockIdx.y, N = p.n[l], K = p.k[l];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;  // 8 columns of one row
    if (i >= N * (K / 8)) return;
    const int n = i / (K / 8), k = i % (K / 8) * 8;
    *reinterpret_cast<uint4*>(p.out + p.off[l] + (size_t)(k / SC_BK) * N * SC_BK * 2 + canon(n, k % SC_BK, N)) =
        *reinterpret_cast<const uint4*>(p.w[l] + (size_t)n * p.ld[l] + k);
}

// One Adam step on every weight matrix and bias vector (grid.y: matrices, then
// biases), with the arithmetic of adam_kernel; 32 x 32 tiles of a matrix, so
// that its BF16 copy and its transposed BF16 copy are both written in rows.
struct AdamAll {
    float *w[2 * TR_L], *m1[2 * TR_L], *m2[2 * TR_L];
    const float* g[2 * TR_L];
    __nv_bfloat16 *wb[TR_L], *wbT[TR_L];
    int rows[2 * TR_L], cols[2 * TR_L];
    float lr, b1, b2, eps, c1, c2, wd;
};
__global__ void __launch_bounds__(256) train_adam_kernel(const __grid_constant__ AdamAll p) {
    __shared__ __nv_bfloat16 t[32][33];
    const int l = blockIdx.y, rows = p.rows[l], cols = p.cols[l];
    const int tc = (cols + 31) / 32, r0 = (int)(blockIdx.x / tc) * 32, c0 = (int)(blockIdx.x % tc) * 32;
    if (r0 >= rows) return;
    const int x = threadIdx.x % 32, y0 = threadIdx.x / 32;
    const float wd = l < TR_L ? p.wd : 0.0f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int r = r0 + y0 + 8 * j, c = c0 + x;
        if (r >= rows || c >= cols) continue;
        const size_t i = (size_t)r * cols + c;
        const float w0 = p.w[l][i];
        const float gi = p.g[l][i] + wd * w0;
        const float a = p.b1 * p.m1[l][i] + (1.0f - p.b1) * gi;
        const float b = p.b2 * p.m2[l][i] + (1.0f - p.b2) * gi * gi;
        p.m1[l][i] = a;
        p.m2[l][i] = b;
        const float wi = w0 - p.lr * (a / p.c1) / (sqrtf(b / p.c2) + p.eps);
        p.w[l][i] = wi;
        if (l < TR_L) {
            const __nv_bfloat16 hb = __float2bfloat16(wi);
            p.wb[l][i] = hb;
            t[y0 + 8 * j][x] = hb;
        }
    }
    if (l >= TR_L) return;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int c = c0 + y0 + 8 * j, r = r0 + x;
        if (c < cols && r < rows) p.wbT[l][(size_t)c * rows + r] = t[x][y0 + 8 * j];
    }
}

}  // namespace mlp
}  // namespace ctl
