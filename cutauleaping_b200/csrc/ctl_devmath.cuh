// Device arithmetic shared by every sweep kernel and by the model-specialised
// kernels compiled at run time (NVRTC): the random stream, the elementary
// functions, the Poisson sampler, Cao's g_i, the sum-tree step and the run
// parameters.  Self-contained: under NVRTC it needs no host header.
//
// Determinism contract (what makes any launch shape give identical bits):
//   * every random word comes from Philox4x32-10 with key = seed and counter
//     (block, tag, step, sim): a draw depends on which simulation, which step
//     and what it is for, never on which thread computes it;
//   * every FP64 sum over reactions is the root of a fixed binary tree over
//     the reactions padded to P = 2^k leaves, and the searches descend it;
//   * the elementary functions are this file's own (no CUDA math library
//     calls on the path), so the CPU oracle (oracle/ctl_oracle.c) computes
//     the same bits.
// Built with -fmad=false: no implicit FMA contraction; fma() is called
// explicitly where it is meant.
#pragma once

#ifdef __CUDACC_RTC__
typedef unsigned char uint8_t;
typedef signed char int8_t;
typedef unsigned short uint16_t;
typedef int int32_t;
typedef unsigned int uint32_t;
typedef long long int64_t;
typedef unsigned long long uint64_t;
typedef unsigned long size_t;
typedef unsigned long uintptr_t;
#define FLT_MAX 3.402823466e+38F
// The per-simulation record of include/ctl.h (same layout).
typedef struct {
    double t_final;
    uint64_t firings;
    uint32_t status;
    uint32_t steps, leaps, ssa_steps, rejections, pad;
} ctl_sim_info;
enum { CTL_SIM_OK = 0, CTL_SIM_STEP_LIMIT = 1, CTL_SIM_OVERFLOW = 2, CTL_SIM_ATTEMPT_LIMIT = 3 };
#else
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>

#include "../../include/ctl.h"
#endif

namespace ctl {
namespace dev {

constexpr uint32_t TAG_SSA = 0x40000000u;   // SSA steps 2b, 2b+1: block b, (w0,w1) / (w2,w3)
constexpr uint32_t TAG_MISC = 0x40000001u;  // leap: (w0,w1) tau2, (w2,w3) critical pick
constexpr uint32_t MAX_ATTEMPTS = 1024u;    // 10-bit attempt field of the Poisson tag
constexpr uint32_t PTRS_MAX_TRIALS = 256u;

enum : uint32_t {
    F_FORCE_SSA = 1u << 0, F_Q1_OFF = 1u << 1, F_Q2_OFF = 1u << 2, F_Q3_OFF = 1u << 3,
    F_Q4_OFF = 1u << 4, F_Q5_OFF = 1u << 5, F_Q6_OFF = 1u << 6, F_Q9_OFF = 1u << 7, F_Q10_OFF = 1u << 8
};

__device__ __forceinline__ uint32_t tag_pois(uint32_t attempt, uint32_t pair) {
    return 0x80000000u | (attempt << 20) | pair;
}

struct Run {
    uint64_t seed;
    float eps;
    uint32_t nc;
    double ssa_factor;
    uint32_t ssa_steps, flags, max_steps, sim_base, n;
    uint32_t uniform_c;              // all simulations share row 0 of c
    uint32_t ssa_budget, dec_budget; // work per slot and round (SSA steps / decisions)
    uint32_t warp_local;             // 1: warp-local scheduling (no block rounds)
    uint32_t tail_sims;              // register-resident block rounds: live simulations at or
                                     // below which a block with a closed queue finishes them in
                                     // warp lockstep (0: never)
    unsigned long long* sums;        // fitness mode: [sets][ns][s_out] sample sums, else null
    uint32_t sum_threads, sum_prep;  // simulation -> parameter set (the reference's layout)
    uint32_t* done;                  // optional: finished simulations per chunk of 2^done_shift
    uint32_t* out_host;              // optional: the caller's pinned rows [n][ns][s_out] (device view);
                                     // each finished row is copied there by the kernel
    uint32_t done_shift;
    const int32_t* __restrict__ X0;  // [n][S]
    const float* __restrict__ c;     // [n][R]
    uint32_t* __restrict__ out;      // [n][ns][s_out]
    ctl_sim_info* __restrict__ info; // [n]
    uint32_t* queue;                 // work-queue ticket
};


// ---------------------------------------------------------------------------
// Random numbers and elementary functions (bitwise identical to the oracle)
// ---------------------------------------------------------------------------

template <int UNROLL = 10>
__device__ __forceinline__ uint4 philox10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll UNROLL
    for (int i = 0; i < 10; i++) {
        uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
        uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
        c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

__device__ __forceinline__ uint4 draw(uint64_t seed, uint32_t blk, uint32_t tag, uint32_t step,
                                      uint32_t sim) {
    return philox10(make_uint4(blk, tag, step, sim), (uint32_t)seed, (uint32_t)(seed >> 32));
}

// The same block from half the code, for callers whose loops the instruction
// cache would otherwise not hold (the shared-memory sweep's leap: 64 x 128
// network on one B200, 253 -> 242 ms).
__device__ __forceinline__ uint4 draw_small(uint64_t seed, uint32_t blk, uint32_t tag, uint32_t step, uint32_t sim) {
    return philox10<5>(make_uint4(blk, tag, step, sim), (uint32_t)seed, (uint32_t)(seed >> 32));
}

__device__ __forceinline__ double u32d(uint32_t w) { return ((double)w + 0.5) * 0x1p-32; }
__device__ __forceinline__ double u53(uint32_t wa, uint32_t wb) {
    uint64_t m = ((uint64_t)wb << 20) | (uint64_t)(wa >> 12);
    return ((double)m + 0.5) * 0x1p-52;
}

// Correctly rounded quotients and roots in straight-line code (Markstein
// 1990): the approximate reciprocal is refined until it is the rounded one,
// and the quotient corrected by its exact remainder; a root likewise from the
// approximate reciprocal root (Goldschmidt's two products).  A general division's
// test for special operands and the call behind it end the code that the
// scheduler can overlap: without them an exact step of a lone Schlogl
// simulation takes 0.29 instead of 0.50 us, and 65,537 perturbed simulations,
// with many PTRS draws, 73 instead of 81 ms.  For operands whose reciprocal,
// quotient and remainder stay in the normal range (the callers'), a = 0
// included.  A divisor whose significand is all ones is the one that refines to
// a neighbour of its rounded reciprocal; some quotients by it (a power of two
// above it) are then the lower neighbour.
__device__ __forceinline__ float div_near(float a, float b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    y = fmaf(fmaf(-b, y, 1.0f), y, y);
    y = fmaf(fmaf(-b, y, 1.0f), y, y);
    const float q = a * y;
    return fmaf(fmaf(-b, q, a), y, q);
}

__device__ __forceinline__ double div_near(double a, double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    y = fma(fma(-b, y, 1.0), y, y);
    y = fma(fma(-b, y, 1.0), y, y);
    y = fma(fma(-b, y, 1.0), y, y);
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

__device__ __forceinline__ double sqrt_near(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const double r = fma(-g, h, 0.5);
        g = fma(g, r, g);
        h = fma(h, r, h);
    }
    return fma(fma(-g, g, x), h, g);
}

// Whether div_near divides by b exactly as `/` for any a that is 0 or within
// 2^-30 .. 2^60 (num_fits: 0 or 2^-30 <= |a| < 2^30).
__device__ __forceinline__ bool div_fits(float b) {
    const uint32_t u = __float_as_uint(b) & 0x7fffffffu;
    return u - 0x21800000u < 0x5d800000u - 0x21800000u && (u & 0x7fffffu) != 0x7fffffu;  // 2^-60 <= |b| < 2^60
}
__device__ __forceinline__ bool num_fits(float a) {
    const uint32_t u = __float_as_uint(a) & 0x7fffffffu;
    return u == 0u || u - 0x30800000u < 0x4e800000u - 0x30800000u;
}

#define CTL_LN2_HI 0x1.62e42fee00000p-1
#define CTL_LN2_LO 0x1.a39ef35793c76p-33

// log(x) = e ln2 + 2 atanh(s), s = (m-1)/(m+1), m in (sqrt(1/2), sqrt(2)], of
// N positive normal numbers at once: the polynomials' steps interleave, so
// that N logarithms take little longer than one.
template <int N>
__device__ __forceinline__ void dlog_of(const double (&x)[N], double (&out)[N], int eadj = 0) {
    double ed[N], s[N], z[N], p[N];
#pragma unroll
    for (int i = 0; i < N; i++) {
        const uint64_t b = (uint64_t)__double_as_longlong(x[i]);
        int e = (int)((b >> 52) & 0x7ff) - 1023 + eadj;
        double m = __longlong_as_double((long long)((b & 0x000fffffffffffffULL) | 0x3ff0000000000000ULL));
        if (m > 0x1.6a09e667f3bcdp+0) { m = m * 0.5; e = e + 1; }
        const double f = m - 1.0;
        s[i] = div_near(f, 2.0 + f);
        if (f == -0x1p-52) s[i] = -0x1.0000000000001p-53;  // the divisor of all ones
        z[i] = s[i] * s[i];
        p[i] = 0x1.8618618618618p-5;
        ed[i] = (double)e;
    }
    constexpr double C[9] = {0x1.af286bca1af28p-5, 0x1.e1e1e1e1e1e1ep-5, 0x1.1111111111111p-4, 0x1.3b13b13b13b14p-4,
                             0x1.745d1745d1746p-4, 0x1.c71c71c71c71cp-4, 0x1.2492492492492p-3, 0x1.999999999999ap-3,
                             0x1.5555555555555p-2};
#pragma unroll
    for (int k = 0; k < 9; k++)
#pragma unroll
        for (int i = 0; i < N; i++) p[i] = fma(p[i], z[i], C[k]);
#pragma unroll
    for (int i = 0; i < N; i++) {
        const double r = z[i] * p[i], two_s = s[i] + s[i];
        out[i] = fma(ed[i], CTL_LN2_HI, two_s + fma(two_s, r, ed[i] * CTL_LN2_LO));
    }
}

static __device__ double dlog(double x) {
    if (!(x > 0.0)) return x == 0.0 ? __longlong_as_double(0xfff0000000000000ULL)
                                     : __longlong_as_double(0x7ff8000000000000ULL);
    if (x == __longlong_as_double(0x7ff0000000000000ULL)) return x;
    const bool small = x < 0x1p-1022;
    const double in[1] = {small ? x * 0x1p54 : x};
    double out[1];
    dlog_of<1>(in, out, small ? -54 : 0);
    return out[0];
}

// exp(x): Cody-Waite reduction, degree-14 Taylor polynomial, 2^k scaling.
static __device__ double dexp(double x) {
    if (x != x) return x;
    if (x > 709.0) return __longlong_as_double(0x7ff0000000000000ULL);
    if (x < -745.0) return 0.0;
    double k = rint(x * 0x1.71547652b82fep+0);
    double r = fma(-k, CTL_LN2_HI, x);
    r = fma(-k, CTL_LN2_LO, r);
    double p = 0x1.93974a8c07c9dp-37;
    p = fma(p, r, 0x1.6124613a86d09p-33);
    p = fma(p, r, 0x1.1eed8eff8d898p-29);
    p = fma(p, r, 0x1.ae64567f544e4p-26);
    p = fma(p, r, 0x1.27e4fb7789f5cp-22);
    p = fma(p, r, 0x1.71de3a556c734p-19);
    p = fma(p, r, 0x1.a01a01a01a01ap-16);
    p = fma(p, r, 0x1.a01a01a01a01ap-13);
    p = fma(p, r, 0x1.6c16c16c16c17p-10);
    p = fma(p, r, 0x1.1111111111111p-7);
    p = fma(p, r, 0x1.5555555555555p-5);
    p = fma(p, r, 0x1.5555555555555p-3);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = fma(p, r, 1.0);
    int ki = (int)k;
    if (ki < -1000) { p = p * 0x1p-200; ki = ki + 200; }
    return p * __longlong_as_double((long long)((uint64_t)(ki + 1023) << 52));
}

// FP32 log(x) for normal x > 0: the reduction of dlog in single precision,
// series 2s(1 + s^2/3 + s^4/5 + s^6/7 + s^8/9).
__device__ __forceinline__ float flog(float x) {
    const uint32_t b = __float_as_uint(x);
    int e = (int)((b >> 23) & 0xffu) - 127;
    float m = __uint_as_float((b & 0x007fffffu) | 0x3f800000u);
    if (m > 0x1.6a09e6p+0f) { m = m * 0.5f; e = e + 1; }
    const float f = m - 1.0f;
    float sv = div_near(f, 2.0f + f);
    sv = f == -0x1p-23f ? -0x1.000002p-24f : sv;  // the divisor of all ones
    const float z = sv * sv;
    float p = 0x1.c71c72p-4f;
    p = fmaf(p, z, 0x1.24924ap-3f);
    p = fmaf(p, z, 0x1.99999ap-3f);
    p = fmaf(p, z, 0x1.555556p-2f);
    const float r = z * p;
    const float ef = (float)e;
    const float two_s = sv + sv;
    return fmaf(ef, 0x1.62e4p-1f, two_s + fmaf(two_s, r, ef * 0x1.7f7d1cp-20f));
}

__device__ __forceinline__ float u24f(uint32_t w) { return ((float)(w >> 8) + 0.5f) * 0x1p-24f; }

static __constant__ double c_logfact[16] = {
    0.0, 0.0, 0x1.62e42fefa39efp-1, 0x1.cab0bfa2a2002p+0, 0x1.96ca77c922cf9p+1,
    0x1.326643c4479c9p+2, 0x1.a51273acf01cap+2, 0x1.10ce1f32dcc30p+3,
    0x1.5358e82fcb70dp+3, 0x1.99a8921a7f7cfp+3, 0x1.e357590954d15p+3,
    0x1.180973f3a8d74p+4, 0x1.3fcba16d50143p+4, 0x1.68d5a9c3b32cep+4,
    0x1.930f3df162a42p+4, 0x1.be636a63fd346p+4};

// log(k!) : table below 16, Stirling series above.
static __device__ double dlogfact(double k) {
    if (k < 16.0) return c_logfact[(int)k];
    double x = k + 1.0;
    double ix = 1.0 / x;
    double ix2 = ix * ix;
    double ser = ix * (0x1.5555555555555p-4 -
                       ix2 * (0x1.6c16c16c16c17p-9 -
                              ix2 * (0x1.a01a01a01a01ap-11 - ix2 * 0x1.3813813813814p-11)));
    return (x - 0.5) * dlog(x) - x + 0x1.d67f1c864beb5p-1 + ser;
}

__device__ __forceinline__ uint32_t clamp_k(double k) {
    return k > 2147483647.0 ? 2147483647u : (uint32_t)k;
}

// 1/k for k = 1..64, correctly rounded: the inversion's recurrence
// multiplies by these instead of dividing (an FP64 division is a long
// instruction sequence on the GPU); the oracle holds the same literals.
static __constant__ double c_recip[64] = {
    0x1.0000000000000p+0, 0x1.0000000000000p-1, 0x1.5555555555555p-2, 0x1.0000000000000p-2,
    0x1.999999999999ap-3, 0x1.5555555555555p-3, 0x1.2492492492492p-3, 0x1.0000000000000p-3,
    0x1.c71c71c71c71cp-4, 0x1.999999999999ap-4, 0x1.745d1745d1746p-4, 0x1.5555555555555p-4,
    0x1.3b13b13b13b14p-4, 0x1.2492492492492p-4, 0x1.1111111111111p-4, 0x1.0000000000000p-4,
    0x1.e1e1e1e1e1e1ep-5, 0x1.c71c71c71c71cp-5, 0x1.af286bca1af28p-5, 0x1.999999999999ap-5,
    0x1.8618618618618p-5, 0x1.745d1745d1746p-5, 0x1.642c8590b2164p-5, 0x1.5555555555555p-5,
    0x1.47ae147ae147bp-5, 0x1.3b13b13b13b14p-5, 0x1.2f684bda12f68p-5, 0x1.2492492492492p-5,
    0x1.1a7b9611a7b96p-5, 0x1.1111111111111p-5, 0x1.0842108421084p-5, 0x1.0000000000000p-5,
    0x1.f07c1f07c1f08p-6, 0x1.e1e1e1e1e1e1ep-6, 0x1.d41d41d41d41dp-6, 0x1.c71c71c71c71cp-6,
    0x1.bacf914c1bad0p-6, 0x1.af286bca1af28p-6, 0x1.a41a41a41a41ap-6, 0x1.999999999999ap-6,
    0x1.8f9c18f9c18fap-6, 0x1.8618618618618p-6, 0x1.7d05f417d05f4p-6, 0x1.745d1745d1746p-6,
    0x1.6c16c16c16c17p-6, 0x1.642c8590b2164p-6, 0x1.5c9882b931057p-6, 0x1.5555555555555p-6,
    0x1.4e5e0a72f0539p-6, 0x1.47ae147ae147bp-6, 0x1.4141414141414p-6, 0x1.3b13b13b13b14p-6,
    0x1.3521cfb2b78c1p-6, 0x1.2f684bda12f68p-6, 0x1.29e4129e4129ep-6, 0x1.2492492492492p-6,
    0x1.1f7047dc11f70p-6, 0x1.1a7b9611a7b96p-6, 0x1.15b1e5f75270dp-6, 0x1.1111111111111p-6,
    0x1.0c9714fbcda3bp-6, 0x1.0842108421084p-6, 0x1.0410410410410p-6, 0x1.0000000000000p-6};

// exp(-lam) for 0 <= lam < 10: dexp's reduction, polynomial and scaling
// without its tests for arguments out of range.
__device__ __forceinline__ double dexp_neg10(double lam) {
    const double x = -lam;
    double k = rint(x * 0x1.71547652b82fep+0);
    double r = fma(-k, CTL_LN2_HI, x);
    r = fma(-k, CTL_LN2_LO, r);
    double p = 0x1.93974a8c07c9dp-37;
    p = fma(p, r, 0x1.6124613a86d09p-33);
    p = fma(p, r, 0x1.1eed8eff8d898p-29);
    p = fma(p, r, 0x1.ae64567f544e4p-26);
    p = fma(p, r, 0x1.27e4fb7789f5cp-22);
    p = fma(p, r, 0x1.71de3a556c734p-19);
    p = fma(p, r, 0x1.a01a01a01a01ap-16);
    p = fma(p, r, 0x1.a01a01a01a01ap-13);
    p = fma(p, r, 0x1.6c16c16c16c17p-10);
    p = fma(p, r, 0x1.1111111111111p-7);
    p = fma(p, r, 0x1.5555555555555p-5);
    p = fma(p, r, 0x1.5555555555555p-3);
    p = fma(p, r, 0.5);
    p = fma(p, r, 1.0);
    p = fma(p, r, 1.0);
    return p * __longlong_as_double((long long)((uint64_t)((int)k + 1023) << 52));
}

// Poisson(lam) given the reaction's primary uniform pair (wa, wb).
// lam < 10: sequential inversion, p_k = p_{k-1} lam (1/k) with tabulated
// reciprocals.  Four terms per trip: the cumulative sum never falls, so the
// count is the number of partial sums below u.
__device__ __forceinline__ uint32_t poisson_inversion(double lam, uint32_t wa) {
    if (!(lam > 0.0)) return 0u;
    const double u = u32d(wa);
    double p = dexp_neg10(lam);
    double F = p;
    uint32_t k = 0;
    for (uint32_t i = 0; i < 64u && u > F; i += 4u) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            k += u > F ? 1u : 0u;
            p = (p * lam) * c_recip[i + j];
            F = F + p;
        }
    }
    return k;
}

// lam >= 10: Hormann's PTRS (1993); extra trials read blocks 1 + 2j + odd of
// the same (tag, step, sim) stream.
__device__ __forceinline__ uint32_t poisson_ptrs(double lam, uint32_t wa, uint32_t wb, uint64_t seed, uint32_t tag,
                                                 uint32_t step, uint32_t sim, uint32_t odd) {
    double slam = sqrt(lam);
    double b = 0.931 + 2.53 * slam;
    double a = -0.059 + 0.02483 * b;
    double vr = 0.9277 - 3.6224 / (b - 2.0);
    // log(lam) and log(1/alpha) only serve the slow acceptance test; most
    // draws are accepted before it, so they are computed on its first use
    double loglam = 0.0, log_invalpha = 0.0;
    bool slow = false;
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t t = 0; t < PTRS_MAX_TRIALS; t++) {
        if (t > 0) {
            uint32_t j = (t - 1) >> 1;
            if (((t - 1) & 1u) == 0u) w = draw_small(seed, 1u + 2u * j + odd, tag, step, sim);
            wa = ((t - 1) & 1u) ? w.z : w.x;
            wb = ((t - 1) & 1u) ? w.w : w.y;
        }
        double U = u32d(wa) - 0.5;
        double V = u32d(wb);
        double us = 0.5 - fabs(U);
        double k = floor((2.0 * a / us + b) * U + lam + 0.43);
        if (us >= 0.07 && V <= vr) return clamp_k(k);
        if (k < 0.0 || (us < 0.013 && V > us)) continue;
        if (!slow) {
            loglam = dlog(lam);
            log_invalpha = dlog(1.1239 + 1.1328 / (b - 3.4));
            slow = true;
        }
        double lhs = dlog(V) + log_invalpha - dlog(a / (us * us) + b);
        double rhs = -lam + k * loglam - dlogfact(k);
        if (lhs <= rhs) return clamp_k(k);
    }
    return clamp_k(floor(lam));
}

// poisson_ptrs after a first trial (wa, wb) that the squeeze did not accept,
// for the shortest chain of dependent operations: straight-line quotients, and
// the five logarithms of the acceptance test side by side (a lone leaping
// Schlogl simulation: 4.0 -> 3.3 us a leap, with tau_bound's).  Below a mean of 2^40 every operand, k (below 2^50) included,
// is in their range; a larger one takes poisson_ptrs.  The shared-memory sweep,
// whose registers are short, is faster with that (32 x 64 network: 221 against 231 ms).
static __device__ __noinline__ uint32_t poisson_ptrs_call(double lam, uint32_t wa, uint32_t wb, uint64_t seed,
                                                          uint32_t tag, uint32_t step, uint32_t sim, uint32_t odd) {
    return poisson_ptrs(lam, wa, wb, seed, tag, step, sim, odd);
}
__device__ __forceinline__ uint32_t poisson_ptrs_wide(double lam, uint32_t wa, uint32_t wb, uint64_t seed, uint32_t tag,
                                                      uint32_t step, uint32_t sim, uint32_t odd) {
    if (!(lam < 0x1p40)) return poisson_ptrs_call(lam, wa, wb, seed, tag, step, sim, odd);
    const double b = 0.931 + 2.53 * sqrt_near(lam), a = -0.059 + 0.02483 * b;
    const double vr = 0.9277 - div_near(3.6224, b - 2.0);
    uint4 w = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
    for (uint32_t t = 0; t < PTRS_MAX_TRIALS; t++) {
        if (t > 0) {
            const uint32_t j = (t - 1) >> 1;
            if (((t - 1) & 1u) == 0u) w = draw_small(seed, 1u + 2u * j + odd, tag, step, sim);
            wa = ((t - 1) & 1u) ? w.z : w.x;
            wb = ((t - 1) & 1u) ? w.w : w.y;
        }
        const double U = u32d(wa) - 0.5, V = u32d(wb), us = 0.5 - fabs(U);
        const double k = floor((div_near(2.0 * a, us) + b) * U + lam + 0.43);
        if (us >= 0.07 && V <= vr) return clamp_k(k);
        if (k < 0.0 || (us < 0.013 && V > us)) continue;
        const double x[5] = {V, 1.1239 + div_near(1.1328, b - 3.4), div_near(a, us * us) + b, lam, k + 1.0};
        double l[5];
        dlog_of<5>(x, l);
        const double ix = div_near(1.0, x[4]), ix2 = ix * ix;  // dlogfact(k)
        const double ser = ix * (0x1.5555555555555p-4 -
                                 ix2 * (0x1.6c16c16c16c17p-9 -
                                        ix2 * (0x1.a01a01a01a01ap-11 - ix2 * 0x1.3813813813814p-11)));
        const double lf = k < 16.0 ? c_logfact[(int)k] : (x[4] - 0.5) * l[4] - x[4] + 0x1.d67f1c864beb5p-1 + ser;
        if (l[0] + l[1] - l[2] <= -lam + k * l[3] - lf) return clamp_k(k);
    }
    return clamp_k(floor(lam));
}

// The first trial of poisson_ptrs as far as its squeeze: true with the count
// when that accepts; a mean above 2^40 is left to it.
__device__ __forceinline__ bool poisson_ptrs_quick(double lam, uint32_t wa, uint32_t wb, uint32_t& k_out) {
    double slam = sqrt_near(lam);
    double b = 0.931 + 2.53 * slam;
    double a = -0.059 + 0.02483 * b;
    double vr = 0.9277 - div_near(3.6224, b - 2.0);
    double U = u32d(wa) - 0.5;
    double V = u32d(wb);
    double us = 0.5 - fabs(U);
    double k = floor((div_near(2.0 * a, us) + b) * U + lam + 0.43);
    k_out = clamp_k(k);
    return lam < 0x1p40 && us >= 0.07 && V <= vr;
}

// Cao's g_i (tau.cu:1741-1789) in FP32.
__device__ __forceinline__ float gfun(uint32_t hor, uint32_t hort, int32_t x) {
    float xf = (float)x;
    switch (hor) {
        case 1: return 1.0f;
        case 2: return hort == 2 ? 2.0f + 1.0f / (xf - 1.0f) : 2.0f;
        case 3:
            if (hort == 3) return 3.0f + 1.0f / (xf - 1.0f) + 2.0f / (xf - 2.0f);
            if (hort == 2) return 3.0f + 1.5f / (xf - 1.0f);
            return 3.0f;
        default: return 1.0f;
    }
}

// Cao's bound on the leap for one species (tau.cu:1741-1922): the smaller of
// m / |mu| and m^2 / sigma^2 with m = max(eps x / g, 1).  sigma^2 is not 0, mu
// is 0 only where the bound by mu is infinite.
static __device__ __noinline__ float tau_bound_any(uint32_t hor, uint32_t hort, int32_t x, float eps, float mu, float sg) {
    const float tmp2 = (eps * (float)x) / gfun(hor, hort, x);
    const float macs = tmp2 > 1.0f ? tmp2 : 1.0f;
    const float t3 = mu != 0.0f ? macs / fabsf(mu) : __int_as_float(0x7f800000);
    const float t4 = (macs * macs) / sg;
    return t3 < t4 ? t3 : t4;
}
__device__ __forceinline__ float tau_bound(uint32_t hor, uint32_t hort, int32_t x, float eps, float mu, float sg) {
    const float xf = (float)x, ex = eps * xf, d1 = xf - 1.0f, d2 = xf - 2.0f;
    bool fits = num_fits(ex) & div_fits(mu) & div_fits(sg);
    float tmp2 = ex;  // g = 1
    if (hor == 2u || hor == 3u) {
        float g = hor == 2u ? 2.0f : 3.0f;
        if (hort >= 2u && hort <= hor) {  // g depends on x
            fits &= div_fits(d1);
            if (hort == 3u) {
                fits &= div_fits(d2);
                g = 3.0f + div_near(1.0f, d1) + div_near(2.0f, d2);
            } else {
                g = g + div_near(hor == 2u ? 1.0f : 1.5f, d1);
            }
            fits &= div_fits(g);
        }
        tmp2 = div_near(ex, g);
    }
    const float macs = tmp2 > 1.0f ? tmp2 : 1.0f;
    const float t3 = div_near(macs, fabsf(mu)), t4 = div_near(macs * macs, sg);
    if (!(fits & (macs < 0x1p30f))) return tau_bound_any(hor, hort, x, eps, mu, sg);
    return t3 < t4 ? t3 : t4;
}

// One binary level: left unless the target lies beyond a positive left
// weight and the right weight is positive.  Weights are >= 0 and the target is
// positive and stays so (a uniform above 0 times a positive sum, less a left
// weight it exceeds), so "beyond" is x > L also where L is 0.
__device__ __forceinline__ bool go_right(double& x, double L, double R) {
    const bool right = (x > L) & (R != 0.0);
    if (right) x = x - L;
    return right;
}


}  // namespace dev
}  // namespace ctl
