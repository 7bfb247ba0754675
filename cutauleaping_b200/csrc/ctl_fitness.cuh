// calculateFitness (2phase_n-tau-leaping.cu:3324-3408) on sm_100a: the
// kernels behind ctl_fitness_device, ctl_fitness_sums_device and the
// host-buffer fitness calls, and the rule that picks one.
//
// A parameter set's fitness is, over instants c, species s and target
// repetitions e in that order, the FP32 running sum of |target - mean| /
// target (|target - mean| where the target is 0), each term computed and
// added in FP64 and the sum rounded to FP32 after every addition; mean is the
// FP64 sum of the set's p_rep samples divided by p_rep.  The FP32 sum makes
// the order of the terms part of the result, so it stays a serial chain; the
// means do not: integer sums below 2^53 equal the FP64 running sum exactly.
#pragma once

#include <cuda_runtime.h>
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdint>

namespace ctl {
namespace fit {

namespace cg = cooperative_groups;

struct Args {
    const uint32_t* samples;           // [threads * blocks][ns][so], or null:
    const unsigned long long* sums;    // [nsets][ns][so] sums of the p_rep samples
    const uint32_t* target;            // [ns][E][REP][so]
    const uint8_t* swarm;              // [nsets] experiment of each set
    double* fitness;                   // [nsets]
    uint32_t threads, nsets, p_rep, ns, so, E, REP;
};

// Sample row of simulation `par` of parameter set `set` (the reference's
// layout: simulation (b * p_rep + par) * threads + t belongs to set b * threads + t).
__device__ __forceinline__ size_t row_of(const Args& a, uint32_t set, uint32_t par) {
    return (size_t)(set / a.threads * a.p_rep + par) * a.threads + set % a.threads;
}

// Mean of one (instant, species) word from the integer sum of its samples.
// Above 2^53 the reference's FP64 running sum may round: it is redone.
__device__ __forceinline__ double mean_of(const Args& a, uint32_t set, size_t word, unsigned long long sum) {
    double acc = (double)sum;
    if (a.samples && sum > (1ull << 53)) {
        acc = 0.0;
        for (uint32_t par = 0; par < a.p_rep; par++)
            acc = acc + (double)a.samples[row_of(a, set, par) * ((size_t)a.ns * a.so) + word];
    }
    return acc / (double)a.p_rep;
}

__device__ __forceinline__ double term(uint32_t target, double mean) {
    const int tgt = (int)target;
    double d = fabs((double)tgt - mean);
    if (tgt != 0) d = d / (double)tgt;
    return d;
}

// The running sum s (FP32 values held in FP64): s = (double)(float)(s + d).
// While s + d keeps the sign and exponent of s, adding and subtracting
// 1.5 * 2^(e+29) rounds it to 24 bits (nearest even) just as the conversion
// does, without the two conversions in the chain; `key` is the sign and
// exponent that `magic` was made for, and `none` is set while s is zero, not
// finite or outside FP32's normal range (then every addition converts).
struct Chain {
    double s = 0.0, magic = 0.0;
    uint32_t key = 0u, none = 1u;
    __device__ __forceinline__ void convert(double d) {
        s = (double)(float)(s + d);
        const uint32_t hi = (uint32_t)__double2hiint(s), ex = (hi >> 20) & 0x7ffu;
        key = hi & 0xfff00000u;
        none = ex >= 1023u - 126u && ex < 1023u + 127u ? 0u : 1u;
        magic = __hiloint2double((int)((hi & 0xfff00000u) + (29u << 20) + 0x80000u), 0);
    }
    // the next `n` terms, from shared memory (16-byte aligned; every lane of
    // the warp runs the same chain on broadcast loads)
    __device__ __forceinline__ void add(const double* t, uint32_t n) {
        const double2* t2 = reinterpret_cast<const double2*>(t);
        uint32_t i = 0;
        double2 nx[4];
        if (n >= 8u)
#pragma unroll
            for (int j = 0; j < 4; j++) nx[j] = t2[j];
        for (; i + 8u <= n; i += 8u) {
            double d[8], v = s;
            uint32_t off = none;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                d[2 * j] = nx[j].x;
                d[2 * j + 1] = nx[j].y;
            }
            if (i + 16u <= n)
#pragma unroll
                for (int j = 0; j < 4; j++) nx[j] = t2[i / 2 + 4 + j];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const double r = v + d[j];
                off |= ((uint32_t)__double2hiint(r) ^ key) & 0xfff00000u;
                v = (r + magic) - magic;
            }
            if (off == 0u) {
                s = v;
            } else {
#pragma unroll
                for (int j = 0; j < 8; j++) convert(d[j]);
            }
        }
        for (; i < n; i++) convert(t[i]);
    }
};

constexpr int CHUNK = 256;   // words per CTA and step, at most
constexpr int TERMS = 512;   // terms per CTA and step, at most (words x target repetitions)

// One parameter set per cluster of CL CTAs.  The words (instant, species) are
// cut into chunks; in every step each CTA's loaders (LOADERS threads) sum the
// p_rep samples of one chunk (coalesced rows, 16 bytes per thread when VEC is
// 4) and leave the chunk's terms in its shared memory, and while the next
// step's chunks are being summed the last warp of CTA 0 runs the serial chain
// over this step's terms (through distributed shared memory).  Bound: the
// samples read once from HBM, then the chain over one step's terms.
template <int VEC, int LOADERS>
__global__ void __launch_bounds__(LOADERS + 32) set_kernel(Args a, uint32_t chunk) {
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t CL = cl.num_blocks(), rank = cl.block_rank();
    __shared__ unsigned long long red[LOADERS * VEC];
    __shared__ __align__(16) double terms[2][TERMS];
    const size_t words = (size_t)a.ns * a.so;
    const size_t step_words = (size_t)chunk * CL;
    const uint32_t steps = (uint32_t)((words + step_words - 1) / step_words);
    const uint32_t tid = threadIdx.x;
    const bool loader = tid < (uint32_t)LOADERS;
    const uint32_t cols = chunk / VEC, groups = LOADERS / cols;  // row groups per column
    const uint32_t col = tid % cols, grp = tid / cols;
    for (uint32_t set = blockIdx.x / CL; set < a.nsets; set += gridDim.x / CL) {
        const uint32_t ex = a.swarm[set];
        Chain ch;
        for (uint32_t k = 0; k <= steps; k++) {
            const size_t w0 = (size_t)k * step_words + (size_t)rank * chunk;  // this CTA's chunk
            const uint32_t n = k < steps && w0 < words ? (uint32_t)min((size_t)chunk, words - w0) : 0u;
            if (loader && n) {
                if (a.samples) {
                    unsigned long long s[VEC];
#pragma unroll
                    for (int v = 0; v < VEC; v++) s[v] = 0ull;
                    if (grp < groups && col * VEC < n) {
                        const size_t row = words * a.threads;  // between simulations of the set
                        const size_t stride = row * groups;
                        const uint32_t* p = a.samples + row_of(a, set, grp) * words + w0 + col * VEC;
                        uint32_t par = grp;
                        constexpr int U = 8;  // rows in flight per thread
                        for (; par + (U - 1) * groups < a.p_rep; par += U * groups, p += U * stride) {
                            if constexpr (VEC == 4) {
                                uint4 x[U];
#pragma unroll
                                for (int u = 0; u < U; u++) x[u] = __ldcs(reinterpret_cast<const uint4*>(p + u * stride));
#pragma unroll
                                for (int u = 0; u < U; u++) {
                                    s[0] += x[u].x;
                                    s[1] += x[u].y;
                                    s[2] += x[u].z;
                                    s[3] += x[u].w;
                                }
                            } else {
                                uint32_t x[U];
#pragma unroll
                                for (int u = 0; u < U; u++) x[u] = __ldcs(p + u * stride);
#pragma unroll
                                for (int u = 0; u < U; u++) s[0] += x[u];
                            }
                        }
                        for (; par < a.p_rep; par += groups, p += stride)
#pragma unroll
                            for (int v = 0; v < VEC; v++) s[v] += __ldcs(p + v);
                    }
                    if (grp < groups)
#pragma unroll
                        for (int v = 0; v < VEC; v++) red[grp * chunk + col * VEC + v] = s[v];
                    asm volatile("bar.sync 1, %0;" ::"n"(LOADERS) : "memory");
                }
                for (uint32_t w = tid; w < n; w += LOADERS) {
                    unsigned long long t = 0ull;
                    if (a.samples)
                        for (uint32_t g = 0; g < groups; g++) t += red[g * chunk + w];
                    else
                        t = a.sums[(size_t)set * words + w0 + w];
                    const double m = mean_of(a, set, w0 + w, t);
                    const uint32_t c = (uint32_t)((w0 + w) / a.so), sp = (uint32_t)((w0 + w) % a.so);
                    const uint32_t* tg = a.target + ((size_t)c * a.E + ex) * a.REP * a.so + sp;
                    for (uint32_t e = 0; e < a.REP; e++) terms[k & 1u][w * a.REP + e] = term(tg[(size_t)e * a.so], m);
                }
            } else if (!loader && rank == 0 && k > 0) {
                for (uint32_t q = 0; q < CL; q++) {  // the chunks of step k - 1, in order
                    const size_t c0 = (size_t)(k - 1) * step_words + (size_t)q * chunk;
                    if (c0 >= words) break;
                    const uint32_t m = (uint32_t)min((size_t)chunk, words - c0) * a.REP;
                    ch.add(cl.map_shared_rank(&terms[(k - 1) & 1u][0], (int)q), m);
                }
            }
            // the step's terms are visible, the buffer of step k - 1 and the
            // partial sums are free
            if (CL > 1) cl.sync();
            else __syncthreads();
        }
        if (rank == 0 && tid == (uint32_t)LOADERS)
            a.fitness[set] = ((1.0 / (double)a.ns) * (1.0 / (double)a.so)) * ch.s;
    }
}

// One thread per parameter set: many sets with little work each, where a
// chain per lane keeps the chip busier than a CTA per set.
__global__ void __launch_bounds__(128) lane_kernel(Args a) {
    const uint32_t set = blockIdx.x * blockDim.x + threadIdx.x;
    if (set >= a.nsets) return;
    const uint32_t ex = a.swarm[set];
    const size_t words = (size_t)a.ns * a.so;
    float sub = 0.0f;
    for (uint32_t c = 0; c < a.ns; c++) {
        for (uint32_t s = 0; s < a.so; s++) {
            const size_t word = (size_t)c * a.so + s;
            double acc = 0.0;
            if (a.samples) {
                for (uint32_t par = 0; par < a.p_rep; par++)
                    acc = acc + (double)a.samples[row_of(a, set, par) * words + word];
            } else {
                acc = (double)a.sums[(size_t)set * words + word];
            }
            acc = acc / (double)a.p_rep;
            for (uint32_t e = 0; e < a.REP; e++)
                sub = (float)((double)sub + term(a.target[(((size_t)c * a.E + ex) * a.REP + e) * a.so + s], acc));
        }
    }
    a.fitness[set] = ((1.0 / (double)a.ns) * (1.0 / (double)a.so)) * (double)sub;
}

struct Shape {
    int cl, loaders;  // CTAs per parameter set (0: one thread per set), loader threads per CTA
};

// Microseconds of the two kernels, as measured on one B200 over 64 to 262,144
// sets of 3 to 1,600 words, 1 to 128 samples (or sums) a word and 1 to 16 target
// repetitions (13,459 shapes).
//
// A thread per set: the latency of its serial loads, whatever the number of
// sets, then the sectors that the sets load together.  A warp's lanes share
// sectors where neighbouring sets' rows lie side by side (`threads` of 16 or
// more, or sums) and are shorter than one; a word's sectors serve the words
// after it while the rows under way fit an SM's L1, else they come from L2 or
// HBM again, whole lines apart when a row is longer than one.
inline double lane_us(const Args& a, int sms) {
    const double words = (double)a.ns * a.so, sets = a.nsets, rep = a.REP;
    const double rows = a.samples ? a.p_rep : 1.0;
    const bool side = !a.samples || a.threads >= 16u;
    const double share = std::min(1.0, (side ? words : words * rows) / 8.0);  // of a 32-byte sector
    const bool keeps = std::min(sets / sms, 2048.0) * rows * share * 32.0 <= 200e3;
    const double sector = keeps ? 1.1e-6 : words <= 32.0 ? 4.0e-6 : 14e-6;
    return 3.3 + words * (0.26 + (side ? 0.030 : 0.048) * rows + 0.13 * rep) +
           sets * words * (share * rows * sector + 0.72e-6 * rep);
}

// A CTA of 128 loaders per set: a launch and one set, or what the sets of an SM
// cost it -- the chain of their terms above all.
inline double cta_us(const Args& a, int sms) {
    const double words = (double)a.ns * a.so, sets = a.nsets, rep = a.REP, rows = a.samples ? a.p_rep : 1.0;
    return std::max(7.0 + 0.15 * rep + 0.002 * sets,
                    sets / sms * (1.2 + 0.0005 * rows + 0.06 * rep + words * (0.0051 * rep + 0.000072 * rows)));
}

// The kernel with the smaller estimate: 0.7 % slower than the faster kernel on
// the average of those shapes, and at most 2.5 us slower than a thread per set.
// 65,536 sets of 6 words and 64 samples take 103 us with a thread per set and 400
// with a CTA; 32,768 of 60 words and 32 samples 915 and 363; 256 of 60 words and
// one sample 29 and 7.
// Large sets (from 2^18 samples, 1 MB): 256 sets of 512 x 1,600 samples take
// 182 on two CTAs of 128 loaders each, 190 on one of 512, 273 on one of 128;
// 8 such sets take 62, 48 and 102, so fewer sets than half the SMs get 512.
// More CTAs per set lose: their steps end in a cluster barrier (8 x 512 on
// 256 sets: 860).  The thread per set also takes targets of more repetitions
// than a step's term buffer holds.
inline Shape shape_for(const Args& a, int sms) {
    if (a.REP > (uint32_t)TERMS / 4 || lane_us(a, sms) < cta_us(a, sms)) return {0, 0};
    const uint64_t words = (uint64_t)a.ns * a.so;
    if (words * (a.samples ? a.p_rep : 1u) < (1ull << 18)) return {1, 128};
    if (2ull * a.nsets <= (uint64_t)sms) return {1, 512};
    return {2, 128};
}

template <int VEC, int LOADERS>
inline cudaError_t launch_set(const Args& a, int cl, cudaStream_t s) {
    const uint64_t words = (uint64_t)a.ns * a.so;
    uint64_t chunk = (words + cl - 1) / cl;
    const uint64_t most = (uint64_t)(LOADERS * VEC < CHUNK ? LOADERS * VEC : CHUNK);
    chunk = chunk < most ? chunk : most;
    chunk = (chunk + VEC - 1) / VEC * VEC;
    while (chunk * a.REP > (uint64_t)TERMS) chunk -= VEC;
    cudaLaunchConfig_t cfg = {};
    const uint64_t clusters = a.nsets < (1u << 20) ? a.nsets : (1u << 20);
    cfg.gridDim = dim3((unsigned)(clusters * (unsigned)cl));
    cfg.blockDim = dim3(LOADERS + 32);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cl;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, set_kernel<VEC, LOADERS>, a, (uint32_t)chunk);
}

inline cudaError_t launch(const Args& a, Shape sh, cudaStream_t s) {
    if (sh.cl == 0) {
        lane_kernel<<<(a.nsets + 127) / 128, 128, 0, s>>>(a);
        return cudaGetLastError();
    }
    const bool vec = a.samples && ((uint64_t)a.ns * a.so) % 4 == 0 && (reinterpret_cast<uintptr_t>(a.samples) & 15) == 0;
    if (sh.loaders == 128) return vec ? launch_set<4, 128>(a, sh.cl, s) : launch_set<1, 128>(a, sh.cl, s);
    return vec ? launch_set<4, 512>(a, sh.cl, s) : launch_set<1, 512>(a, sh.cl, s);
}

}  // namespace fit
}  // namespace ctl
