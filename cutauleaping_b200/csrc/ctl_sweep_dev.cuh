// Device side of the persistent tau-leaping / SSA sweep for sm_100a
// (shared by ctl_sweep.cu and the per-group-size kernel files
// ctl_sweep_g*.cu, which the build compiles in parallel).
//
// Replaces the reference's host loop (kernel.cu:242-345) and its kernels
// PreCalculations (2phase_n-tau-leaping.cu:1568-2093), EventualSSASteps
// (2099-2273), LightweightSSA (2280-2454), setup_random (2974-2988),
// PrepareVariables (1269-1297) and ParallelVoting (2990-3002) with ONE
// launch: blocks hold simulations in shared-memory slots, run each to the end
// (leaps, SSA bursts, samples; a group of G lanes at a time, which need not be
// the same one from one stretch of work to the next) and pull the next one from
// a device work queue (atomic ticket).  No host round trip per leap, no per-pass
// reload of state from global memory.
//
// Determinism contract (what makes any launch shape give identical bits):
//   * every random word comes from Philox4x32-10 with key = seed and counter
//     (block, tag, step, sim): a draw depends on which simulation, which step
//     and what it is for, never on which thread computes it;
//   * every FP64 sum over reactions (A0, the critical sum a0c) is the root of
//     a fixed binary tree over the reactions padded to P = 2^k leaves, and
//     the SSA / critical-reaction searches descend that same tree;
//   * per-species sums (mu, sigma^2, population updates) run over a fixed
//     entry order by one lane.
// The CPU oracle (oracle/ctl_oracle.c) implements the same contract.
//
// Built with -fmad=false: no implicit FMA contraction; fma() is called
// explicitly where it is meant.
//
// The device code is written against a model type M with the fields of
// Model below.  The library's kernels read the network's geometry (species,
// reactions, tree levels, sample counts) from that parameter block at run
// time; a kernel compiled for one network at run time by NVRTC
// (ctl_sweep.cu, sweep_spec_kernel) instantiates the same code with a type
// whose geometry fields are static constexpr members of the same names, so
// that loops over leaves, species and samples have constant bounds and the
// slots' offsets fold into the code.  Both give the same bits.
#pragma once
#ifndef __CUDACC_RTC__
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>

#include "ctl_internal.h"
#endif
#include "ctl_devmath.cuh"

namespace ctl {
namespace dev {

// The model's tables in device memory (and the end time): the part of the
// model that every kernel reads at run time.
struct Tables {
    const uint32_t* __restrict__ reac_off;
    const uint32_t* __restrict__ reac_ent;
    const uint2* __restrict__ reac_desc;  // [R] packed reactants, x == 0xffffffff: general list
    // Species by their number of entries, most first (lanes that take
    // neighbouring places then run loops of about the same length): species,
    // first entry, entries, HOR | HORtype << 8.
    const uint4* __restrict__ v_sp;      // V or F species-major (quirk Q5)
    const uint32_t* __restrict__ v_ent;
    const uint4* __restrict__ fs_sp;     // F species-major
    const uint32_t* __restrict__ fs_ent;
    const uint32_t* __restrict__ fr_ent;
    const uint4* __restrict__ fire;       // [R] first entry and entries of F's row, first and number of dependents
    const uint4* __restrict__ dep;        // dependents: reaction, its two reactant descriptors, leaf_pos
    const double* __restrict__ tvec;
    const uint32_t* __restrict__ cs;
    double tmax;
};

// Tables plus the geometry, read at run time (the library's own kernels).
struct Model : Tables {
    int S, R, P, ns, s_out;
    static constexpr int LEAVES = 0;  // P, where it is a compile-time constant
    int general;  // some reaction's descriptor is DESC_GENERAL
    int changes;  // most species a reaction changes
};

// Reactant descriptors: species * 4 + coefficient, coefficient 1 or 2; a
// reaction with fewer than two reactant entries names the dummy species S
// (count 1, coefficient 0): factor 1, never short, never critical.
constexpr uint32_t DESC_GENERAL = 0xffffffffu;

// Shared-memory slots: one contiguous block per simulation slot, X [S + 1]
// (X[S] = 1, the dummy species), a [P], K [P], then the rate constants [P]
// unless the block shares them and, in fitness mode, the last recorded row
// [s_out].  A leap's list of reactions (16-bit) and then its proposed state X1
// [S] take the propensities' place, which are computed anew after it (and
// before another attempt).  Offsets in bytes, from the geometry (P a power of
// two, at least 4).
struct Layout {
    uint32_t slot;  // bytes per slot, an odd multiple of 16 (slots in different banks)
    uint32_t ns;    // slots per block, at least one per group
    uint32_t off_state, off_c, off_grp;
    uint32_t oc, olast;  // within the slot
};
__host__ __device__ constexpr uint32_t lay_a(int S) { return ((uint32_t)(S + 1) * 4u + 15u) & ~15u; }
__host__ __device__ constexpr uint32_t lay_k(int S, int P) {
    return lay_a(S) + (((uint32_t)(S > P ? S : P) * 4u + 15u) & ~15u);
}
__host__ __device__ constexpr uint32_t lay_end(int S, int P) { return lay_k(S, P) + (uint32_t)P * 4u; }

// Leaves are read four at a time (16 bytes); chunk q of a slot's propensities
// lies at q ^ ((q >> 3) & 3), so that the lanes of a group, each reading its
// own run of 1 to 4 chunks, hit distinct banks.
__host__ __device__ constexpr int chunk_pos(int q) { return q ^ ((q >> 3) & 3); }
__host__ __device__ constexpr int leaf_pos(int r) { return r ^ ((r >> 3) & 12); }
// Chunks of four leaves per lane for groups of G lanes.
__host__ __device__ constexpr int chunks_per_lane(int P, int G) { return P > 4 * G ? P / (4 * G) : 1; }

// Per-slot scalars, one array each (index = slot).
struct StateArrays {
    double *T, *tl, *tnext;
    unsigned long long* fire;  // firings of the leaps
    uint32_t *sim, *cursor, *n, *burst, *leaps, *ssa, *rej, *status;
};
constexpr uint32_t ST_NOTHING = 0x100u;  // status: A0 == 0, the remaining rows are still to be filled (finish_zero)
constexpr uint32_t STATE_BYTES = 4 * 8 + 8 * 4;  // per slot
constexpr uint32_t FULL = 0xffffffffu;
// Phase of a simulation between two stretches of work.
constexpr uint32_t PH_SSA = 0u, PH_DECIDE = 1u, PH_DONE = 2u, PH_CLOSED = 3u;

// ---------------------------------------------------------------------------
// Groups and slots
// ---------------------------------------------------------------------------

// The lanes that work on one simulation.  G <= 32: a slice of one warp; every
// collective below is a full-warp instruction that all 32 lanes execute
// together (groups without work take part and commit nothing), so the groups
// of a warp never wait on masks of their own.  G = 64, 128, 256: whole warps,
// synchronised by named barrier 1 + group index, cross-warp reductions
// through a small per-group scratch area in shared memory.
template <int G>
struct Grp {
    static constexpr int W = G > 32 ? G / 32 : 1;  // warps per group
    static constexpr int L = G < 32 ? G : 32;      // lanes of the group in a warp
    static constexpr int SCRATCH = 24 * W + 16;    // bytes per group
    uint32_t lane, bar;
    double* ts;                  // [W] sum tree: each warp's total (G > 32)
    unsigned long long* us;      // [W]
    float* fs;                   // [W]
    uint32_t* ws;                // [1]
    __device__ __forceinline__ Grp() {
        lane = threadIdx.x % G;
        bar = 1u + threadIdx.x / G;
        ts = nullptr;
        us = nullptr;
        fs = nullptr;
        ws = nullptr;
    }
    __device__ __forceinline__ void scratch(unsigned char* base) {
        unsigned char* b = base + (threadIdx.x / G) * SCRATCH;
        ts = reinterpret_cast<double*>(b);
        us = reinterpret_cast<unsigned long long*>(b + 8 * W);
        fs = reinterpret_cast<float*>(b + 16 * W);
        ws = reinterpret_cast<uint32_t*>(b + 24 * W);
    }
    __device__ __forceinline__ uint32_t warp() const { return lane >> 5; }
    // this group's bits of a full-warp ballot
    __device__ __forceinline__ uint32_t seg(uint32_t b) const {
        if constexpr (G >= 32) return b;
        return (b >> ((threadIdx.x & 31u) & ~(uint32_t)(G - 1))) & ((1u << (G & 31)) - 1u);
    }
    __device__ __forceinline__ void sync() const {
        if constexpr (G > 32) asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(G) : "memory");
        else if constexpr (G > 1) __syncwarp();
    }
    __device__ __forceinline__ bool any(bool p) const {
        if constexpr (G == 1) return p;
        if constexpr (G > 32) {
            uint32_t r;
            asm volatile(
                "{\n\t.reg .pred a, b;\n\t"
                "setp.ne.u32 a, %1, 0;\n\t"
                "bar.red.or.pred b, %2, %3, a;\n\t"
                "selp.u32 %0, 1, 0, b;\n\t}"
                : "=r"(r)
                : "r"((uint32_t)p), "r"(bar), "r"(G)
                : "memory");
            return r != 0;
        }
        return seg(__ballot_sync(FULL, p)) != 0u;
    }
    __device__ __forceinline__ float fmin(float v) const {
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) {
            float t = __shfl_xor_sync(FULL, v, o);
            v = t < v ? t : v;
        }
        if constexpr (G > 32) {
            sync();  // earlier readers of the scratch are done
            if ((lane & 31u) == 0) fs[lane >> 5] = v;
            sync();
            v = fs[0];
#pragma unroll
            for (int i = 1; i < W; i++) v = fs[i] < v ? fs[i] : v;
        }
        return v;
    }
    __device__ __forceinline__ unsigned long long sum(unsigned long long v) const {
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
        if constexpr (G > 32) {
            sync();
            if ((lane & 31u) == 0) us[lane >> 5] = v;
            sync();
            v = us[0];
#pragma unroll
            for (int i = 1; i < W; i++) v += us[i];
        }
        return v;
    }
    __device__ __forceinline__ uint32_t bcast(uint32_t v) const {
        if constexpr (G == 1) return v;
        if constexpr (G > 32) {
            sync();
            if (lane == 0) ws[0] = v;
            sync();
            return ws[0];
        }
        return __shfl_sync(FULL, v, 0, G <= 32 ? G : 32);
    }
};

template <class M>
struct Slot {
    unsigned char* b;
    float* c;                // rate constants: the slot's own, or the block's
    uint32_t* last;          // fitness mode: the simulation's last recorded sample [s_out]
    __device__ __forceinline__ int32_t& xb(uint32_t byte) const { return *reinterpret_cast<int32_t*>(b + byte); }
    __device__ __forceinline__ int32_t& x(int i) const { return reinterpret_cast<int32_t*>(b)[i]; }
    __device__ __forceinline__ int32_t& x1(const M& m, int i) const { return reinterpret_cast<int32_t*>(b + lay_a(m.S))[i]; }
    __device__ __forceinline__ float* a(const M& m) const { return reinterpret_cast<float*>(b + lay_a(m.S)); }
    __device__ __forceinline__ float& pa(const M& m, int r) const { return a(m)[leaf_pos(r)]; }
    __device__ __forceinline__ float4 chunk(const M& m, int q) const {
        return reinterpret_cast<const float4*>(a(m))[chunk_pos(q)];
    }
    __device__ __forceinline__ uint32_t* k(const M& m) const { return reinterpret_cast<uint32_t*>(b + lay_k(m.S, m.P)); }
    // propensities of the non-critical reactions (0 for critical ones): K's
    // place, until the Poisson counts take it
    __device__ __forceinline__ float* am(const M& m) const { return reinterpret_cast<float*>(b + lay_k(m.S, m.P)); }
    __device__ __forceinline__ uint16_t* list(const M& m) const {
        return reinterpret_cast<uint16_t*>(b + lay_a(m.S));
    }
};

// One reactant factor: X for coefficient 1 (or the dummy's 0), 0.5 X (X-1) for 2.
__device__ __forceinline__ float react_factor(int32_t x, uint32_t two) {
    const float hx = (float)x;
    return two ? (0.5f * hx) * (hx - 1.0f) : hx;
}

// Reactions with more than two reactant entries or a coefficient above 2.
template <class M>
__device__ __forceinline__ float prop_general(const M& m, Slot<M> sl, int r) {
    float v = sl.c[r];
    const uint32_t e1 = m.reac_off[r + 1];
    for (uint32_t e = m.reac_off[r]; e < e1; e++) {
        const uint32_t ent = m.reac_ent[e];
        const int32_t x = sl.x((int)(ent >> 8));
        const int st = (int)(ent & 0xffu);
        if (x < st) return 0.0f;
        if (st == 1) {
            v = v * (float)x;
        } else if (st == 2) {
            float hx = (float)x;
            v = v * ((0.5f * hx) * (hx - 1.0f));
        } else {
            for (int j = 1; j <= st; j++) v = v * ((float)(x - j + 1) / (float)j);
        }
    }
    return v;
}

// Mass-action propensity in FP32 (CalculatePropensity, tau.cu:1443-1470):
// c times, per reactant entry in species order, X (coefficient 1),
// 0.5 X (X-1) (coefficient 2) or the product of (X-e+1)/e (higher); zero when
// a reactant count is below its coefficient.  Reactions with at most two
// entries of coefficient <= 2 go by their packed descriptors, without a
// branch: a missing entry is the dummy species, whose factor is exactly 1.
template <class M>
__device__ __forceinline__ float prop(const M& m, const Slot<M>& sl, int r, uint32_t dx, uint32_t dy) {
    if (m.general && dx == DESC_GENERAL) return prop_general(m, sl, r);
    const int32_t x = sl.xb(dx & ~3u), y = sl.xb(dy & ~3u);
    const float v = (sl.c[r] * react_factor(x, dx & 2u)) * react_factor(y, dy & 2u);
    return x < (int32_t)(dx & 3u) || y < (int32_t)(dy & 3u) ? 0.0f : v;
}

// ---------------------------------------------------------------------------
// The sum tree
// ---------------------------------------------------------------------------

// The binary sum tree over the P leaves lives in the group's registers.  Lane
// l owns the leaves of its run of `chunks_per_lane` chunks and keeps each
// chunk's FP64 sum; one exchange per level then gives every lane the sum of
// its sibling subtree (part), so that the descent needs no memory above the
// chunk it ends in, and nothing of the tree is stored.  Rebuilt after every
// firing from the propensities: 4 loads, 16 conversions and 15 additions per
// lane for 16 leaves, against the paths of the changed leaves through stored
// levels (three barriers, 8 loads per node and lane).  The sums are those of
// the binary tree, level by level.  Lanes with more chunks than registers hold
// (a group smaller than the library would take) sum them again as they descend.
// Groups of several warps exchange their totals through the group's scratch:
// tree_build and descend read them until the next tree_build, which waits for
// the group before it writes (a leap builds two critical trees in a row).
template <int G, class M>
struct Tree {
    // chunks kept in registers
    static constexpr int NC = !M::LEAVES ? 4 : chunks_per_lane(M::LEAVES, G) < 16 ? chunks_per_lane(M::LEAVES, G) : 16;
    static constexpr int LOG = G >= 32 ? 5 : G >= 16 ? 4 : G >= 8 ? 3 : G >= 4 ? 2 : G >= 2 ? 1 : 0;
    double c4[NC];
    double tot;                    // this lane's leaves
    double part[LOG > 0 ? LOG : 1];  // sibling subtrees, 1, 2, 4, ... lanes wide
    double root;
};

// Chunk q's leaves.  Mode 0: propensities; 1: those of critical reactions (whose
// am is 0, where the others' am is a copy of a); 2: as 1 but leaf 0 unmasked (the
// reference's critical pick, tau.cu:1997).  By a select, by the exclusive or of
// the two words (0 for equal words, a against 0), or, FAST, by a - am, which is no
// number where a non-critical propensity overflows FP32.  Groups of several
// warps subtract and look again where that gives no number; exclusive ors take
// the busier integer pipe there (512 x 1024 to t 0.06, 4,736 simulations: 528.6
// against 537 ms).  In smaller groups the second look's code costs more (the
// uneven batch: 344.0 against 332.9).
constexpr int BY_SELECT = 0, BY_XOR = 1, FAST = 2;
template <int G>
constexpr int SOUND = G > 32 ? BY_SELECT : BY_XOR;
template <int HOW, class M>
__device__ __forceinline__ float4 leaves(const M& m, const Slot<M>& sl, int q, int mode) {
    float4 v = sl.chunk(m, q);
    if (mode) {
        const float4 n = reinterpret_cast<const float4*>(sl.am(m))[q];
        auto critical = [](float a, float am) {
            if constexpr (HOW == FAST) return a - am;
            else if constexpr (HOW == BY_XOR) return __uint_as_float(__float_as_uint(a) ^ __float_as_uint(am));
            else return am == 0.0f ? a : 0.0f;
        };
        v.x = mode == 2 && q == 0 ? v.x : critical(v.x, n.x);
        v.y = critical(v.y, n.y);
        v.z = critical(v.z, n.z);
        v.w = critical(v.w, n.w);
    }
    return v;
}
__device__ __forceinline__ double sum4(const float4& v) {
    return ((double)v.x + (double)v.y) + ((double)v.z + (double)v.w);
}

// Binary-tree sum of chunks [q, q + n), n a power of two.
template <int HOW, class M>
__device__ __forceinline__ double range_sum(const M& m, Slot<M> sl, int q, int n, int mode) {
    double st[16];  // st[l]: a finished subtree of 2^l chunks
    for (int i = 0; i < n; i++) {
        double v = sum4(leaves<HOW>(m, sl, q + i, mode));
        int l = 0;
        for (int b = i; b & 1; b >>= 1) v = st[l++] + v;
        st[l] = v;
    }
    return st[31 - __clz(n)];
}

template <int G, class M>
__device__ __forceinline__ void tree_build(const Grp<G>& g, const M& m, const Slot<M>& sl, int mode, Tree<G, M>& t) {
    const int nch = chunks_per_lane(m.P, G), q0 = (int)g.lane * nch;
    const bool own = m.P >= 4 * G || q0 * 4 < m.P;
    constexpr int NC = Tree<G, M>::NC;
    if (nch <= NC) {
#pragma unroll
        for (int k = 0; k < NC; k++) t.c4[k] = k < nch && own ? sum4(leaves<(G > 32 ? FAST : BY_XOR)>(m, sl, q0 + k, mode)) : 0.0;
        double v[NC];
        auto add_up = [&]() {
#pragma unroll
            for (int k = 0; k < NC; k++) v[k] = t.c4[k];
#pragma unroll
            for (int w = 1; w < NC; w *= 2)  // chunks beyond nch are zeros on the right: x + 0 = x
#pragma unroll
                for (int k = 0; k < NC; k += 2 * w) v[k] = v[k] + v[k + w];
        };
        add_up();
        if (G > 32 && mode && v[0] != v[0]) {  // an overflowed propensity less itself
#pragma unroll
            for (int k = 0; k < NC; k++) t.c4[k] = k < nch && own ? sum4(leaves<SOUND<G>>(m, sl, q0 + k, mode)) : 0.0;
            add_up();
        }
        t.tot = v[0];
    } else {
        t.tot = range_sum<SOUND<G>>(m, sl, q0, nch, mode);
    }
    double s = t.tot;
#pragma unroll
    for (int j = 0; j < Tree<G, M>::LOG; j++) {
        t.part[j] = __shfl_xor_sync(FULL, s, 1 << j);
        s = s + t.part[j];
    }
    if constexpr (G > 32) {
        g.sync();  // the totals of the tree before have been read
        if ((g.lane & 31u) == 0) g.ts[g.warp()] = s;
        g.sync();
        if constexpr (G == 64) s = g.ts[0] + g.ts[1];
        if constexpr (G == 128) s = (g.ts[0] + g.ts[1]) + (g.ts[2] + g.ts[3]);
        if constexpr (G == 256)
            s = ((g.ts[0] + g.ts[1]) + (g.ts[2] + g.ts[3])) + ((g.ts[4] + g.ts[5]) + (g.ts[6] + g.ts[7]));
    }
    t.root = s;
}

// Leftmost leaf whose cumulative weight reaches x (ties go left); never a
// zero leaf.  The lanes walk the levels above them together, each testing its
// own side; the one on the path ends in its chunk and tells the others.
template <int G, class M>
__device__ __forceinline__ int descend(const Grp<G>& g, const M& m, const Slot<M>& sl, const Tree<G, M>& t, double x,
                                       int mode) {
    const int nch = chunks_per_lane(m.P, G), q0 = (int)g.lane * nch;
    bool on = true;
    if constexpr (G > 32) {  // the group's warps
        constexpr int W = Grp<G>::W;
        int lo = 0;
#pragma unroll
        for (int half = W / 2; half > 0; half >>= 1) {
            double L = 0.0, R = 0.0;
            const double* v = g.ts + lo;
            if (half == 1) {
                L = v[0];
                R = v[1];
            } else if (half == 2) {
                L = v[0] + v[1];
                R = v[2] + v[3];
            } else {
                L = (v[0] + v[1]) + (v[2] + v[3]);
                R = (v[4] + v[5]) + (v[6] + v[7]);
            }
            if (go_right(x, L, R)) lo += half;
        }
        on = (uint32_t)lo == g.warp();
    }
    constexpr int LOG = Tree<G, M>::LOG;
    double s[LOG > 0 ? LOG : 1];
    s[0] = t.tot;
#pragma unroll
    for (int j = 1; j < LOG; j++) s[j] = s[j - 1] + t.part[j - 1];
#pragma unroll
    for (int j = LOG - 1; j >= 0; j--) {
        const bool upper = (g.lane >> j) & 1u;
        const bool right = go_right(x, upper ? t.part[j] : s[j], upper ? s[j] : t.part[j]);
        on = on & (right == upper);
    }
    int k = 0;
    constexpr int NC = Tree<G, M>::NC;
    if (nch <= NC) {
        double c[NC];
#pragma unroll
        for (int i = 0; i < NC; i++) c[i] = t.c4[i];
#pragma unroll
        for (int h = NC / 2; h > 0; h /= 2) {  // c[0 .. 2h): the chunks below this node
            double L[NC / 2 > 0 ? NC / 2 : 1], R[NC / 2 > 0 ? NC / 2 : 1];
#pragma unroll
            for (int i = 0; i < h; i++) {
                L[i] = c[i];
                R[i] = c[h + i];
            }
#pragma unroll
            for (int w = 1; w < h; w *= 2)
#pragma unroll
                for (int i = 0; i < h; i += 2 * w) {
                    L[i] = L[i] + L[i + w];
                    R[i] = R[i] + R[i + w];
                }
            const bool right = go_right(x, L[0], R[0]);
#pragma unroll
            for (int i = 0; i < h; i++) c[i] = right ? c[h + i] : c[i];
            k += right ? h : 0;
        }
    } else if (on) {
        for (int h = nch / 2; h > 0; h >>= 1) {
            const double L = range_sum<SOUND<G>>(m, sl, q0 + k, h, mode), R = range_sum<SOUND<G>>(m, sl, q0 + k + h, h, mode);
            if (go_right(x, L, R)) k += h;
        }
    }
    // a lane beyond the leaves (P < 4 G) is never on the path
    const int q = m.P >= 4 * G || (q0 + k) * 4 < m.P ? q0 + k : 0;
    const float4 v = leaves<SOUND<G>>(m, sl, q, mode);
    const double v0 = (double)v.x, v1 = (double)v.y, v2 = (double)v.z, v3 = (double)v.w;
    const bool h1 = go_right(x, v0 + v1, v2 + v3);
    const bool h2 = go_right(x, h1 ? v2 : v0, h1 ? v3 : v1);
    const int r = 4 * q + (h1 ? 2 : 0) + (h2 ? 1 : 0);
    if constexpr (G == 1) return r;
    if constexpr (G > 32) {
        if (on) g.ws[0] = (uint32_t)r;
        g.sync();
        return (int)g.ws[0];
    }
    const uint32_t b = g.seg(__ballot_sync(FULL, on));
    return __shfl_sync(FULL, r, __ffs(b) - 1, G <= 32 ? G : 32);
}

// Every propensity from X (all lanes; nothing is written where !act).
template <int G, class M>
__device__ __forceinline__ void all_props(const Grp<G>& g, const M& m, const Slot<M>& sl, bool act) {
#pragma unroll 2
    for (int r = (int)g.lane; r < m.P; r += G) {
        float v = 0.0f;
        if (r < m.R) {
            const uint2 d = m.reac_desc[r];
            v = prop(m, sl, r, d.x, d.y);
        }
        if (act) sl.pa(m, r) = v;
    }
    g.sync();
}

// Where a simulation's samples go: its own rows [ns][s_out] (dynamics), or,
// in fitness mode, added into the 64-bit sums [ns][s_out] of its parameter
// set (integer sums: exact and independent of the order simulations finish
// in), with the last recorded row kept in the slot for the copy-forward.
struct Out {
    uint32_t* samples;
    unsigned long long* sums;
    uint32_t* last;
    __device__ __forceinline__ void put(uint32_t i, int so, int k, uint32_t v) const {
        if (samples) {
            samples[(size_t)i * so + k] = v;
        } else {
            atomicAdd(sums + (size_t)i * so + k, (unsigned long long)v);
            last[k] = v;
        }
    }
    __device__ __forceinline__ uint32_t get(uint32_t i, int so, int k) const {
        return samples ? samples[(size_t)i * so + k] : last[k];
    }
};

template <class M>
__device__ __forceinline__ Out out_of(const M& m, const Run& run, const Slot<M>& sl, uint32_t sim) {
    const size_t row_words = (size_t)m.ns * (size_t)m.s_out;
    Out o;
    if (run.sums) {
        const uint32_t tp = run.sum_threads * run.sum_prep;
        const uint32_t set = (sim / tp) * run.sum_threads + sim % run.sum_threads;
        o.samples = nullptr;
        o.sums = run.sums + (size_t)set * row_words;
    } else {
        o.samples = run.out + (size_t)sim * row_words;
        o.sums = nullptr;
    }
    o.last = sl.last;
    return o;
}

// A0 == 0 (tau.cu:1665-1697, 2165-2196): the reference copies the last
// recorded sample forward (writing the current state first if none exists).
// No collectives: groups may take it alone.
template <int G, class M>
__device__ __forceinline__ void finish_zero(const M& m, const Run& run, Slot<M> sl, uint32_t lane, uint32_t sim,
                                                uint32_t cursor) {
    const int so = m.s_out;
    const uint32_t ns = (uint32_t)m.ns;
    const Out out = out_of(m, run, sl, sim);
    if (!(run.flags & F_Q10_OFF)) {
        if (cursor == 0) {
            for (int k = (int)lane; k < so; k += G) out.put(0u, so, k, (uint32_t)sl.x((int)m.cs[k]));
            cursor = 1;
        }
        // the row copied forward may be another warp's: its writes lie before
        // the fence with which that warp put the simulation back into the pool,
        // these reads behind the one with which this warp took it
        for (uint32_t i = cursor; i < ns; i++)
            for (int k = (int)lane; k < so; k += G) out.put(i, so, k, out.get(cursor - 1, so, k));
    } else {
        for (uint32_t i = cursor; i < ns; i++)
            for (int k = (int)lane; k < so; k += G) out.put(i, so, k, (uint32_t)sl.x((int)m.cs[k]));
    }
}

// PrepareVariables (tau.cu:1269-1297): simulation `sim` into slot j.  All
// lanes; groups with !act only take part in the barriers.
template <int G, class M>
__device__ __forceinline__ void init_sim(const Grp<G>& g, const M& m, const Run& run, const Slot<M>& sl,
                                         const StateArrays& sa, int j, uint32_t sim, bool act) {
    const int S = m.S, R = m.R, P = m.P;
    g.sync();
    if (act) {
        for (int s = (int)g.lane; s < S; s += G) sl.x(s) = run.X0[(size_t)sim * S + s];
        if (g.lane == 0) sl.x(S) = 1;
        for (int r = (int)g.lane; r < P; r += G) {
            if (!run.uniform_c) sl.c[r] = r < R ? run.c[(size_t)sim * R + r] : 0.0f;
            sl.am(m)[r] = 0.0f;
        }
    }
    g.sync();
    all_props<G>(g, m, sl, act);
    if (act && g.lane == 0) {
        sa.T[j] = 0.0;
        sa.tl[j] = 0.0;
        sa.tnext[j] = m.tvec[0];
        sa.fire[j] = 0ull;
        sa.sim[j] = sim;
        sa.cursor[j] = sa.n[j] = sa.burst[j] = sa.leaps[j] = sa.ssa[j] = sa.rej[j] = 0u;
        sa.status[j] = CTL_SIM_OK;
    }
    g.sync();
}

// ---------------------------------------------------------------------------
// Exact SSA
// ---------------------------------------------------------------------------

// Random parts of the next SSA steps, one Philox block (two steps) per lane:
// pick word and negated log of the waiting-time uniform.  They depend on the
// counters only, so a group prepares as many blocks at once as it has lanes
// in a warp instead of every lane computing every block.
struct Rng {
    uint32_t base;      // block of lane 0, or RNG_NONE
    uint32_t we, wo;    // pick words of the even and odd step
    float le, lo;       // -log(u) of the even and odd step
};
constexpr uint32_t RNG_NONE = 0x80000000u;

__device__ __forceinline__ void rng_fill(const Run& run, uint32_t wl, uint32_t sim, uint32_t step, Rng& q) {
    q.base = step >> 1;
    const uint4 w = draw_small(run.seed, 0u, TAG_SSA, q.base + wl, run.sim_base + sim);
    q.we = w.x;
    q.le = -flog(u24f(w.y));
    q.wo = w.z;
    q.lo = -flog(u24f(w.w));
}

// EventualSSASteps / LightweightSSA (tau.cu:2099-2454): up to run.ssa_budget
// direct-method steps of the simulations in the warp's groups (has: this group
// holds one, in slot j), all in lockstep; a group that has left the burst runs
// along without effect.  Returns the simulation's phase.
template <int G, class M>
__device__ __forceinline__ uint32_t run_ssa(const Grp<G>& g, const M& m, const Run& run, const Slot<M>& sl,
                                            const StateArrays& sa, int j, bool has) {
    const uint32_t ns = (uint32_t)m.ns;
    const uint32_t lane = g.lane;
    constexpr uint32_t L = (uint32_t)Grp<G>::L;
    const double T = sa.T[j];
    double tl = sa.tl[j], t_next = sa.tnext[j];
    const uint32_t sim = sa.sim[j], n0 = sa.n[j];
    uint32_t cursor = sa.cursor[j], n = n0, burst = sa.burst[j];
    uint32_t phase = PH_SSA, status = CTL_SIM_OK;
    Rng q;
    q.base = RNG_NONE;
    bool act = has;
    for (uint32_t b = 0; b < run.ssa_budget; b++) {
        if (G >= 32 ? !act : !__any_sync(FULL, act)) break;
        Tree<G, M> t;
        tree_build<G>(g, m, sl, 0, t);
        const double A0 = t.root;
        if (act & ((n >= run.max_steps) | (A0 == 0.0))) {
            status = n >= run.max_steps ? (uint32_t)CTL_SIM_STEP_LIMIT : ST_NOTHING;
            phase = PH_DONE;
            act = false;
        }
        // one Philox block per two SSA steps: (w0,w1) for even steps, (w2,w3)
        // for odd ones; 32-bit pick uniform, FP32 waiting time
        if (__any_sync(FULL, act && (n >> 1) - q.base >= L)) rng_fill(run, lane & (L - 1u), sim, n, q);
        uint32_t w = (n & 1u) ? q.wo : q.we;
        float lg = (n & 1u) ? q.lo : q.le;
        if constexpr (G > 1) {
            const int src = (int)(((n >> 1) - q.base) & (L - 1u));
            w = __shfl_sync(FULL, w, src, (int)L);
            lg = __shfl_sync(FULL, lg, src, (int)L);
        }
        int r = descend<G>(g, m, sl, t, u32d(w) * A0, 0);
        r = act ? r : 0;
        const uint4 f = m.fire[r];
        const uint32_t ne = act ? f.y : 0u, nd = act ? f.w : 0u;
        // the first dependent's descriptors are on their way while X changes
        uint4 d = make_uint4(0u, 0u, 0u, 0u);
        if (lane < nd) d = m.dep[f.z + lane];
        uint32_t ent = 0u;
        if (lane < ne) ent = m.fr_ent[f.x + lane];
        const float dtf = lg / (float)A0;
        tl = act ? tl + (double)dtf : tl;
        if (act & (T + tl > t_next) & (cursor < ns)) {
            const int so = m.s_out;
            const Out out = out_of(m, run, sl, sim);
            do {
                for (int k = (int)lane; k < so; k += G) out.put(cursor, so, k, (uint32_t)sl.x((int)m.cs[k]));
                cursor++;
                t_next = cursor < ns ? m.tvec[cursor] : 0.0;
            } while (cursor < ns && T + tl > t_next);
        }
        g.sync();
        // |change| <= 127: the sum wraps negative exactly when it leaves [0, 2^31)
        bool lovf = false;
        if (lane < ne) {
            int32_t& x = sl.x((int)(ent >> 8));
            const int32_t nx = (int32_t)((uint32_t)x + (uint32_t)(int32_t)(int8_t)(ent & 0xffu));
            lovf = nx < 0;
            x = nx;
        }
        if (m.changes > G)
            for (uint32_t e = lane + G; e < ne; e += G) {
                const uint32_t en = m.fr_ent[f.x + e];
                int32_t& x = sl.x((int)(en >> 8));
                const int32_t nx = (int32_t)((uint32_t)x + (uint32_t)(int32_t)(int8_t)(en & 0xffu));
                lovf |= nx < 0;
                x = nx;
            }
        n += act ? 1u : 0u;
        burst += act ? 1u : 0u;
        const bool ovf = g.any(lovf);
        if (ovf) {
            status = CTL_SIM_OVERFLOW;
            phase = PH_DONE;
        }
        g.sync();
        // new propensities of the reactions that depend on the changed species
        for (uint32_t i = lane; i < nd;) {
            const uint4 e = d;
            i += G;
            if (i < nd) d = m.dep[f.z + i];
            sl.a(m)[e.w] = prop(m, sl, (int)e.x, e.y, e.z);
        }
        g.sync();
        if (act) {
            if (cursor == ns && phase == PH_SSA) phase = PH_DONE;
            act = phase == PH_SSA && burst != run.ssa_steps;
        }
    }
    if (has) {
        const uint32_t ran = n - n0;
        double Te = status == ST_NOTHING ? m.tmax + (double)0.1f : T;
        if (phase == PH_SSA && burst == run.ssa_steps) {
            Te = T + tl;
            tl = 0.0;
            burst = 0;
            if (!(run.flags & F_FORCE_SSA)) phase = PH_DECIDE;
            else if (Te >= m.tmax) phase = PH_DONE;
        }
        if (lane == 0) {
            sa.T[j] = Te;
            sa.tl[j] = tl;
            sa.tnext[j] = t_next;
            sa.cursor[j] = cursor;
            sa.n[j] = n;
            sa.burst[j] = burst;
            sa.ssa[j] += ran;
            sa.status[j] = status;
        }
    }
    g.sync();
    return phase;
}

// ---------------------------------------------------------------------------
// Leap decisions
// ---------------------------------------------------------------------------

// Critical reactions (tau.cu:1727-1733): some reactant with
// 0 < floor(x / L) < n_c.  floor(x / L) < n_c  <=>  x < n_c * L and
// floor(x / L) > 0  <=>  x >= L (x >= 0, L >= 1): the reference's integer
// test without a division.  Fills am (0 for critical reactions); true when
// this lane saw a critical one.
template <int G, class M>
__device__ __forceinline__ bool critical_pass(const Grp<G>& g, const M& m, const Run& run, const Slot<M>& sl,
                                              bool act) {
    const bool q6off = (run.flags & F_Q6_OFF) != 0;
    // n_c L, saturated above every count; x - low < span is then the test for
    // coefficients 1 and 2 (and never true for the dummy's 0)
    const uint32_t lim1 = run.nc < 0x80000000u ? run.nc : 0x80000000u;
    const uint32_t lim2 = run.nc < 0x40000000u ? 2u * run.nc : 0x80000000u;
    const uint32_t low = q6off ? 0u : 3u;
    const uint32_t span1 = q6off ? lim1 : lim1 > 1u ? lim1 - 1u : 0u;
    const uint32_t span2 = q6off ? lim2 : lim2 > 2u ? lim2 - 2u : 0u;
    bool lany = false;
#pragma unroll 2
    for (int r = (int)g.lane; r < m.R; r += G) {
        bool cr = false;
        const uint2 d = m.reac_desc[r];
        if (!m.general || d.x != DESC_GENERAL) {
            const uint32_t x = (uint32_t)sl.xb(d.x & ~3u) - (d.x & low), y = (uint32_t)sl.xb(d.y & ~3u) - (d.y & low);
            cr = (x < ((d.x & 2u) ? span2 : (d.x & 1u) ? span1 : 0u)) | (y < ((d.y & 2u) ? span2 : (d.y & 1u) ? span1 : 0u));
        } else {
            const uint32_t e1 = m.reac_off[r + 1];
            for (uint32_t e = m.reac_off[r]; e < e1; e++) {
                const uint32_t ent = m.reac_ent[e];
                const uint32_t x = (uint32_t)sl.x((int)(ent >> 8)), Lc = ent & 0xffu;
                const bool below = (uint64_t)x < (uint64_t)run.nc * Lc;
                cr = cr || (q6off ? below : (x >= Lc && below));
            }
        }
        if (act) sl.am(m)[r] = cr ? 0.0f : sl.pa(m, r);
        lany |= cr;
    }
    return lany;
}

// The leap's Poisson counts.  A warp's reactions are first sorted by how they
// are drawn: inversion with a mean below 1 (a few trips), inversion with a mean
// below 10, and PTRS; its lanes then run one of these at a time, each on a full
// warp's worth of reactions, instead of every pair of reactions paying for the
// longest path of 32 lanes.  PTRS draws that its squeeze does not accept (about
// one in seven) are collected likewise for the full test.  Reaction r reads
// words (0, 1) or (2, 3) of the block of its pair r / 2.
template <int G, class M>
__device__ __forceinline__ void poisson_pass(const Grp<G>& g, const M& m, const Run& run, const Slot<M>& sl,
                                             uint32_t simg, uint32_t step, uint32_t attempt, double tau, int pick,
                                             bool act) {
    constexpr int L = Grp<G>::L;
    const uint32_t wl = g.lane & (uint32_t)(L - 1), below = (1u << wl) - 1u;
    const bool keep = attempt == 0 || (run.flags & F_Q3_OFF);
    // this warp's share of the two list areas: [0] tiny means from the front,
    // small ones from the back; [1] PTRS
    const int room = G > 32 ? m.P / Grp<G>::W : m.P;
    uint16_t* list = sl.list(m) + (G > 32 ? (int)g.warp() * room : 0);
    uint16_t* large = list + m.P;
    int nt = 0, nsm = 0, nlg = 0;
    uint32_t* K = sl.k(m);
    const float* am = sl.am(m);
#pragma unroll 1
    for (int r0 = 0; r0 < m.R; r0 += G) {
        const int r = r0 + (int)g.lane;
        bool ti = false, sm = false, lg = false;
        if (act && r < m.R) {
            const float a = am[r];
            if (a > 0.0f) {
                const double lam = tau * (double)a;
                ti = lam < 1.0;
                sm = !ti & (lam < 10.0);
                lg = !(ti | sm);
            } else {
                K[r] = (r == pick) & keep ? 1u : 0u;
            }
        }
        uint32_t bt = ti ? 1u : 0u, bs = sm ? 1u : 0u, bl = lg ? 1u : 0u;
        if constexpr (G > 1) {
            bt = g.seg(__ballot_sync(FULL, ti));
            bs = g.seg(__ballot_sync(FULL, sm));
            bl = g.seg(__ballot_sync(FULL, lg));
        }
        if (ti) list[nt + __popc(bt & below)] = (uint16_t)r;
        if (sm) list[room - 1 - nsm - __popc(bs & below)] = (uint16_t)r;
        if (lg) large[nlg + __popc(bl & below)] = (uint16_t)r;
        nt += __popc(bt);
        nsm += __popc(bs);
        nlg += __popc(bl);
    }
    __syncwarp();
    auto words = [&](int r) {
        const uint4 w = draw_small(run.seed, 0u, tag_pois(attempt, (uint32_t)r >> 1), step, simg);
        return (r & 1) ? make_uint2(w.z, w.w) : make_uint2(w.x, w.y);
    };
    // the tiny means, then the small ones
#pragma unroll 1
    for (int part = 0; part < 2; part++) {
        const int n = part ? nsm : nt;
        for (int i = (int)wl; i < n; i += L) {
            const int r = list[part ? room - 1 - i : i];
            K[r] = poisson_inversion(tau * (double)am[r], words(r).x);
        }
        __syncwarp();
    }
    int nslow = 0;
    for (int i0 = 0; (G == 1 ? i0 < nlg : __any_sync(FULL, i0 < nlg)); i0 += L) {
        const int i = i0 + (int)wl;
        bool slow = false;
        int r = 0;
        if (i < nlg) {
            r = large[i];
            const uint2 w = words(r);
            uint32_t k;
            slow = !poisson_ptrs_quick(tau * (double)am[r], w.x, w.y, k);
            if (!slow) K[r] = k;
        }
        if constexpr (G > 1) {
            const uint32_t b = g.seg(__ballot_sync(FULL, slow));  // also orders the reads above before the writes below
            if (slow) large[nslow + __popc(b & below)] = (uint16_t)r;
            nslow += __popc(b);
        } else {
            if (slow) large[nslow] = (uint16_t)r;
            nslow += slow ? 1 : 0;
        }
    }
    __syncwarp();
    for (int i = (int)wl; i < nslow; i += L) {
        const int r = large[i];
        const uint2 w = words(r);
        K[r] = poisson_ptrs(tau * (double)am[r], w.x, w.y, run.seed, tag_pois(attempt, (uint32_t)r >> 1), step, simg,
                            (uint32_t)r & 1u);
    }
    __syncwarp();
}

struct Sim {
    double T, tl, t_next;
    unsigned long long fire;  // this lane's share of the leap firings
    uint32_t sim, cursor, n, burst, leaps, rej, status;
    bool in_ssa;
};
constexpr int CONT = 0, DONE = 1;

// PreCalculations (tau.cu:1568-2093): the SSA hand-off decision and, unless
// it hands off, one Cao tau-leap with critical reactions and rejection, for
// every group with act.
template <int G, class M>
__device__ __forceinline__ int decide_step(const Grp<G>& g, const M& m, const Run& run, const Slot<M>& sl, Sim& st,
                                           bool act) {
    const int S = m.S, R = m.R, so = m.s_out;
    const uint32_t ns = (uint32_t)m.ns;
    const uint32_t fl = run.flags;
    const uint32_t lane = g.lane;
    const uint32_t simg = run.sim_base + st.sim;
    int res = CONT;
    double A0;
    {
        Tree<G, M> t;
        tree_build<G>(g, m, sl, 0, t);
        A0 = t.root;
    }
    const uint32_t step = st.n;
    if (act) {
        if (st.T >= m.tmax) {
            res = DONE;
        } else if (step >= run.max_steps) {
            st.status = CTL_SIM_STEP_LIMIT;
            res = DONE;
        } else {
            st.n = step + 1u;
            if (A0 == 0.0) {
                st.status = ST_NOTHING;
                st.T = m.tmax + (double)0.1f;
                res = DONE;
            }
        }
    }
    act = act && res == CONT;
    int pick = -1;
    double tau = 0.0;
    bool todo = act;
    for (uint32_t attempt = 0;; attempt++) {
        // (again after a rejection: the counts took am's place)
        const bool anycrit = g.any(critical_pass<G>(g, m, run, sl, todo));
        g.sync();
        if (attempt == 0u) {
            float t1 = FLT_MAX;
#pragma unroll 1
            for (int i = (int)lane; i < S; i += G) {
                const uint4 sp = m.v_sp[i];
                if (sp.z == 0u) continue;
                float mu = 0.0f, sg = 0.0f;
#pragma unroll 2
                for (uint32_t e = sp.y; e < sp.y + sp.z; e++) {
                    // critical reactions add an exact +-0: mu and sg start at +0 and
                    // are never -0, so the sums equal those that skip them
                    const uint32_t ent = m.v_ent[e];
                    const float a = sl.am(m)[(int)(ent >> 8)];
                    const float fv = (float)(int8_t)(ent & 0xffu);
                    mu = mu + fv * a;
                    sg = sg + (fv * fv) * a;
                }
                const int32_t xs = sl.x((int)sp.x);
                // division by g_i = 1 and 2 is exact scaling
                float tmp2 = run.eps * (float)xs;
                if (sp.w != 1u) {
                    const float gg = gfun(sp.w & 0xffu, sp.w >> 8, xs);
                    tmp2 = gg == 2.0f ? tmp2 * 0.5f : tmp2 / gg;
                }
                const float macs = tmp2 > 1.0f ? tmp2 : 1.0f;
                const bool use = (fl & F_Q9_OFF) ? (sg != 0.0f) : (mu != 0.0f && sg != 0.0f);
                if (use) {
                    const float t3 = mu != 0.0f ? macs / fabsf(mu) : __int_as_float(0x7f800000);
                    const float t4 = (macs * macs) / sg;
                    const float tt = t3 < t4 ? t3 : t4;
                    if (tt < t1) t1 = tt;
                }
            }
            const float tau1 = g.fmin(t1);
            if (act && (double)tau1 < run.ssa_factor / A0) {
                st.in_ssa = true;
                st.burst = 0;
                st.tl = 0.0;
                act = false;
            }
            todo = act;
            // from here on only the leaping groups
            if (G > 32 ? !act : !__any_sync(FULL, act)) return res;
            tau = (double)tau1;
            if (G > 32 ? anycrit : __any_sync(FULL, act && anycrit)) {
                // the critical tree, then, for the pick, the one with leaf 0
                // unmasked: the reference's linear search starts from PROP[0] (Q2)
                const int pick_mode = (fl & F_Q2_OFF) ? 1 : 2;
                Tree<G, M> tc;
                double a0c = 0.0;
                uint4 wd = make_uint4(0u, 0u, 0u, 0u);
                bool crit_first = false;
#pragma unroll 1
                for (int mode = 1; mode <= pick_mode; mode++) {
                    tree_build<G>(g, m, sl, mode, tc);
                    if (mode == 1) {
                        a0c = anycrit ? tc.root : 0.0;
                        double tau2 = (double)FLT_MAX;
                        if (act && a0c > 0.0) {
                            wd = draw_small(run.seed, 0u, TAG_MISC, step, simg);
                            tau2 = -dlog(u53(wd.x, wd.y)) / a0c;
                        }
                        crit_first = act && (double)tau1 > tau2;
                        tau = (double)tau1 < tau2 ? (double)tau1 : tau2;
                        if (G > 32 ? !crit_first : !__any_sync(FULL, crit_first)) break;
                    }
                }
                if (G > 32 ? crit_first : __any_sync(FULL, crit_first)) {
                    const int p = descend<G>(g, m, sl, tc, u53(wd.z, wd.w) * a0c, pick_mode);
                    if (crit_first) pick = p;
                }
            }
            g.sync();  // the lists take the propensities' place
        }
        poisson_pass<G>(g, m, run, sl, simg, step, attempt, tau, pick, todo);
        g.sync();
        // test_update (tau.cu:1300-1351): rejected as soon as a partial sum, in
        // reaction order, is negative (Q4)
        bool lfail = false, lovf = false;
        const bool every = !(fl & F_Q4_OFF);
        if (todo) {
#pragma unroll 1
            for (int i = (int)lane; i < S; i += G) {
                const uint4 sp = m.fs_sp[i];
                int64_t x1 = sl.x((int)sp.x);
#pragma unroll 2
                for (uint32_t e = sp.y; e < sp.y + sp.z; e++) {
                    const uint32_t ent = m.fs_ent[e];
                    x1 += (int64_t)(int8_t)(ent & 0xffu) * (int64_t)(int32_t)sl.k(m)[(int)(ent >> 8)];
                    lfail |= (x1 < 0) & every;
                }
                lfail |= x1 < 0;
                lovf |= x1 > 2147483647LL;
                sl.x1(m, (int)sp.x) = (int32_t)x1;
            }
        }
        const bool fail = g.any(lfail), ovf = g.any(lovf);
        const bool again = todo && fail;
        bool commit = todo && !fail;
        if (again) {
            tau = tau * 0.5;
            st.rej++;
            if (attempt + 1u >= MAX_ATTEMPTS) {
                st.status = CTL_SIM_ATTEMPT_LIMIT;
                res = DONE;
            }
        } else if (commit && ovf) {
            st.status = CTL_SIM_OVERFLOW;
            res = DONE;
            commit = false;
        }
        todo = again && res == CONT;
        if (commit) {
            // check_time_instant (tau.cu:1507-1562)
            const double T = st.T;
            if (st.cursor < ns && T + tau >= st.t_next) {
                const Out out = out_of(m, run, sl, st.sim);
                do {
                    for (int k = (int)lane; k < so; k += G) {
                        const int s = (int)m.cs[k];
                        const int32_t xs = sl.x(s);
                        const double d = (double)((int64_t)sl.x1(m, s) - (int64_t)xs);
                        const double delta = (d * (st.t_next - T)) / tau;
                        const double ri = rint(delta);
                        uint32_t v;
                        if (!(fl & F_Q1_OFF))
                            v = (uint32_t)xs + (ri > 0.0 ? (uint32_t)ri : 0u);
                        else
                            v = (uint32_t)((int64_t)xs + (int64_t)ri);
                        out.put(st.cursor, so, k, v);
                    }
                    st.cursor++;
                    st.t_next = st.cursor < ns ? m.tvec[st.cursor] : 0.0;
                } while (st.cursor < ns && T + tau >= st.t_next);
            }
            unsigned long long fs = 0;
#pragma unroll 4
            for (int r = (int)lane; r < R; r += G) fs += sl.k(m)[r];
            st.fire += fs;
            st.leaps++;
            st.T = T + tau;
            if (st.cursor == ns) res = DONE;
        }
        g.sync();
        if (commit)
#pragma unroll 2
            for (int s = (int)lane; s < S; s += G) sl.x(s) = sl.x1(m, s);
        g.sync();
        // of the new state, or, before another attempt, of the old one (the
        // lists and X1 took their place)
        all_props<G>(g, m, sl, commit || todo);
        if (G > 32 ? !todo : !__any_sync(FULL, todo)) break;
    }
    return res;
}

// Up to run.dec_budget decisions of the simulations in the warp's groups, as
// run_ssa.
template <int G, class M>
__device__ __forceinline__ uint32_t run_dec(const Grp<G>& g, const M& m, const Run& run, const Slot<M>& sl,
                                            const StateArrays& sa, int j, bool has) {
    Sim st;
    st.T = sa.T[j];
    st.tl = sa.tl[j];
    st.t_next = sa.tnext[j];
    st.fire = 0ull;
    st.sim = sa.sim[j];
    st.cursor = sa.cursor[j];
    st.n = sa.n[j];
    st.burst = sa.burst[j];
    st.leaps = st.rej = 0u;
    st.status = CTL_SIM_OK;
    st.in_ssa = false;
    int res = CONT;
    for (uint32_t b = 0; b < run.dec_budget; b++) {
        const bool act = has && res == CONT && !st.in_ssa;
        if (G >= 32 ? !act : !__any_sync(FULL, act)) break;
        const int x = decide_step<G>(g, m, run, sl, st, act);
        res = act ? x : res;
    }
    const unsigned long long f = g.sum(st.fire);
    if (has && g.lane == 0) {
        sa.T[j] = st.T;
        sa.tl[j] = st.tl;
        sa.tnext[j] = st.t_next;
        sa.fire[j] += f;
        sa.cursor[j] = st.cursor;
        sa.n[j] = st.n;
        sa.burst[j] = st.burst;
        sa.leaps[j] += st.leaps;
        sa.rej[j] += st.rej;
        sa.status[j] = st.status;
    }
    g.sync();
    return res == DONE ? PH_DONE : st.in_ssa ? PH_SSA : PH_DECIDE;
}

// The record and, if asked, the host copy of a finished simulation's rows,
// for every group with act.
template <int G, class M>
__device__ __forceinline__ void finish_sim(const Grp<G>& g, const M& m, const Run& run, const Slot<M>& sl,
                                           const StateArrays& sa, int j, bool act) {
    const int so = m.s_out;
    const uint32_t sim = act ? sa.sim[j] : 0u;
    const Out out = out_of(m, run, sl, sim);
    const bool nothing = act && sa.status[j] == ST_NOTHING;
    if (nothing) finish_zero<G>(m, run, sl, g.lane, sim, sa.cursor[j]);
    if (act && !nothing && out.samples)  // rows never reached read 0 (a sum gains nothing from them)
        for (uint32_t i = sa.cursor[j]; i < (uint32_t)m.ns; i++)
            for (int k = (int)g.lane; k < so; k += G) out.samples[(size_t)i * so + k] = 0u;
    if (act && g.lane == 0) {
        ctl_sim_info inf;
        inf.t_final = sa.T[j] + sa.tl[j];
        inf.firings = sa.fire[j] + sa.ssa[j];  // every SSA step fires one reaction
        inf.status = nothing ? (uint32_t)CTL_SIM_OK : sa.status[j];
        inf.steps = sa.n[j];
        inf.leaps = sa.leaps[j];
        inf.ssa_steps = sa.ssa[j];
        inf.rejections = sa.rej[j];
        inf.pad = 0;
        run.info[sim] = inf;
    }
    if (run.out_host && out.samples) {
        // rows that this group wrote are visible to its lanes after the barrier,
        // those of warps that held the simulation before by the pool's fences;
        // the group copies them all to the caller's pinned buffer (16-byte
        // stores when the row allows)
        g.sync();
        if (act) {
            const size_t words = (size_t)m.ns * (size_t)so;
            const uint32_t* src = out.samples;
            uint32_t* dst = run.out_host + (size_t)sim * words;
            if ((words & 3u) == 0u &&
                ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0u) {
                const uint4* s4 = reinterpret_cast<const uint4*>(src);
                uint4* d4 = reinterpret_cast<uint4*>(dst);
                for (size_t i = g.lane; i < words / 4; i += G) d4[i] = s4[i];
            } else {
                for (size_t i = g.lane; i < words; i += G) dst[i] = src[i];
            }
        }
    }
    if (run.done) {  // publish: this simulation's rows and record are complete
        __threadfence();
        g.sync();
        if (act && g.lane == 0) atomicAdd(run.done + (sim >> run.done_shift), 1u);
    }
}

template <class M>
__device__ __forceinline__ Slot<M> slot_of(unsigned char* smem, const Layout& lay, int j, bool uniform_c) {
    Slot<M> sl;
    sl.b = smem + (size_t)j * lay.slot;
    sl.c = reinterpret_cast<float*>(uniform_c ? smem + lay.off_c : sl.b + lay.oc);
    sl.last = reinterpret_cast<uint32_t*>(sl.b + lay.olast);
    return sl;
}

// The next simulation from the device work queue into slot j (groups with
// want); its phase, PH_CLOSED when the queue is empty.
template <int G, class M>
__device__ __forceinline__ uint32_t refill(const Grp<G>& g, const M& m, const Run& run, const Slot<M>& sl,
                                           const StateArrays& sa, int j, bool want) {
    uint32_t sim = 0;
    if (want && g.lane == 0) sim = atomicAdd(run.queue, 1u);
    sim = g.bcast(sim);
    const bool got = want && sim < run.n;
    init_sim<G>(g, m, run, sl, sa, j, got ? sim : 0u, got);
    return !got ? PH_CLOSED : (run.flags & F_FORCE_SSA) ? PH_SSA : PH_DECIDE;
}

// The simulations of a block that wait for a warp, one bit per slot and
// phase.  A warp takes as many as it has groups with one atomic per word and
// puts them back when their stretch of work is over: no barrier, and no
// simulation waits for another warp's.
constexpr int POOL_WORDS = 10;  // slots per block / 32, at most
struct Pool {
    uint32_t ready[2][POOL_WORDS];
    uint32_t live;  // slots not closed
};
// Polls of an idle warp (other warps hold the pool's simulations) before it
// leaves the block; whoever holds them carries on.
constexpr uint32_t IDLE_POLLS = 1u << 16;

// Takes up to `want` simulations of phase ph from the bits `within` of words
// [w0, w1): the slot of the `mine`-th one, or -1.  All lanes of the warp.
__device__ __forceinline__ int pool_take(Pool& p, uint32_t ph, uint32_t w0, uint32_t w1, uint32_t within, uint32_t want,
                                         uint32_t mine) {
    const uint32_t lane = threadIdx.x & 31u;
    int slot = -1;
    uint32_t have = 0;
    for (uint32_t w = w0; w < w1 && have < want; w++) {
        uint32_t got = 0;
        if (lane == 0) {
            uint32_t pick = *(volatile uint32_t*)&p.ready[ph][w] & within, n = have;
            uint32_t m = 0;
            while (pick && n < want) {
                m |= pick & (0u - pick);
                pick &= pick - 1u;
                n++;
            }
            if (m) got = atomicAnd(&p.ready[ph][w], ~m) & m;
        }
        got = __shfl_sync(FULL, got, 0);
        const uint32_t c = __popc(got);
        if (mine >= have && mine < have + c) {
            uint32_t b = got;
            for (uint32_t i = have; i < mine; i++) b &= b - 1u;
            slot = (int)(32u * w) + __ffs(b) - 1;
        }
        have += c;
    }
    return slot;
}

// Persistent sweep.  Every slot of a block holds a simulation until the device
// work queue is empty.  Groups of one warp or more keep their slot and run its
// phases in turn.  The smaller groups' warps take simulations of one phase
// from the block's pool (or, warp-local, from their own slots), as many as
// they have groups, advance them in lockstep by a stretch of SSA steps or
// decisions, and put them back: with more slots than groups, decisions wait
// until a warp's worth of them has come together while the other warps go on
// stepping.  MINB selects the register budget: compiled so that MINB blocks of
// 256 threads can be resident per SM (2: up to 128 registers per thread, 3:
// 80, 4: 64, spilling to local memory as needed).  sweep_body is the kernel's
// body for either model type; sweep_kernel is the library's kernel.
template <int G, class M>
__device__ __forceinline__ void sweep_body(const M& m, const Run& run, const Layout& lay) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Pool pool;
    const int NS = (int)lay.ns, NG = (int)(blockDim.x / G);
    const int gi = (int)(threadIdx.x / G);
    Grp<G> g;
    if constexpr (G > 32) g.scratch(smem + lay.off_grp);
    StateArrays sa;
    {
        unsigned char* b = smem + lay.off_state;
        sa.T = reinterpret_cast<double*>(b);
        sa.tl = sa.T + NS;
        sa.tnext = sa.tl + NS;
        sa.fire = reinterpret_cast<unsigned long long*>(sa.tnext + NS);
        uint32_t* u = reinterpret_cast<uint32_t*>(sa.fire + NS);
        sa.sim = u;
        sa.cursor = u + NS;
        sa.n = u + 2 * NS;
        sa.burst = u + 3 * NS;
        sa.leaps = u + 4 * NS;
        sa.ssa = u + 5 * NS;
        sa.rej = u + 6 * NS;
        sa.status = u + 7 * NS;
    }
    const bool uni = run.uniform_c != 0;
    if (uni) {
        float* cs = reinterpret_cast<float*>(smem + lay.off_c);
        for (int r = (int)threadIdx.x; r < m.P; r += (int)blockDim.x) cs[r] = r < m.R ? run.c[r] : 0.0f;
    }
    // slots and scalars start as zeros: groups without a simulation run along
    // on theirs, and every index they form from it is in range
    for (uint32_t i = threadIdx.x; i < lay.off_c / 4u; i += blockDim.x) reinterpret_cast<uint32_t*>(smem)[i] = 0u;
    if (threadIdx.x < 2u * POOL_WORDS) (&pool.ready[0][0])[threadIdx.x] = 0u;
    if (threadIdx.x == 0) pool.live = (uint32_t)NS;
    __syncthreads();
    if constexpr (G >= 32) {
        const Slot<M> sl = slot_of<M>(smem, lay, gi, uni);
        uint32_t ph = refill<G>(g, m, run, sl, sa, gi, true);
        while (ph != PH_CLOSED) {
            if (ph == PH_SSA) ph = run_ssa<G>(g, m, run, sl, sa, gi, true);
            else ph = run_dec<G>(g, m, run, sl, sa, gi, true);
            if (ph == PH_DONE) {
                finish_sim<G>(g, m, run, sl, sa, gi, true);
                ph = refill<G>(g, m, run, sl, sa, gi, true);
            }
        }
    } else {
        constexpr uint32_t GPW = 32u / G;  // groups per warp
        const uint32_t warp = threadIdx.x >> 5, mine = (threadIdx.x & 31u) / G;
        // the pool's words: the block's, or this warp's own slots
        uint32_t w0 = 0, w1 = ((uint32_t)NS + 31u) / 32u;
        uint32_t within = FULL;
        if (run.warp_local) {
            w0 = warp * GPW / 32u;
            w1 = w0 + 1u;
            within = (GPW == 32u ? FULL : (1u << (GPW & 31u)) - 1u) << (warp * GPW % 32u);
        }
        int j = -1;            // the slot this group holds
        uint32_t ph = PH_DONE; // its phase; PH_DONE: a slot to fill
        int fresh = gi;        // the next slot this group fills at the start
        uint32_t idle = 0;
        for (;;) {
            // fill the slots this group starts with, then work
            const bool filling = fresh < NS;
            if (__any_sync(FULL, filling)) {
                if (filling) j = fresh;
                fresh += NG;
                ph = filling ? PH_DONE : PH_CLOSED;
            } else {
                if (run.warp_local) __syncwarp();
                uint32_t nready[2] = {0u, 0u};
                for (uint32_t w = w0; w < w1; w++) {
                    nready[0] += __popc(*(volatile uint32_t*)&pool.ready[0][w] & within);
                    nready[1] += __popc(*(volatile uint32_t*)&pool.ready[1][w] & within);
                }
                nready[0] = __shfl_sync(FULL, nready[0], 0);
                nready[1] = __shfl_sync(FULL, nready[1], 0);
                if (nready[0] + nready[1] == 0u) {
                    // other warps hold what is left (or nothing is)
                    const uint32_t left = __shfl_sync(FULL, *(volatile uint32_t*)&pool.live, 0);
                    if (left == 0u || run.warp_local || ++idle > IDLE_POLLS) break;
                    __nanosleep(200);
                    continue;
                }
                idle = 0;
                const uint32_t take = nready[1] >= GPW || nready[1] > nready[0] ? PH_DECIDE : PH_SSA;
                j = pool_take(pool, take, w0, w1, within, GPW, mine);
                ph = j < 0 ? PH_CLOSED : take;
                __threadfence_block();  // the slots as their last warp left them
                __syncwarp();
                const bool has = j >= 0;
                const Slot<M> sl = slot_of<M>(smem, lay, has ? j : gi, uni);
                const uint32_t x = take == PH_SSA ? run_ssa<G>(g, m, run, sl, sa, has ? j : gi, has)
                                                  : run_dec<G>(g, m, run, sl, sa, has ? j : gi, has);
                if (has) ph = x;
                if (__any_sync(FULL, ph == PH_DONE)) finish_sim<G>(g, m, run, sl, sa, has ? j : gi, ph == PH_DONE);
            }
            if (__any_sync(FULL, ph == PH_DONE)) {
                const bool want = ph == PH_DONE;
                const Slot<M> sl = slot_of<M>(smem, lay, j >= 0 ? j : gi, uni);
                const uint32_t x = refill<G>(g, m, run, sl, sa, j >= 0 ? j : gi, want);
                if (want) {
                    ph = x;
                    if (x == PH_CLOSED && g.lane == 0) atomicSub(&pool.live, 1u);
                }
            }
            __threadfence_block();
            __syncwarp();
            if (j >= 0 && ph <= PH_DECIDE && g.lane == 0) atomicOr(&pool.ready[ph][(uint32_t)j >> 5], 1u << (j & 31));
            j = -1;
            __syncwarp();
        }
    }
}

template <int G, int MINB>
__global__ void __launch_bounds__(256, MINB) sweep_kernel(const __grid_constant__ Model m, const __grid_constant__ Run run,
                                                         const __grid_constant__ Layout lay) {
    sweep_body<G>(m, run, lay);
}

#ifndef __CUDACC_RTC__
// Host-side handle of the sweep kernel for G lanes per simulation in
// register budget minb (2, 3 or 4 resident 256-thread blocks per SM).
template <int G>
const void* sweep_kernel_ptr(int minb) {
    switch (minb) {
        case 3: return reinterpret_cast<const void*>(&sweep_kernel<G, 3>);
        case 4: return reinterpret_cast<const void*>(&sweep_kernel<G, 4>);
        default: return reinterpret_cast<const void*>(&sweep_kernel<G, 2>);
    }
}

}  // namespace dev

// One translation unit per group size (ctl_sweep_g<G>.cu) instantiates these.
const void* sweep_kernel_g1(int minb);
const void* sweep_kernel_g2(int minb);
const void* sweep_kernel_g4(int minb);
const void* sweep_kernel_g8(int minb);
const void* sweep_kernel_g16(int minb);
const void* sweep_kernel_g32(int minb);
const void* sweep_kernel_g64(int minb);
const void* sweep_kernel_g128(int minb);
const void* sweep_kernel_g256(int minb);

}  // namespace ctl
#else
}  // namespace dev
}  // namespace ctl
#endif
