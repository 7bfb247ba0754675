"""The sum tree of the shared-memory sweep for groups of several warps, run on
the CPU: ctl_sweep_dev.cuh is compiled by g++ with each lane as a coroutine, and
between two barriers one warp runs as far ahead of the others as the barriers
let it, first or last warp first.  Two trees built in a row, as a leap does with
its critical reactions, must both come out whole in every lane."""
import os
import re
import shutil
import subprocess

import pytest

import cutauleaping_b200 as ctl

CSRC = os.path.join(os.path.dirname(ctl.__file__), "csrc")

# What the device code takes from CUDA, for coroutines on one host thread.
SHIM = r'''
#pragma once
#include <ucontext.h>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#define __device__
#define __host__
#define __global__
#define __shared__
#define __constant__
#define __grid_constant__
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))
#define __restrict__
struct dim3u { unsigned x; };
inline dim3u threadIdx, blockIdx, blockDim;
struct uint2 { unsigned x, y; };
struct uint4 { unsigned x, y, z, w; };
struct float4 { float x, y, z, w; };
inline uint2 make_uint2(unsigned a, unsigned b) { return {a, b}; }
inline uint4 make_uint4(unsigned a, unsigned b, unsigned c, unsigned d) { return {a, b, c, d}; }
template <class T, class U> T bits(U v) { T r; static_assert(sizeof(T) == sizeof(U)); memcpy(&r, &v, sizeof r); return r; }
inline unsigned __float_as_uint(float v) { return bits<unsigned>(v); }
inline float __uint_as_float(unsigned v) { return bits<float>(v); }
inline float __int_as_float(int v) { return bits<float>(v); }
inline long long __double_as_longlong(double v) { return bits<long long>(v); }
inline double __longlong_as_double(long long v) { return bits<double>(v); }
inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)((uint64_t)a * b >> 32); }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __clz(int v) { return v ? __builtin_clz(v) : 32; }
inline void __threadfence() {}
inline void __threadfence_block() {}
inline void __nanosleep(unsigned) {}
template <class T> T atomicAdd(T* p, T v) { T o = *p; *p += v; return o; }
template <class T> T atomicSub(T* p, T v) { T o = *p; *p -= v; return o; }
template <class T> T atomicAnd(T* p, T v) { T o = *p; *p &= v; return o; }
template <class T> T atomicOr(T* p, T v) { T o = *p; *p |= v; return o; }

// Lanes: coroutines; one that waits names the counter it waits for.
struct Lane {
    ucontext_t ctx;
    std::vector<char> stack;
    const unsigned* gate = nullptr;
    unsigned past = 0;
    bool done = false;
};
inline std::vector<Lane> lanes;
inline ucontext_t home;
inline unsigned current;
inline void wait_for(const unsigned* gate, unsigned past) {
    lanes[current].gate = gate;
    lanes[current].past = past;
    while (*gate == past) swapcontext(&lanes[current].ctx, &home);
    lanes[current].gate = nullptr;
}
struct Meeting { unsigned here = 0, gen = 0; };
inline void meet(Meeting& m, unsigned n) {
    const unsigned g = m.gen;
    if (++m.here == n) { m.here = 0; m.gen++; }
    else wait_for(&m.gen, g);
}
inline Meeting warp_meet[8], bar_meet[16];
inline uint64_t slots[8][2][32];
inline const uint64_t* exchange(uint64_t v) {
    const unsigned w = current / 32;
    uint64_t* s = slots[w][warp_meet[w].gen & 1];
    s[current % 32] = v;
    meet(warp_meet[w], 32);
    return s;
}
template <class T> uint64_t widen(T v) { uint64_t r = 0; memcpy(&r, &v, sizeof v); return r; }
template <class T> T narrow(uint64_t v) { T r; memcpy(&r, &v, sizeof r); return r; }
template <class T> T __shfl_xor_sync(unsigned, T v, int o) { return narrow<T>(exchange(widen(v))[(current % 32) ^ o]); }
template <class T> T __shfl_sync(unsigned, T v, int l, int w = 32) {
    return narrow<T>(exchange(widen(v))[(current % 32) / w * w + (l & (w - 1))]);
}
inline unsigned __ballot_sync(unsigned, bool p) {
    const uint64_t* s = exchange(p);
    unsigned r = 0;
    for (int i = 0; i < 32; i++) r |= (unsigned)s[i] << i;
    return r;
}
inline bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }
inline void __syncwarp() { exchange(0); }
inline void __syncthreads() { meet(bar_meet[0], (unsigned)lanes.size()); }
inline void emu_bar(unsigned id, unsigned n) { meet(bar_meet[id], n); }
'''

MAIN = r'''
#include "sweep_dev.h"
using namespace ctl::dev;
constexpr int G = LANES, P = 1024, S = 4;
static Model model;
static std::vector<unsigned char> slot(lay_end(S, P)), scratch(Grp<G>::SCRATCH);
struct Seen { double root[2]; int leaf[2]; };
static std::vector<Seen> seen(G);
static double where(const Tree<G, Model>& t) { return 0.37 * t.root; }
static void lane_main() {
    Grp<G> g;
    g.scratch(scratch.data());
    Slot<Model> sl;
    sl.b = slot.data();
    Tree<G, Model> t;
    const unsigned me = current;
    for (int mode = 1; mode <= 2; mode++) {  // the critical tree, then with leaf 0 unmasked
        tree_build<G>(g, model, sl, mode, t);
        seen[me].root[mode - 1] = t.root;
    }
    seen[me].leaf[1] = descend<G>(g, model, sl, t, where(t), 2);
    lanes[me].done = true;
    swapcontext(&lanes[me].ctx, &home);
}
static double tree_sum(const std::vector<double>& v, size_t i, size_t n) {
    return n == 1 ? v[i] : tree_sum(v, i, n / 2) + tree_sum(v, i + n / 2, n / 2);
}
int main() {
    model.S = S;
    model.R = model.P = P;
    Slot<Model> sl;
    sl.b = slot.data();
    std::vector<double> crit(P);
    uint32_t x = 12345;
    for (int r = 0; r < P; r++) {
        x = x * 1664525u + 1013904223u;
        const float a = (float)(x >> 8) * 1e-3f;
        const bool critical = r % 3 == 1;
        sl.pa(model, r) = a;
        sl.am(model)[r] = critical ? 0.0f : a;
        crit[r] = critical ? (double)a : 0.0;
    }
    const double root1 = tree_sum(crit, 0, P);
    crit[0] = (double)sl.pa(model, 0);
    const double root2 = tree_sum(crit, 0, P);
    size_t lo = 0;
    double rest = 0.37 * root2;
    for (size_t n = P / 2; n; n /= 2) {
        const double L = tree_sum(crit, lo, n), R = tree_sum(crit, lo + n, n);
        if (rest > L && R != 0.0) { rest = rest - L; lo += n; }
    }
    int bad = 0;
    for (int order = 0; order < 2; order++) {
        lanes = std::vector<Lane>(G);
        for (unsigned i = 0; i < G; i++) {
            lanes[i].stack.resize(1 << 16);
            getcontext(&lanes[i].ctx);
            lanes[i].ctx.uc_stack.ss_sp = lanes[i].stack.data();
            lanes[i].ctx.uc_stack.ss_size = lanes[i].stack.size();
            makecontext(&lanes[i].ctx, lane_main, 0);
        }
        for (;;) {  // always the first (or last) lane that can run
            int next = -1;
            for (int k = 0; k < G && next < 0; k++) {
                const int i = order ? G - 1 - k : k;
                if (!lanes[i].done && (!lanes[i].gate || *lanes[i].gate != lanes[i].past)) next = i;
            }
            if (next < 0) break;
            current = threadIdx.x = (unsigned)next;
            swapcontext(&home, &lanes[next].ctx);
        }
        for (int i = 0; i < G; i++)
            if (!lanes[i].done || seen[i].root[0] != root1 || seen[i].root[1] != root2 || seen[i].leaf[1] != (int)lo) bad++;
    }
    printf("%d wrong\n", bad);
    return bad != 0;
}
'''


def _host_source(name):
    """The header with its inline assembly as calls of the shim."""
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r'asm volatile\("bar\.sync %0, %1;"[^;]*?"memory"\);', "emu_bar(bar, G);", text)
    text = re.sub(r'asm volatile\(\s*"\{\\n\\t\.reg \.pred a, b;.*?"memory"\);', "abort(); r = 0;", text, flags=re.S)
    return re.sub(r'asm\("r\w+\.approx\.ftz\.f(?:32|64) %0, %1;" : "=\w"\(y\) : "\w"\((\w)\)\);', r"y = 1 / \1;", text)


@pytest.mark.parametrize("G", [32, 64, 128, 256])
def test_trees_in_a_row_with_warps_apart(G, tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ is not installed")
    (tmp_path / "cuda_runtime.h").write_text(SHIM)
    for name, as_ in (("ctl_devmath.cuh", "ctl_devmath.cuh"), ("ctl_sweep_dev.cuh", "sweep_dev.h")):
        text = _host_source(name)
        assert not re.search(r"\basm\b", text), "inline assembly that the shim does not know"
        text = text.replace('"../../include/ctl.h"', f'"{os.path.join(CSRC, "..", "..", "include", "ctl.h")}"')
        (tmp_path / as_).write_text(text)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "tree")
    subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-w", f"-DLANES={G}", f"-I{tmp_path}", f"-I{CSRC}",
                    "-o", exe, str(tmp_path / "main.cpp")], check=True)
    p = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, p.stdout + p.stderr
