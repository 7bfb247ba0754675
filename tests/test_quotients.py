"""The straight-line quotients, roots and logarithms of ctl_devmath.cuh, and what
is built on them (tau_bound, the Poisson samplers), against IEEE division and
square root and the oracle, bit for bit: every FP32 divisor significand, every
waiting-time uniform, and the edges of the ranges in which they may be used.  On
the GPU with its own approximate reciprocals; on the CPU with a reciprocal that
is off by up to 2 ulp (FP32) or 2^-20 (FP64)."""
import os
import shutil
import subprocess

import pytest

import cutauleaping_b200 as ctl
from tests.test_group_tree_cpu import SHIM

CSRC = os.path.join(os.path.dirname(ctl.__file__), "csrc")
ORACLE = os.path.join(os.path.dirname(CSRC), "..", "oracle", "ctl_oracle.c")

MAIN = r'''
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "devmath.h"
extern "C" {
double ctlo_log(double x);
float ctlo_logf(float x);
uint32_t ctlo_poisson(double lam, uint64_t seed, uint32_t sim, uint32_t step, uint32_t attempt, uint32_t r);
}
#ifdef __CUDACC__
#define BOTH __host__ __device__
#else
#define BOTH
#endif
using namespace ctl::dev;
enum { Q32, EDGE32, LOGF, Q64, ROOT, LOG, TAU, POISSON, KINDS };

template <class T, class U> BOTH T as(U v) { T r; memcpy(&r, &v, sizeof r); return r; }
BOTH inline uint64_t mix(uint64_t x) {  // splitmix64
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
BOTH inline float f32(uint32_t sign, int e, uint32_t m) { return as<float>(sign << 31 | (uint32_t)(e + 127) << 23 | (m & 0x7fffffu)); }
BOTH inline double f64(int e, uint64_t m) { return as<double>((uint64_t)(e + 1023) << 52 | (m & 0xfffffffffffffull)); }
// significands at random, and often near their ends
BOTH inline uint32_t sig32(uint64_t h) {
    const uint32_t k = (uint32_t)(h >> 32) & 15u;
    return k < 6u ? k - 3u : k < 8u ? 0x400000u + k : (uint32_t)h;
}
BOTH inline uint64_t sig64(uint64_t h) {
    const uint64_t k = h >> 60;
    return k < 6u ? k - 3u : k < 8u ? (1ull << 51) + k : h;
}

struct In {
    float a, b;
    double x, y;
    uint32_t hor, hort, u[4];
    int32_t n;
    float eps, mu, sg;
};
BOTH inline In make(int kind, uint64_t i) {
    In v = {};
    const uint64_t h = mix(2 * i + 1000003ull * kind), g = mix(h);
    switch (kind) {
    case Q32:  // every significand but the last of a divisor, numerators as in div_fits' promise
        v.b = f32((uint32_t)g >> 31, (int)(g % 120) - 60, (uint32_t)(i % 0x7fffffu));
        v.a = (h & 63u) == 0u ? 0.0f : f32((uint32_t)h >> 31, (int)((h >> 32) % 90) - 30, sig32(mix(g)));
        break;
    case EDGE32: {
        const int e[6] = {-62, -61, -60, 59, 60, 61};
        v.b = f32((uint32_t)h & 1u, e[g % 6], sig32(mix(g)));
        v.a = f32((uint32_t)h >> 1 & 1u, (int)(h >> 32 & 1u) ? (int)(g >> 32 & 3u) - 32 : (int)(g >> 32 & 3u) + 28, sig32(mix(h)));
        if ((h >> 40 & 7u) == 0u) v.a = 0.0f;
        break;
    }
    case LOGF: v.a = ((float)(uint32_t)i + 0.5f) * 0x1p-24f; break;  // u24f
    case Q64: {
        uint64_t m = sig64(g) & 0xfffffffffffffull;
        if (m == 0xfffffffffffffull) m--;
        v.y = f64((int)(h % 160) - 80, m);
        v.x = f64((int)((h >> 32) % 160) - 80, sig64(mix(g)));
        break;
    }
    case ROOT:
        v.x = f64(4 + (int)(h % 36), sig64(g));
        if (h >> 62 == 0) v.x = as<double>(as<uint64_t>((double)(g >> 45) * (double)(g >> 45) + 10.0) + (h >> 32) % 5 - 2);
        break;
    case LOG:
        v.x = f64((int)(h % 2046) - 1022, sig64(g));
        if ((i & 15u) == 0u) v.x = as<double>(g & 0xfffffffffffffull);  // subnormal
        if (i < 4u) v.x = i == 0u ? 0.0 : i == 1u ? INFINITY : i == 2u ? -1.0 : 1.0;
        break;
    case TAU: {
        v.hor = 1u + (uint32_t)(h % 4);
        v.hort = 1u + (uint32_t)(h >> 8) % 3u;
        v.n = (h >> 16 & 3u) == 0u ? (int32_t)(g % 5) : (int32_t)((uint32_t)g >> (1 + (h >> 20) % 31));
        v.eps = (h >> 18 & 1u) ? 0.03f : f32(0u, (int)(h >> 52 & 63u) - 40, (uint32_t)g);
        const uint64_t k = mix(g), l = mix(k);
        v.mu = f32((uint32_t)k & 1u, (int)((k >> 32) % 128) - 64, sig32(l));
        v.sg = f32(0u, (int)((l >> 32) % 128) - 64, sig32(mix(l)));
        if ((k >> 8 & 31u) == 0u) v.mu = 0.0f;
        break;
    }
    case POISSON:
        v.x = (h & 1u) ? f64((int)((h >> 8) % 46) - 4, g) : 100.0 * f64(0, g) - 99.9;
        for (int q = 0; q < 4; q++) v.u[q] = (uint32_t)(mix(g + q) >> 32);
        v.u[3] &= 1023u;
        break;
    }
    return v;
}

__device__ inline uint64_t got(int kind, const In& v) {
    switch (kind) {
    case Q32: return as<uint32_t>(div_near(v.a, v.b)) | (uint64_t)div_fits(v.b) << 32;
    case EDGE32: {
        const bool a_in = v.a == 0.0f || (fabsf(v.a) >= 0x1p-30f && fabsf(v.a) < 0x1p60f);
        return (div_fits(v.b) && a_in ? as<uint32_t>(div_near(v.a, v.b)) : 1u) | (uint64_t)div_fits(v.b) << 32 |
               (uint64_t)num_fits(v.a) << 33;
    }
    case LOGF: return as<uint32_t>(flog(v.a));
    case Q64: return as<uint64_t>(div_near(v.x, v.y));
    case ROOT: return as<uint64_t>(sqrt_near(v.x));
    case LOG: return as<uint64_t>(dlog(v.x));
    case TAU: return as<uint32_t>(tau_bound(v.hor, v.hort, v.n, v.eps, v.mu, v.sg));
    default: {  // as the register-resident sweep draws
        const uint32_t tag = tag_pois(v.u[3], v.u[2] >> 1);
        const uint4 w = draw(0x1234567890ull, 0u, tag, v.u[1], v.u[0]);
        const uint32_t wa = v.u[2] & 1u ? w.z : w.x, wb = v.u[2] & 1u ? w.w : w.y;
        if (v.x < 10.0) return poisson_inversion(v.x, wa);
        uint32_t k;
        const bool quick = poisson_ptrs_quick(v.x, wa, wb, k);
        const uint32_t a = poisson_ptrs_wide(v.x, wa, wb, 0x1234567890ull, tag, v.u[1], v.u[0], v.u[2] & 1u);
        const uint32_t b = poisson_ptrs(v.x, wa, wb, 0x1234567890ull, tag, v.u[1], v.u[0], v.u[2] & 1u);
        return a == b && (!quick || k == a) ? a : 0xdeadbeefcafeull;
    }
    }
}

// The same in IEEE arithmetic on the host.
static float g_of(uint32_t hor, uint32_t hort, float x) {
    if (hor == 2) return hort == 2 ? 2.0f + 1.0f / (x - 1.0f) : 2.0f;
    if (hor == 3) return hort == 3 ? 3.0f + 1.0f / (x - 1.0f) + 2.0f / (x - 2.0f) : hort == 2 ? 3.0f + 1.5f / (x - 1.0f) : 3.0f;
    return 1.0f;
}
static uint64_t want(int kind, const In& v) {
    switch (kind) {
    case Q32: return as<uint32_t>(v.a / v.b) | 1ull << 32;
    case EDGE32: {
        const float b = fabsf(v.b), a = fabsf(v.a);
        const bool db = b >= 0x1p-60f && b < 0x1p60f && (as<uint32_t>(b) & 0x7fffffu) != 0x7fffffu;
        const bool in = v.a == 0.0f || (a >= 0x1p-30f && a < 0x1p60f);
        return (db && in ? as<uint32_t>(v.a / v.b) : 1u) | (uint64_t)db << 32 | (uint64_t)(a == 0.0f || (a >= 0x1p-30f && a < 0x1p30f)) << 33;
    }
    case LOGF: return as<uint32_t>(ctlo_logf(v.a));
    case Q64: return as<uint64_t>(v.x / v.y);
    case ROOT: return as<uint64_t>(sqrt(v.x));
    case LOG: return as<uint64_t>(ctlo_log(v.x));
    case TAU: {
        const float t2 = (v.eps * (float)v.n) / g_of(v.hor, v.hort, (float)v.n), m = t2 > 1.0f ? t2 : 1.0f;
        const float t3 = v.mu != 0.0f ? m / fabsf(v.mu) : INFINITY, t4 = (m * m) / v.sg;
        return as<uint32_t>(t3 < t4 ? t3 : t4);
    }
    default: return ctlo_poisson(v.x, 0x1234567890ull, v.u[0], v.u[1], v.u[3], v.u[2]);
    }
}
static uint64_t count(int kind, int log_n) { return kind == Q32 ? 0x7fffffu : 1ull << (kind == LOGF ? 24 : log_n); }

#ifdef __CUDACC__
__global__ void run(int kind, uint64_t n, uint64_t* out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = got(kind, make(kind, i));
}
#endif
int main(int, char** argv) {
    const int log_n = atoi(argv[1]);
    int bad_kinds = 0;
    for (int kind = 0; kind < KINDS; kind++) {
        const uint64_t n = count(kind, log_n);
        std::vector<uint64_t> out(n);
#ifdef __CUDACC__
        uint64_t* d = nullptr;
        if (cudaMalloc(&d, n * 8) != cudaSuccess) return 2;
        run<<<592, 256>>>(kind, n, d);
        if (cudaMemcpy(out.data(), d, n * 8, cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
        cudaFree(d);
#else
        for (uint64_t i = 0; i < n; i++) {
            off = (int)(i % 5) - 2;
            out[i] = got(kind, make(kind, i));
        }
#endif
        uint64_t bad = 0;
        for (uint64_t i = 0; i < n; i++) {
            const In v = make(kind, i);
            if (out[i] != want(kind, v) && bad++ == 0)
                printf("kind %d, input %llu: %llx, not %llx\n", kind, (unsigned long long)i, (unsigned long long)out[i],
                       (unsigned long long)want(kind, v));
        }
        printf("kind %d: %llu of %llu differ\n", kind, (unsigned long long)bad, (unsigned long long)n);
        bad_kinds += bad != 0;
    }
    return bad_kinds != 0;
}
'''


def _oracle(tmp_path):
    obj = str(tmp_path / "oracle.o")
    subprocess.run(["gcc", "-O2", "-std=c11", "-ffp-contract=off", "-c", "-o", obj, ORACLE], check=True)
    return obj


def test_on_the_cpu_from_perturbed_reciprocals(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ is not installed")
    start = r'''
inline int off;
inline float approx(float v) { return bits<float>(bits<int>(v) + off); }
inline double approx(double v) { return v * (1.0 + off * 0x1p-21); }
'''
    (tmp_path / "cuda_runtime.h").write_text(SHIM + start)
    (tmp_path / "ctl.h").write_text(open(os.path.join(CSRC, "..", "..", "include", "ctl.h")).read())
    text = open(os.path.join(CSRC, "ctl_devmath.cuh")).read().replace("rsqrt.approx.ftz.f64 %0, %1;\" : \"=d\"(y) : \"d\"(x)", "ROOT")
    text = text.replace('asm("ROOT);', "y = approx(1.0 / sqrt(x));")
    for b, t in (("b", "f"), ("b", "d")):
        bits = "f32" if t == "f" else "f64"
        text = text.replace(f'asm("rcp.approx.ftz.{bits} %0, %1;" : "={t}"(y) : "{t}"({b}));', f"y = approx(1 / {b});")
    assert "asm" not in text
    (tmp_path / "devmath.h").write_text(text.replace('"../../include/ctl.h"', '"ctl.h"'))
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-w", f"-I{tmp_path}", "-o", exe,
                    str(tmp_path / "main.cpp"), _oracle(tmp_path), "-lm", "-lpthread"], check=True)
    p = subprocess.run([exe, "20"], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr


@pytest.mark.gpu
def test_on_the_gpu(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    (tmp_path / "devmath.h").write_text(f'#include "{os.path.join(CSRC, "ctl_devmath.cuh")}"\n')
    (tmp_path / "main.cu").write_text(MAIN)
    exe = str(tmp_path / "check")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "-fmad=false",
                    "-Xcompiler", "-ffp-contract=off", f"-I{tmp_path}", "-o", exe, str(tmp_path / "main.cu"),
                    _oracle(tmp_path)], check=True)
    p = subprocess.run([exe, "23"], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr
