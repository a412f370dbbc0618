"""The integer division, square root and product of the FP64 kernels (neofiz_gb300/csrc/nf_ifp.h)
against the machine's, and the logarithm and power that use integer arithmetic (nf_ilog.h)
against nf_math.h's, bit for bit.

One check compiles from the header for the host, where the FP32 approximation the methods start
from is moved through its whole documented error range (and past it), and for the device, where
it is the real one. Operands are random significands and the patterns where a digit, a
remainder or the rounding can go wrong: powers of two, all ones, a few bits at either end,
exact quotients and squares, their neighbours, every exponent, zeros, subnormals, infinities
and NaN.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "neofiz_gb300", "csrc")

CHECK = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include "nf_ilog.h"
#ifdef __CUDACC__
#define FN static __host__ __device__
#else
#define FN static
#endif
FN double dval(uint64_t u) { double d; memcpy(&d, &u, 8); return d; }
FN uint64_t dbits(double d) { uint64_t u; memcpy(&u, &d, 8); return u; }
FN bool same(double a, double b) { return dbits(a) == dbits(b) || (a != a && b != b); }
struct Rng {                                         // SplitMix64
    uint64_t s;
    FN uint64_t mix(uint64_t z) {
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        return z ^ (z >> 31);
    }
#ifdef __CUDACC__
    __host__ __device__
#endif
    uint64_t next() { s += 0x9E3779B97F4A7C15ULL; return mix(s); }
};
FN uint64_t significand(Rng &r) {
    const uint64_t m = r.next() & 0xfffffffffffffULL;
    switch (r.next() & 7) {
    case 0: return 0;
    case 1: return 0xfffffffffffffULL;
    case 2: return m & 0xff;
    case 3: return m | 0xffffffffff000ULL;
    case 4: return m & ~0xffffffULL;
    case 5: return 1ULL << (r.next() % 52);
    default: return m;
    }
}
FN double number(Rng &r) {
    const uint64_t sign = r.next() & (1ULL << 63);
    switch (r.next() & 15) {
    case 0: return dval(r.next());                   // any bits at all
    case 1: return dval(sign);                       // a zero
    case 2: return dval(sign | ((r.next() % 2047) << 52) | significand(r));
    default: return dval(sign | ((1023 - 40 + r.next() % 80) << 52) | significand(r));
    }
}
// bad logarithms in the low word, bad powers in the high word
FN uint64_t check_log(uint64_t seed, int n) {
    Rng r{seed};
    uint64_t bad = 0;
    for (int i = 0; i < n; i++) {
        double x;
        switch (r.next() & 15) {
        case 0: x = number(r); break;
        case 1: x = 1.0 + (double)(int64_t)r.next() * 0x1p-70; break;    // near log 1 = 0
        // a table interval's end, and its neighbours
        case 2: x = dval(NF_LOG_OFF + ((r.next() % 128) << 45) + (r.next() % 5) - 2); break;
        // the ends of the fixed-point sum's range
        case 3: x = dval((r.next() & 1 ? 0x3bf0000000000000ULL : 0x43f0000000000000ULL)
                         + (r.next() % 5) - 2); break;
        default: x = dval(((1023 - 66 + r.next() % 132) << 52) | significand(r));
        }
        if (!same(nf_log_fast(x), nf_log(x))) bad++;
        double y = (double)(r.next() >> 11) * 0x1p-53;
        switch (r.next() & 7) {
        case 0: y = number(r); break;
        case 1: y = 1.0; break;
        case 2: y = dval(((1013 + r.next() % 13) << 52) | significand(r)); break;
        case 3: y = 1.0 + 0.2 * y; break;
        }
        if (!same(nf_pow_fast(x, y), nf_pow(x, y))) bad += 1ULL << 32;
    }
    return bad;
}
// bad divisions in the low word, bad roots in the high word
FN uint64_t check(uint64_t seed, int n) {
    Rng r{seed};
    uint64_t bad = 0;
    for (int i = 0; i < n; i++) {
        double a = number(r);
        const double b = number(r);
        switch (r.next() & 7) {
        case 0: a = b * (double)(r.next() & 0xffff); break;          // exact or near it
        case 1: a = dval(dbits(b * (double)(r.next() & 0xffff)) + (r.next() % 3) - 1); break;
        }
        const nf_divisor v = nf_divisor_of(b);
        if (!same(nf_div(a, b), a / b) || !same(nf_div_by(b, b, v), b / b)) bad++;
        double x = fabs(number(r));
        switch (r.next() & 7) {
        case 0: x = dval(dbits(x) & ~0x7ffffffULL); x = x * x; break;  // squares, neighbours
        case 1: x = dval(dbits(x) & ~0x7ffffffULL); x = dval(dbits(x * x) + (r.next() % 3) - 1); break;
        case 2: x = -x; break;
        }
        if (!same(nf_sqrt(x), sqrt(x))) bad += 1ULL << 32;
        // products and scalings: the machine's bits, or refused; the path's range is not refused
        uint32_t no = 0;
        const double p = nf_mul_try(a, b, &no);
        const bool near1 = fabs(a) > 0x1p-200 && fabs(a) < 0x1p200 && fabs(b) > 0x1p-200 && fabs(b) < 0x1p200;
        if (no ? near1 : !same(p, a * b)) bad++;
        no = 0;
        const int k = (int)(r.next() % 17) - 8;
        const double q = nf_scale_try(a, k, &no);
        if (no ? near1 : !same(q, a * dval((uint64_t)(1023 + k) << 52))) bad++;
    }
    return bad;
}
#ifdef __CUDACC__
__global__ void k_check(uint64_t seed, int n, unsigned long long *bad) {
    const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t at = seed + t * 0xD1B54A32D192ED03ULL;
    const uint64_t b = check(at, n) + check_log(at, n);
    if (b) atomicAdd(bad, (unsigned long long)b);
}
int main() {
    unsigned long long *d, h = 0;
    if (cudaMalloc(&d, 8) || cudaMemset(d, 0, 8)) return 2;
    k_check<<<608, 256>>>(20251206, 1000, d);
    if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost)) return 2;
    printf("bad %llu\n", h);
    return h != 0;
}
#else
int main() {
    uint64_t bad = 0;
    for (nf_ifp_off = -2; nf_ifp_off <= 2; nf_ifp_off++) bad += check(7 + nf_ifp_off, 6000000);
    bad += check_log(11, 6000000);
    // the integer forms are what ran: few of the path's arguments take nf_math.h's sequence
    nf_ilog_slow_count = 0;
    Rng r{5};
    for (int i = 0; i < 1000000; i++) {
        const double x = dval(((1003 + r.next() % 40) << 52) | (r.next() & 0xfffffffffffffULL));
        if (fabs(nf_log(x)) < 0.004) continue;
        nf_log_fast(x);
        nf_pow_fast(x, 0.1 + 1.0 * (double)(r.next() >> 11) * 0x1p-53);
    }
    if (nf_ilog_slow_count > 4000) bad++;
    printf("bad %llu\n", (unsigned long long)bad);
    return bad != 0;
}
#endif
"""


def _run(tmp_path, name, command):
    src = tmp_path / name
    src.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run([*command, "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.split() == ["bad", "0"], out.stdout + out.stderr


def test_host_results_are_correctly_rounded(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    _run(tmp_path, "check.cpp", [cxx, "-O2", "-ffp-contract=off"])


@pytest.mark.gpu
def test_device_results_are_correctly_rounded(tmp_path):
    from neofiz_gb300 import build
    _run(tmp_path, "check.cu", [build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false"])
