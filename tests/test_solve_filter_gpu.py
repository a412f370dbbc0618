"""The Johnson-Cook solve's FP32 decision (Newton::bisects, neofiz_gb300/csrc/nf_device.cuh)
against the FP64 iteration, on the device with its own approximations: where it decides, the FP64
residual has that sign, is above the tolerance and its Newton step leaves the bracket; and the
solve that uses it gives the plain loop's bits, at a reference rate of 1/s and at others."""
import subprocess

import pytest

from test_ifp import CSRC

CHECK = r"""
#include <cstdio>
#include "nf_device.cuh"
using namespace nf;
struct Rng {                                         // SplitMix64
    uint64_t s;
    __device__ double uniform(double lo, double hi) {
        uint64_t z = (s += 0x9E3779B97F4A7C15ULL);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        return lo + (hi - lo) * (double)((z ^ (z >> 31)) >> 11) * 0x1p-53;
    }
    __device__ double spread(double lo, double hi) { return exp(uniform(log(lo), log(hi))); }
};
__global__ void k_check(int n, unsigned long long *count) {
    Rng r{(blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) * 0xD1B54A32D192ED03ULL};
    unsigned long long decided = 0, wrong = 0, other = 0;
    for (int i = 0; i < n; i++) {
        MatDev jc{};
        jc.a = r.spread(1.0e6, 3.0e9);
        jc.b = r.uniform(0.0, 1.0) < 0.1 ? 0.0 : jc.a * r.spread(1.0e-3, 10.0);
        jc.n = r.uniform(0.0, 1.0) < 0.1 ? 1.0 : r.spread(2.0e-3, 1.0);
        jc.c = r.uniform(0.0, 1.0) < 0.2 ? 0.0 : r.spread(1.0e-4, 1.0);
        jc.refRate = r.uniform(0.0, 1.0) < 0.8 ? 1.0 : r.spread(1.0e-6, 1.0e4);
        const double thermal = r.uniform(0.0, 1.0) < 0.3 ? 1.0 : r.spread(1.0e-4, 1.0);
        const double plastic = r.uniform(0.0, 1.0) < 0.3 ? 0.0 : r.spread(1.0e-14, 5.0);
        const double dt = r.uniform(0.0, 1.0) < 0.02 ? 0.0 : r.spread(1.0e-11, 1.0e-3);
        const double stiffness = jc.a * r.spread(3.0, 1.0e5);
        const double radius = SQRT_2_3 * (jc_strainTerm(jc, plastic) * thermal);
        const double norm = radius * (1.0 + r.spread(1.0e-12, 100.0));
        const double tolerance = SOLVE_TOLERANCE * jc.a;
        const Newton newton(norm, stiffness, plastic, thermal, dt, jc);
        double lo = 0.0, hi = norm / stiffness, dGamma = hi;
        for (int k = 0; k < SOLVE_ITERATIONS; k++) {
            bool up;
            const bool sure = newton.bisects(dGamma, lo, hi, up);
            const NewtonStep s = newton_slow(norm, stiffness, plastic, thermal, dt, jc, dGamma);
            if (s.g > 0.0) lo = dGamma; else hi = dGamma;
            const bool converged = fabs(s.g) <= tolerance;
            double next = dGamma - s.quotient;
            const bool leaves = !(next > lo && next < hi);
            if (sure) {
                decided++;
                if (up != (s.g > 0.0) || converged || !leaves) wrong++;
            }
            if (converged) break;
            dGamma = leaves ? 0.5 * (lo + hi) : next;
        }
        const double solved = j2_solve(norm, stiffness, plastic, thermal, dt, jc).dGamma;
        if (__double_as_longlong(solved) != __double_as_longlong(dGamma)) other++;
    }
    atomicAdd(count, decided);
    atomicAdd(count + 1, wrong);
    atomicAdd(count + 2, other);
}
int main() {
    unsigned long long *d, h[3] = {0, 0, 0};
    if (cudaMalloc(&d, 24) || cudaMemset(d, 0, 24)) return 2;
    k_check<<<608, 128>>>(40, d);
    if (cudaMemcpy(h, d, 24, cudaMemcpyDeviceToHost)) return 2;
    printf("%llu %llu %llu\n", h[0], h[1], h[2]);
    return 0;
}
"""


@pytest.mark.gpu
def test_decisions_and_solves_are_the_fp64_loops(tmp_path):
    from neofiz_gb300 import build
    src, exe = tmp_path / "solve.cu", tmp_path / "solve"
    src.write_text(CHECK)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--fmad=false", "-I", CSRC,
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    decided, wrong, other = map(int, out.stdout.split())
    assert decided > 1000000 and wrong == 0 and other == 0
