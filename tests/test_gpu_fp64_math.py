"""The FP64 sum's own reciprocal, reciprocal square root and e^{ix} (abt_b200/csrc/k1_math.cuh)
against 80-bit arithmetic on the host, and CUDA's functions beside them, over the ranges of the sum:
phases up to 2^30 rad across the table's cells and their edges, products of phase steps of either
sign, squared distances and squared norms.

Bounds, u = 2^-53: rcp_n rounds once (its series leaves 2^-58): 1.1 u.  rsqrt_n rounds x y and
the result, half of the first: 1.6 u.  e^{ix}: the table's entries 2 units in the last place of
CUDA's sincospi, at most 2 u each, two roundings of at most u / 2 each, s, c and r below
u / 2 together: 4 u absolute.  With a phase split off (reduce_n) the sum r + d rounds once more:
u |r + d| / 2 beside it, taken as u |r + d|.  CUDA's functions are held to their documented
units in the last place (1/x 0.5, rsqrt 1, sin and cos 2), as a check of the measure."""
import os
import subprocess

import pytest

from abt_b200 import build
from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <random>
#include <vector>
#include "k1_math.cuh"
using namespace pbt;
// in: x[n] and d[n]; out: 10 values a point
__global__ void points(const double *x, const double *d, int n, double *out) {
    __shared__ double2 root[kRoots];
    if (threadIdx.x < kRoots) sincospi(threadIdx.x * (2.0 / kRoots), &root[threadIdx.x].y, &root[threadIdx.x].x);
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double *o = out + 10 * (size_t)i, s, c;
    o[0] = rcp_n(x[i]);
    o[1] = 1.0 / x[i];
    o[2] = rsqrt_n(fabs(x[i]));
    o[3] = rsqrt(fabs(x[i]));
    sincos_n(x[i], 0, root, &s, &c);
    o[4] = s;
    o[5] = c;
    sincos(x[i], &s, &c);
    o[6] = s;
    o[7] = c;
    int nk;
    const double r = reduce_n(x[i], &nk);
    sincos_n(r + d[i], nk, root, &s, &c);
    o[8] = s;
    o[9] = c;
}
static std::vector<double> run(const std::vector<double> &x, const std::vector<double> &d) {
    const int n = (int)x.size();
    double *dx, *dd, *dout;
    std::vector<double> out(10 * x.size());
    if (cudaMalloc(&dx, n * 8) || cudaMalloc(&dd, n * 8) || cudaMalloc(&dout, out.size() * 8)) exit(2);
    cudaMemcpy(dx, x.data(), n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(dd, d.data(), n * 8, cudaMemcpyHostToDevice);
    points<<<(n + 255) / 256, 256>>>(dx, dd, n, dout);
    if (cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost) || cudaDeviceSynchronize()) exit(2);
    cudaFree(dx);
    cudaFree(dd);
    cudaFree(dout);
    return out;
}
int main() {
    const long double u = ldexpl(1.0L, -53), h = 8.0L * atanl(1.0L) / 128.0L;
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> U(0.0, 1.0);
    const int n = 1 << 20;
    long double e[8] = {};
    auto worse = [&](int k, long double v) {
        if (!(v <= e[k])) e[k] = v;  // a NaN too
    };
    // reciprocals: magnitudes over the sum's range and beyond it
    std::vector<double> x(n), d(n, 0.0);
    for (int i = 0; i < n; i++) {
        const double m = 1.0 + U(g);
        x[i] = ldexp(i % 64 == 0 ? 1.0 : m, (int)(U(g) * 400.0) - 200) * (i & 1 ? -1.0 : 1.0);
    }
    std::vector<double> o = run(x, d);
    for (int i = 0; i < n; i++) {
        const long double a = x[i], q = sqrtl(fabsl(a));
        worse(0, fabsl(o[10 * i] * a - 1.0L) / u);
        worse(1, fabsl(o[10 * i + 1] * a - 1.0L) / u);
        worse(2, fabsl(o[10 * i + 2] * q - 1.0L) / u);
        worse(3, fabsl(o[10 * i + 3] * q - 1.0L) / u);
    }
    // phases: all magnitudes up to 2^30, the far-field range, cells' edges and middles, zero
    for (int i = 0; i < n; i++) {
        const double s = i & 1 ? -1.0 : 1.0;
        if (i % 4 == 0) x[i] = s * ldexp(1.0 + U(g), (int)(U(g) * 45.0) - 16);
        else if (i % 4 == 1) x[i] = s * (1.18e7 + 200.0 * U(g));
        else if (i % 4 == 2) x[i] = s * (double)((floorl(U(g) * 4096.0L) + 0.5L * (i / 4 % 2)) * h);
        else x[i] = s * 1073741823.0 * U(g);
        d[i] = (U(g) - 0.5) * 200.0;
    }
    x[0] = 0.0;
    o = run(x, d);
    for (int i = 0; i < n; i++) {
        const long double a = x[i];
        worse(4, fmaxl(fabsl(o[10 * i + 4] - sinl(a)), fabsl(o[10 * i + 5] - cosl(a))) / u);
        worse(5, fmaxl(fabsl(o[10 * i + 6] - sinl(a)), fabsl(o[10 * i + 7] - cosl(a))) / u);
        // e^{i (x + d)} from x's fraction: 80 bits hold x + d to 2^-34 at 2^30, so sum the angles
        const long double sx = sinl(a), cx = cosl(a), sd = sinl((long double)d[i]), cd = cosl((long double)d[i]);
        const long double s = sx * cd + cx * sd, c = cx * cd - sx * sd;
        worse(6, fmaxl(fabsl(o[10 * i + 8] - s), fabsl(o[10 * i + 9] - c)) / u - fabsl((long double)d[i]) - 0.03L);
    }
    printf("rcp %.3Lf\ncuda_rcp %.3Lf\nrsqrt %.3Lf\ncuda_rsqrt %.3Lf\nexp %.3Lf\ncuda_exp %.3Lf\nsplit %.3Lf\n", e[0],
           e[1], e[2], e[3], e[4], e[5], e[6]);
}
"""


def test_against_80_bits_and_cuda(tmp_path):
    (tmp_path / "t.cu").write_text(SOURCE)
    subprocess.run([build.NVCC, *build.ARCH, "-O3", "-std=c++17", "-fmad=false",
                    "-I" + os.path.join(ROOT, "abt_b200", "csrc"), str(tmp_path / "t.cu"), "-o", str(tmp_path / "t")],
                   check=True, capture_output=True)
    r = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=300, check=True)
    got = {k: float(v) for k, v in (line.split() for line in r.stdout.splitlines())}
    print(got)
    for name, bound in (("cuda_rcp", 1.0), ("cuda_rsqrt", 2.0), ("cuda_exp", 4.0),
                        ("rcp", 1.1), ("rsqrt", 1.6), ("exp", 4.0), ("split", 4.0)):
        assert got[name] <= bound, (name, got)
