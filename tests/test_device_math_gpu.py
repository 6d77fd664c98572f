"""The kernels' own FP64 reciprocal, fifth root, 1/r^3 and float-float split against CUDA's
division, pow, sqrt and conversions, over random arguments and the edges of their ranges."""
import os
import subprocess

import pytest

from simbuca_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include <cmath>
#include <random>
#include <vector>
#include "dp_stage.cuh"
#include "fp32c_math.cuh"
__global__ void eval(const double* x, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    float h, l;
    split_double(v, h, l);
    out[i] = fabs(stage_rcp(v) - 1.0 / v) * v;
    out[n + i] = fabs(sg_inv_fifth_root(v) - pow(v, -0.2)) / pow(v, -0.2);
    const double r3 = 1.0 / (v * sqrt(v));
    out[2 * n + i] = fabs(inv_r3_fp64(v) - r3) / r3;
    // the conversions' own pair: h rounds v, l the rest; ties may go the other way
    const float hc = __double2float_rn(v), lc = __double2float_rn(v - (double)hc);
    out[3 * n + i] = (h == hc && l == lc) || (double)h + l == (double)hc + lc
                         ? 0.0 : fabs(((double)h + l) - v) / fabs(v);
    split_double(-v, h, l);
    out[4 * n + i] = fabs(((double)h + l) + v) / fabs(v);
}
__global__ void edges(double* out) {
    out[0] = stage_rcp(INFINITY);
    out[1] = stage_rcp(NAN);
    out[2] = stage_rcp(0.0);
    float h, l;
    split_double(0.0, h, l);
    out[3] = (double)h + l;
    split_double(INFINITY, h, l);
    out[4] = h;
    split_double(NAN, h, l);
    out[5] = h;
}
int main() {
    const int n = 1 << 20;
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> e(%LO%, %HI%);
    std::vector<double> x(n), o(5 * (size_t)n);
    for (double& v : x) v = std::pow(10.0, e(g));
    double *dx, *dout;
    if (cudaMalloc(&dx, n * 8) != cudaSuccess || cudaMalloc(&dout, 5 * (size_t)n * 8) != cudaSuccess) return 1;
    cudaMemcpy(dx, x.data(), n * 8, cudaMemcpyHostToDevice);
    eval<<<n / 256, 256>>>(dx, dout, n);
    cudaMemcpy(o.data(), dout, 5 * (size_t)n * 8, cudaMemcpyDeviceToHost);
    for (int f = 0; f < 5; f++) {
        double m = 0.0;
        for (int i = 0; i < n; i++) m = !(o[(size_t)f * n + i] <= m) ? o[(size_t)f * n + i] : m;
        printf("%.3e ", m);
    }
    edges<<<1, 1>>>(dout);
    cudaMemcpy(o.data(), dout, 6 * 8, cudaMemcpyDeviceToHost);
    for (int f = 0; f < 6; f++) printf("%g ", o[f]);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 1;
}
"""


@pytest.mark.parametrize("lo,hi", [(-2.0, 2.0), (-29.0, 29.0), (-150.0, -31.0), (31.0, 150.0)])
def test_against_cuda(tmp_path, lo, hi):
    """In units of 2^-53: the reciprocal is one rounding and 2^-57 from exact, CUDA's division one
    rounding: 3e-16 apart.  The fifth root ends in one rounding after four of a fifth's weight,
    pow is good to 2 ulp: 7e-16.  1/r^3 carries 2.7 roundings, division and sqrt 4: 8e-16.  The
    split leaves out what its low part rounds, 2^-48 (outside the float range, where there is
    none, it is the conversions themselves)."""
    src = tmp_path / "math.cu"
    src.write_text(SOURCE.replace("%LO%", str(lo)).replace("%HI%", str(hi)))
    exe = tmp_path / "math"
    subprocess.run([build.nvcc()] + build.ARCH + ["-O3", "-std=c++17", "-I", build.CSRC, str(src), "-o", str(exe)],
                   check=True)
    out = [float(v) for v in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]
    print(out)
    rcp, root, r3, split, negative = out[:5]
    assert rcp <= 3e-16
    assert root <= 7e-16
    if hi < 100.0 and lo > -100.0:  # 1/r^3 of the others is outside the range of a double or near it
        assert r3 <= 8e-16
        if -29.0 < lo and hi < 29.0:
            assert split <= 2.0 ** -48 and negative <= 2.0 ** -48
    assert out[5] == 0.0 and out[6] != out[6]
    assert out[8] == 0.0 and out[9] == float("inf") and out[10] != out[10]
