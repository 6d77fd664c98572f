// aux_kernels.cu -- the CUNBODY-compatible force kernel and the issue-rate probes.
#include <stdint.h>

#include <algorithm>

#include "fp64_pairs.cuh"
#include "sg_internal.cuh"

namespace {

// ai[i] = sum_j mj[j] (xj[j] - xi[i]) / (|xj[j]-xi[i]|^2 + eps2)^{3/2}
// (the CUNBODY contract, bin/cunbody.h:11-33), FP64.

// Two different sets: ordered pairs, 128 i-rows a block against one of the j-chunks, which
// go to a partial-sum slot each ([chunk][3][ni], sums of xi - xj).  FP64-bound (16
// instructions a pair, 64 cycles each): the j-chunks give every SM several blocks, where a
// block per 128 rows alone left half of them idle (10,007 x 10,007: 7,535 us).  A single
// chunk's sums go straight to ai (null otherwise): one launch for up to 128 j-ions.
constexpr int kCbThreads = 128;
__global__ void __launch_bounds__(kCbThreads) cunbody_kernel(const double* __restrict__ xj,
                                                             const double* __restrict__ mj,
                                                             const double* __restrict__ xi,
                                                             double eps2, double* __restrict__ part,
                                                             int ni, int nj, int jc,
                                                             double* __restrict__ ai) {
    sg_griddep_wait();
    __shared__ double t[4][kCbThreads];
    const int i = blockIdx.x * kCbThreads + threadIdx.x;
    const bool act = i < ni;
    const double x = act ? xi[3 * (size_t)i] : 0.0, y = act ? xi[3 * (size_t)i + 1] : 0.0,
                 z = act ? xi[3 * (size_t)i + 2] : 0.0;
    double ax = 0.0, ay = 0.0, az = 0.0;
    const int je = min(nj, (int)(blockIdx.y + 1) * jc);
    for (int j0 = blockIdx.y * jc; j0 < je; j0 += kCbThreads) {
        const int len = min(kCbThreads, je - j0);
        __syncthreads();
        if ((int)threadIdx.x < len) {
            const size_t j = (size_t)(j0 + threadIdx.x);
            t[0][threadIdx.x] = xj[3 * j];
            t[1][threadIdx.x] = xj[3 * j + 1];
            t[2][threadIdx.x] = xj[3 * j + 2];
            t[3][threadIdx.x] = mj[j];
        }
        __syncthreads();
        // whole warps of absent rows (the last block) have nothing to add up
        if (i - (int)(threadIdx.x & 31) < ni)
            for (int jj = 0; jj < len; jj++) {
                const double dx = x - t[0][jj], dy = y - t[1][jj], dz = z - t[2][jj];
                const double r2 = fma(dz, dz, fma(dy, dy, fma(dx, dx, eps2)));
                // a coincident pair without softening contributes nothing (0 * inf avoided)
                double w = t[3][jj] * inv_r3_fp64(r2);
                if (!(r2 > 0.0)) w = 0.0;
                ax = fma(w, dx, ax);
                ay = fma(w, dy, ay);
                az = fma(w, dz, az);
            }
    }
    if (act && ai != nullptr) {
        ai[3 * (size_t)i] = -ax;
        ai[3 * (size_t)i + 1] = -ay;
        ai[3 * (size_t)i + 2] = -az;
    } else if (act) {
        double* P = part + (size_t)blockIdx.y * 3 * ni;
        P[i] = ax;
        P[ni + i] = ay;
        P[2 * (size_t)ni + i] = az;
    }
}

// One set against itself (the reference's wrapper passes one array as both,
// bin/cunbody.cpp:43-90): each unordered pair once (fp64_pairs.cuh), 9 instructions per
// ordered pair.
struct CbLoad {
    const double *x, *m;
    int n;
    __device__ __forceinline__ double operator()(int a, int k) const {
        if (k < n) return a < 3 ? x[3 * (size_t)k + a] : m[k];
        return a < 3 ? 1.0e3 + 1.0e-3 * k : 0.0;
    }
};

// Issue-rate probes: every thread runs 8 independent FMA chains (4 packed pairs) of
// `iters` steps; the result is stored so the chains are not eliminated.
constexpr int kProbeIters = 4096;

__global__ void probe_ffma(float* sink, float a, float b) {
    sg_griddep_wait();
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = threadIdx.x * 1e-3f + q;
#pragma unroll 16
    for (int it = 0; it < kProbeIters; it++)
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = __fmaf_rn(v[q], a, b);
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) s += v[q];
    if (s == 1.2345f) sink[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

__global__ void probe_ffma2(float* sink, float a, float b) {
    sg_griddep_wait();
    unsigned long long v[4], A, B;
    asm("mov.b64 %0, {%1, %1};" : "=l"(A) : "f"(a));
    asm("mov.b64 %0, {%1, %1};" : "=l"(B) : "f"(b));
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const float lo = threadIdx.x * 1e-3f + q, hi = lo + 0.5f;
        asm("mov.b64 %0, {%1, %2};" : "=l"(v[q]) : "f"(lo), "f"(hi));
    }
#pragma unroll 16
    for (int it = 0; it < kProbeIters; it++)
#pragma unroll
        for (int q = 0; q < 4; q++)
            asm volatile("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(v[q]) : "l"(A), "l"(B));
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        float lo, hi;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v[q]));
        s += lo + hi;
    }
    if (s == 1.2345f) sink[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

__global__ void probe_dfma(float* sink, double a, double b) {
    sg_griddep_wait();
    double v[8];
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = threadIdx.x * 1e-3 + q;
    // FP64 issue is far slower: fewer steps keep the probe short
#pragma unroll 8
    for (int it = 0; it < kProbeIters / 16; it++)
#pragma unroll
        for (int q = 0; q < 8; q++) v[q] = fma(v[q], a, b);
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < 8; q++) s += v[q];
    if (s == 1.2345) sink[blockIdx.x * blockDim.x + threadIdx.x] = (float)s;
}

}  // namespace

static int cb_chunks(int ni, int nj, int n_sm, int* jc) {
    const int ib = (ni + kCbThreads - 1) / kCbThreads;
    int chunks = std::max(1, std::min((nj + kCbThreads - 1) / kCbThreads, 8 * n_sm / ib));
    *jc = ((nj + chunks - 1) / chunks + kCbThreads - 1) / kCbThreads * kCbThreads;
    *jc = std::max(*jc, kCbThreads);
    return std::max(1, (nj + *jc - 1) / *jc);
}

size_t sg_cunbody_scratch(int ni, int nj, int same, int n_sm) {
    if (same) {
        const int npad = (ni + SG_PAD - 1) / SG_PAD * SG_PAD;
        return (size_t)sym_plan(npad, n_sm, SIZE_MAX).slots * 3 * npad;
    }
    int jc = 0;
    return (size_t)cb_chunks(ni, nj, n_sm, &jc) * 3 * ni;
}

cudaError_t sg_cunbody_launch(const double* xj, const double* mj, const double* xi, double eps2,
                              double* ai, int ni, int nj, int same, int uniform, double m0,
                              double* part, int n_sm, cudaStream_t st) {
    if (ni <= 0) return cudaSuccess;
    SymPlan p;
    int stride = ni;
    if (same) {
        stride = (ni + SG_PAD - 1) / SG_PAD * SG_PAD;
        p = sym_plan(stride, n_sm, SIZE_MAX);
        sg_launch(sym_set_kernel<true, CbLoad>, p.items, SG_SYM_IB, 0, st, CbLoad{xj, mj, ni}, ni,
                  stride, p, uniform != 0, m0, eps2, part);
    } else {
        int jc = 0;
        p = SymPlan{0, 1, 0, cb_chunks(ni, nj, n_sm, &jc)};
        sg_launch(cunbody_kernel, dim3((ni + kCbThreads - 1) / kCbThreads, p.slots), kCbThreads, 0,
                  st, xj, mj, xi, eps2, part, ni, nj, jc, p.slots == 1 ? ai : nullptr);
        if (p.slots == 1) return cudaGetLastError();
    }
    sg_launch(sym_sum_kernel<16>, (ni + 15) / 16, 256, 0, st, (const double*)part, ni, stride, p,
              (const double*)nullptr, -1.0, ai);
    return cudaGetLastError();
}

// which: 0 FFMA, 1 FFMA2 (packed), 2 DFMA.  Returns flops per launch via the caller:
// 2 * 8 * iters * blocks * threads (FP32 / FP32x2), iters/16 for FP64.
cudaError_t sg_probe_launch(int which, int blocks, int threads, float* sink, cudaStream_t st) {
    switch (which) {
        case 0: sg_launch(probe_ffma, blocks, threads, 0, st, sink, 0.999f, 1e-4f); break;
        case 1: sg_launch(probe_ffma2, blocks, threads, 0, st, sink, 0.999f, 1e-4f); break;
        case 2: sg_launch(probe_dfma, blocks, threads, 0, st, sink, 0.999, 1e-4); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

int sg_probe_iters(int which) { return which == 2 ? kProbeIters / 16 : kProbeIters; }
