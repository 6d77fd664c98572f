// dp_stage.cuh -- one component of one ion at one stage of the embedded Runge-Kutta pairs,
// shared by the tiled stage kernels (dp45.cu, finish.cu) and the fused small-cloud kernel
// (fused.cu).
#pragma once

#include "dp_tableau.cuh"
#include "sg_internal.cuh"

namespace {

typedef SgDpArgs DpArgs;

// u as float-float: h = u rounded to 24 bits (ties away from zero), l = the rest rounded.
// By integers: a conversion between FP64 and FP32 takes a warp 64 cycles, like any FP64
// instruction, and the three here with the difference were 4 of the ~30 a component of a
// stage takes; the integer path is 10 instructions of 1 to 8 cycles.
__device__ __forceinline__ void split_double(double u, float& h, float& l) {
    const long long b = __double_as_longlong(u);
    const int e = (int)((unsigned long long)b >> 52) & 0x7ff;
    if (e >= 1023 - 70 && e <= 1023 + 100) {
        // the fraction's low 29 bits, as a signed distance from the nearest multiple of 2^29
        const long long r = b + 0x10000000ll;  // a carry into the exponent is the rounded value
        const int d = (int)(b & 0x1fffffffll) - ((b & 0x10000000ll) ? 0x20000000 : 0);
        const unsigned top = (unsigned)((unsigned long long)r >> 32);
        // sign, exponent rebased by 1023 - 127, 23 fraction bits
        const unsigned hb = (top & 0x80000000u) |
                            ((((top & 0x7fffffffu) << 3) | (unsigned)((unsigned long long)r >> 29 & 7)) -
                             ((1023u - 127u) << 23));
        h = __uint_as_float(hb);
        // d units of 2^(e - 1075), with u's sign
        const float s = __uint_as_float((unsigned)(e - 1075 + 127) << 23 | (top & 0x80000000u));
        l = __fmul_rn(__int2float_rn(d), s);
    } else {  // zero, tiny, huge or not finite
        h = __double2float_rn(u);
        l = __double2float_rn(u - (double)h);
    }
}

// Frame coordinate of one component: high part and remainder.
__device__ __forceinline__ float write_coord(const DpArgs& a, const SgCloud& cl, int c, int ig,
                                             double x) {
    const size_t NP = (size_t)a.npad;
    a.c64[c * NP + ig] = x;
    if (!a.fp32c) return 0.f;
    const double u = (x - (c == 0 ? cl.cx : c == 1 ? cl.cy : cl.cz)) * cl.invL;
    float h, l;
    split_double(u, h, l);
    a.c32[c * NP + ig] = h;
    a.c32[(4 + c) * NP + ig] = l;
    return h;
}

// Tableaus of the two embedded pairs: stage s = 1..stages of M::a, M::c, M::e.
struct MethodDP {
    static constexpr int stages = 7;
    static __device__ __forceinline__ double a(int s, int j) { return c_a[s][j]; }
    static __device__ __forceinline__ double c(int s) { return c_c[s]; }
    static __device__ __forceinline__ double e(int j) { return c_e[j]; }
};

// ---- Cash-Karp 5(4), the reference's "RungaKutta4" (bin/ode.cpp:220-345) ----------
__constant__ double c_ck_a[7][6] = {
    {0, 0, 0, 0, 0, 0},
    {0, 0, 0, 0, 0, 0},
    {0.2, 0, 0, 0, 0, 0},
    {3.0 / 40.0, 9.0 / 40.0, 0, 0, 0, 0},
    {0.3, -0.9, 1.2, 0, 0, 0},
    {-11.0 / 54.0, 2.5, -70.0 / 27.0, 35.0 / 27.0, 0, 0},
    {1631.0 / 55296.0, 175.0 / 512.0, 575.0 / 13824.0, 44275.0 / 110592.0, 253.0 / 4096.0, 0}};
__constant__ double c_ck_c[8] = {0, 0.0, 0.2, 0.3, 0.6, 1.0, 0.875, 0.0};
__constant__ double c_ck_b[7] = {0, 37.0 / 378.0, 0.0, 250.0 / 621.0, 125.0 / 594.0, 0.0,
                                 512.0 / 1771.0};
__constant__ double c_ck_e[7] = {0,
                                 37.0 / 378.0 - 2825.0 / 27648.0,
                                 0.0,
                                 250.0 / 621.0 - 18575.0 / 48384.0,
                                 125.0 / 594.0 - 13525.0 / 55296.0,
                                 -277.00 / 14336.0,
                                 512.0 / 1771.0 - 0.25};
struct MethodCK {
    static constexpr int stages = 6;
    static __device__ __forceinline__ double a(int s, int j) { return c_ck_a[s][j]; }
    static __device__ __forceinline__ double c(int s) { return c_ck_c[s]; }
    static __device__ __forceinline__ double e(int j) { return c_ck_e[j]; }
};

// 1/x from the SFU's FP64 reciprocal (rcp.approx.ftz.f64, ~2^-20) and the geometric series
// 1/(x y0) = 1 + e + e^2 + ..., e = 1 - x y0: 3 FP64 instructions where the IEEE division's
// sequence takes ~14, 64 cycles each, for every component of every ion.  |e|^3 < 2^-57: the
// result is within an ulp or so, far inside the error norm's own conditioning (~1e-8).  An
// infinite x (a tolerance that accepts everything) has the reciprocal 0, not the series' NaN.
__device__ __forceinline__ double stage_rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return __double2hiint(y) == 0 ? y : fma(y, fma(e, e, e), y);
}

// Component c of ion i at stage S: finishes its force (P: the Coulomb sum along the axis
// of an acceleration component), stores k_S, and builds stage S+1's state (returned), or
// for the last stage the squared scaled error (bin/ode.cpp:101-205, 220-345) with the
// Cash-Karp solution in sol.  The other components of the ion read this stage's state from
// ys: the caller stores the new one after a block barrier.
template <int S, class M>
__device__ __forceinline__ double stage_one(const DpArgs& a, const SgCloud& cl, const SgCtrl& cs,
                                            const SgFieldCoef& fk, int c, int i, double P,
                                            double& sol) {
    const size_t N = (size_t)a.n;
    const double* st = (S == 1) ? a.y : a.ys;
    const double h = cs.h;
    double kS;
    if (c < 3) {
        kS = st[(3 + c) * N + i];
    } else {
        const int ax = c - 3, o = ax == 0 ? 1 : 0;
        const double f = sg_field_axis(cl.fp, fk, a.qm[i], ax, st[ax * N + i], st[c * N + i],
                                       st[o * N + i], st[(3 + o) * N + i]);
        kS = f + a.kq[i] * P;
    }
    double* k = a.k + (size_t)c * N + i;
    const size_t KS = 6 * N;
    k[(S - 1) * KS] = kS;
    if constexpr (S < M::stages) {
        // y + h sum_j a[S+1][j] k_j   (bin/ode.cpp:107-173)
        double s = 0.0;
#pragma unroll
        for (int j = 1; j < S; j++) s += M::a(S + 1, j - 1) * k[(j - 1) * KS];
        s += M::a(S + 1, S - 1) * kS;
        return a.y[c * N + i] + h * s;
    } else {
        // embedded error of the attempt (bin/ode.cpp:189-205); Dormand-Prince: y5 is the
        // stage-7 state; Cash-Karp: y + h sum b k
        double e = 0.0, b = 0.0;
#pragma unroll
        for (int j = 1; j <= S; j++) {
            const double kj = j < S ? k[(j - 1) * KS] : kS;
            if constexpr (M::stages == 6) {
                b += c_ck_b[j] * kj;
                e += M::e(j) * kj;
            } else {
                if (j != 2) e += M::e(j) * kj;
            }
        }
        const double y0 = a.y[c * N + i];
        const double y5 = M::stages == 6 ? y0 + h * b : a.ys[c * N + i];
        if constexpr (M::stages == 6) sol = y5;
        const double m0 = fabs(y0), m1 = fabs(y5);
        const double sk = cs.atol + cs.rtol * ((m0 < m1) ? m1 : m0);
        const double r = h * e * stage_rcp(sk);
        return r * r;
    }
}

// Component of a thread's slot (threads of R rows); -1: none.  At R = 16 the eight
// half-warp slots are x y | z - | ax ay | az -.
__device__ __forceinline__ int stage_component(int slot, int R) {
    return R > 16 ? slot : slot == 3 || slot == 7 ? -1 : slot < 3 ? slot : slot - 1;
}

// Sum of one value per thread over the block, in a fixed order (thread 0's result).
__device__ __forceinline__ double stage_block_sum(double v) {
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if ((threadIdx.x & 31) == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        const int lane = threadIdx.x & 31;
        v = lane < nw ? red[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;
}

}  // namespace
