// fp32c_math.cuh -- value-only arithmetic of the FP32-compensated Coulomb form, shared
// by the tiled kernels (coulomb.cu) and the fused small-cloud kernel (fused.cu) so that
// both take their pair terms, compensated sums and FP64 re-evaluations with the same
// operations: the SFU reciprocal square root, packed FP32x2 arithmetic, the float-float
// pair term, Kahan summation, float-float close-pair terms, and the FP64 1/r^3.
#pragma once

#include <cuda_runtime.h>

namespace {

__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// packed FP32x2 (two floats in one 64-bit register pair)
typedef unsigned long long f2;
__device__ __forceinline__ f2 pk(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(f2 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Softening added to r^2 in frame units (u ~ 1): below the rounding of any real
// pair distance, it keeps the self pair (dx = 0) finite: 1/r^3 = 1e36 < FLT_MAX.
constexpr float kTiny = 1e-24f;

// One FP32c pair term, scalar form.  Written with explicit rounding intrinsics so the
// close-pair re-evaluation reproduces it bit for bit.
struct PairF {
    float dx, dy, dz, y3;
};
__device__ __forceinline__ PairF pair_f32(float xjh, float yjh, float zjh, float xjl, float yjl,
                                          float zjl, float xih, float yih, float zih, float xil,
                                          float yil, float zil) {
    PairF p;
    p.dx = __fadd_rn(__fsub_rn(xjh, xih), __fsub_rn(xjl, xil));
    p.dy = __fadd_rn(__fsub_rn(yjh, yih), __fsub_rn(yjl, yil));
    p.dz = __fadd_rn(__fsub_rn(zjh, zih), __fsub_rn(zjl, zil));
    float r2 = __fmaf_rn(p.dx, p.dx, kTiny);
    r2 = __fmaf_rn(p.dy, p.dy, r2);
    r2 = __fmaf_rn(p.dz, p.dz, r2);
    const float y = rsqrt_approx(r2);
    p.y3 = __fmul_rn(__fmul_rn(y, y), y);
    return p;
}

__device__ __forceinline__ void kahan_add(float& s, float& c, float x) {
    const float y = __fsub_rn(x, c);
    const float t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
}


// r2^(-3/2) in FP64: the SFU's FP64 reciprocal square root y0 (rsqrt.approx.ftz.f64,
// measured |1 - r2 y0^2| <= 1.9e-6), then y0^3 (1 + 3e/2 + 15 e^2/8), the binomial series
// of (1-e)^(-3/2) with e = 1 - r2 y0^2; the truncation error is 35/16 e^3 < 1.5e-17.
// GB300 runs every FP64 warp instruction, conversions to and from FP32 included, in 64
// cycles of its SM sub-partition and the SFU's FP64 seed in 8: this is 6 such
// instructions, where an FP32 seed with its two conversions, a refined 1/r and its cube
// were 9.
__device__ __forceinline__ double inv_r3_fp64(double r2) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(r2));
    const double t = y0 * y0;
    const double e = fma(-r2, t, 1.0);
    const double y3 = t * y0;
    return fma(y3 * e, fma(e, 1.875, 1.5), y3);
}

// Sums of one value per lane and component: x in lane 0, y in lane 16, z in lane 8.  An FP64
// addition takes a warp 64 cycles whatever its lanes hold: 32 lanes x 3 components in six
// (the upper half-warp takes y while the lower sums x, then every other 8 lanes z).
__device__ __forceinline__ double warp_sum3(double ax, double ay, double az) {
    const int lane = threadIdx.x & 31;
    const bool up = lane & 16, odd = lane & 8;
    double a = up ? ay : ax;
    a += __shfl_xor_sync(0xffffffffu, up ? ax : ay, 16);
    az += __shfl_xor_sync(0xffffffffu, az, 16);
    double v = odd ? az : a;
    v += __shfl_xor_sync(0xffffffffu, odd ? a : az, 8);
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---- float-float (unevaluated sums hi + lo of two floats, ~48 bits) ------------------
struct ff {
    float h, l;
};
__device__ __forceinline__ ff ff_fast_two_sum(float a, float b) {  // |a| >= |b| or a == 0
    const float s = __fadd_rn(a, b);
    return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ ff ff_two_sum(float a, float b) {
    const float s = __fadd_rn(a, b);
    const float t = __fsub_rn(s, a);
    return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ ff ff_two_prod(float a, float b) {
    const float p = __fmul_rn(a, b);
    return {p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ ff ff_add(ff a, ff b) {
    const ff s = ff_two_sum(a.h, b.h);
    return ff_fast_two_sum(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
// (ah + al) - (bh + bl) of two float-float coordinates
__device__ __forceinline__ ff ff_diff(float ah, float al, float bh, float bl) {
    const ff s = ff_two_sum(ah, -bh);
    return ff_fast_two_sum(s.h, __fadd_rn(s.l, __fsub_rn(al, bl)));
}
__device__ __forceinline__ ff ff_sqr(ff a) {
    const ff p = ff_two_prod(a.h, a.h);
    return {p.h, __fmaf_rn(__fmul_rn(2.0f, a.h), a.l, p.l)};
}
__device__ __forceinline__ ff ff_mul(ff a, ff b) {
    const ff p = ff_two_prod(a.h, b.h);
    return {p.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, p.l))};
}

// Beyond this 1/r^3 (frame units: closer than 1e-5 of the cloud's spread) a close pair's
// distance is taken from the SI coordinates in FP64.  Float-float frame coordinates have an
// error of ~2^-49 |u|, so the distance grows with the ion's |u| where that is above 1 (the
// frame stays where the cloud was uploaded, the cloud need not): a pair farther apart than
// 1e-5 max(1, |u|) has its distance to ~4e-10 and its term to ~1e-9.  (Without the factor a
// pair 1.2e-5 spreads apart, 10,000 spreads away from the frame: 6e-7; so: 1e-11.)
constexpr float kVeryClose = 1e15f;
__device__ __forceinline__ bool very_close(float y3, float x, float y, float z) {
    const float m = fmaxf(fmaxf(1.0f, fabsf(x)), fmaxf(fabsf(y), fabsf(z)));
    return y3 * m * m * m > kVeryClose;  // infinity: the FP64 form
}

// A close pair's exact term q u / |u|^3 (u = u_j - u_i in float-float; q the normalized
// charge) minus the capped FP32 term wf d the main loop has summed, per component, in
// frame units.  FP32 instructions only: in FP64 (64 cycles each whatever the active
// lanes) the ~30 operations of one close pair cost its warp ~2,500 cycles, which on
// clouds of a few thousand ions was half of the pair kernel.
__device__ __forceinline__ void close_term_ff(ff ux, ff uy, ff uz, float q, float wf,
                                              const PairF& p, ff& cx, ff& cy, ff& cz) {
    const ff r2 = ff_add(ff_add(ff_sqr(ux), ff_sqr(uy)), ff_sqr(uz));
    const float y = rsqrt_approx(r2.h);
    const ff y2 = ff_two_prod(y, y);
    const ff t = ff_two_prod(r2.h, y2.h);
    // e = 1 - r2 y^2, |e| ~ 2^-22
    float e = __fsub_rn(__fsub_rn(1.0f, t.h), t.l);
    e = __fmaf_rn(-r2.h, y2.l, e);
    e = __fmaf_rn(-r2.l, y2.h, e);
    const ff y3 = ff_two_prod(y2.h, y);
    // y^3 (1-e)^(-3/2), then the charge
    const float c = __fmul_rn(e, __fmaf_rn(e, 1.875f, 1.5f));
    ff w = ff_fast_two_sum(y3.h, __fmaf_rn(y3.h, c, __fmaf_rn(y2.l, y, y3.l)));
    w = ff_mul(w, {q, 0.f});
    const ff dx = ff_two_prod(wf, p.dx), dy = ff_two_prod(wf, p.dy), dz = ff_two_prod(wf, p.dz);
    cx = ff_add(ff_mul(w, ux), {-dx.h, -dx.l});
    cy = ff_add(ff_mul(w, uy), {-dy.h, -dy.l});
    cz = ff_add(ff_mul(w, uz), {-dz.h, -dz.l});
}

// The conditioning estimate of an ion: the sum of squares of its FP32 partial sums, or,
// if larger, the squared magnitude of its strongest single pair term, |f|^2 = (1/r^3)^(4/3)
// in frame units for a unit charge (y3max, self pair excluded; in tiles with a close
// pair, the pairs below the cap and the capped terms, capped_term_y3).  A dominant pair
// whose partial sum is cancelled by other terms of the same block must still flag the ion
// for the FP64 re-evaluation of its row.  A threshold test: FP32 suffices (an overflow to
// infinity only flags the ion).
// A close pair (y3 > wc) enters the main loop's sums with its 1/r^3 capped at wc: a term
// of magnitude wc r, whose rounding in the partial sum stays although the pair itself is
// re-evaluated exactly.  As a strongest-term candidate it counts as the y3 whose |f| is
// that magnitude: (wc r)^(3/2) = wc sqrt(wc / y3) (<= wc).
__device__ __forceinline__ float capped_term_y3(float y3, float wc) {
    return wc * sqrtf(wc / y3);
}

__device__ __forceinline__ float conditioning_s2(float s2, float y3max) {
    const float r1 = cbrtf(y3max);  // 1/r
    const float f = r1 * r1;        // |f| = 1/r^2
    return fmaxf(s2, f * f);
}

}  // namespace
