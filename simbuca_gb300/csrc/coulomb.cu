// coulomb.cu -- direct-sum Coulomb kernels of libsimgb (sm_103a).
//
// Both kernels compute, for every i-ion of a work item and the j-range of the item,
//     P_i = sum_{j != i} q_j (x_i - x_j) / |x_i - x_j|^3          (SI units, m^-2)
// and store P_i in the item's partial-sum slot; the stage kernels multiply the sum of
// the slots by kq_i = coulomb_scale k_e e^2 q_i / m_i.  This is the CPU loop of the
// reference (bin/force.cpp:147-174) regrouped into tiles: same pair terms, no
// softening, self term excluded by index.
//
// FP32c (coulomb_fp32c_kernel): pair terms in FP32 on cloud-frame coordinates
// u = (x - c)/L held as float-float pairs (hi, lo).  The difference
// u_j - u_i = (hi_j - hi_i) + (lo_j - lo_i) keeps the pair distance accurate to an
// FP32 rounding even for ions far from the frame centre.  1/r is the SFU
// approximation (rsqrt.approx), 1/r^3 is capped at wc: the rare close pairs whose
// 1/r^3 exceeds wc are re-evaluated in float-float (the very closest in FP64) once the
// tile is done, and the capped FP32 contribution is taken out again exactly.  Within a 128-ion j-tile the terms
// are summed in FP32; tile sums are added with Kahan compensation.  Arithmetic uses
// the packed FP32x2 instructions of sm_100+ (add/mul/fma.rn.f32x2) on pairs of
// consecutive j-ions.  j-tiles are fetched with TMA bulk copies (cp.async.bulk) into
// a 4-stage shared-memory ring guarded by mbarriers.  Clouds in k-d order (shape 17) take
// each unordered pair of 128-ion leaves once instead (coulomb_leaf_kernel).
//
// FP64 (coulomb_fp64_sym_kernel, fp64_pairs.cuh): the plain form, every operation in
// FP64, each unordered pair evaluated once; 1/r^3 is the SFU's FP64 seed refined by one
// third-order step of the binomial series (inv_r3_fp64), accurate to ~1 ulp.
#include <stdio.h>

#include <algorithm>

#include "fp32c_math.cuh"
#include "fp64_pairs.cuh"
#include "sg_internal.cuh"

namespace {

// ---- PTX helpers ---------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait on an mbarrier phase: false once limit_ns have passed.
__device__ __forceinline__ bool mbar_wait_for(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = globaltimer();
    for (;;) {
        if (mbar_try(bar, parity)) return true;
        if (globaltimer() - t0 > limit_ns) return false;
    }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    return mbar_wait_for(bar, parity, SG_WAIT_NS);
}
// The wait test (flags[SG_FLAG_WAIT_TILE] = t + 1): after tile t has arrived, the block
// also waits on `never`, a barrier that nothing arrives at, until the test's limit runs
// out; the kernel then takes its timeout path, whose drain finds every issued copy landed.
__device__ __forceinline__ bool wait_test(uint64_t* never, const int* flags) {
    const uint64_t limit = 1000ull * (uint64_t)max(flags[SG_FLAG_WAIT_US], 1);
    return mbar_wait_for(never, 0, limit);
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Close pairs of one flagged ion (lane src's, padded index ig) among the j-ions
// [jb, je) of one shared-memory tile, by the whole warp (lanes stride over the j-ions):
// pairs whose FP32 1/r^3 exceeded wc get their exact term minus the capped FP32 term the
// main loop already summed, added in lane order to the ion's float-float corrections
// corr[0..5][li] (hi x, y, z, lo x, y, z; frame units) by lane src.  Returns the strongest
// FP32 term of these j-ions as a y3 (pairs below the cap, capped terms: capped_term_y3),
// which the main loop's y3max cannot give where there is a close pair.
template <int TL, int NI>
__device__ __forceinline__ float close_pairs_warp(const float (*tl)[TL], int jb, int je, int j0,
                                                  int ig, float xih, float yih, float zih,
                                                  float xil, float yil, float zil, float wc,
                                                  double sc, const double* __restrict__ c64,
                                                  int npad_total, int src, float (*corr)[NI],
                                                  int li) {
    const int lane = threadIdx.x & 31;
    float ym = 0.f;
    for (int j1 = jb; j1 < je; j1 += 32) {
        const int jj = j1 + lane;
        bool close = false;
        ff cx{0.f, 0.f}, cy{0.f, 0.f}, cz{0.f, 0.f};
        if (jj < je) {
            const float xh = tl[0][jj], yh = tl[1][jj], zh = tl[2][jj], q = tl[3][jj];
            const float xl = tl[4][jj], yl = tl[5][jj], zl = tl[6][jj];
            const PairF p = pair_f32(xh, yh, zh, xl, yl, zl, xih, yih, zih, xil, yil, zil);
            const int jg = j0 + jj;
            if (jg != ig && q != 0.f) {
                close = p.y3 > wc;
                ym = fmaxf(ym, close ? capped_term_y3(p.y3, wc) : p.y3);
            }
            if (close) {
                const float wf = __fmul_rn(q, wc);
                if (!very_close(p.y3, xih, yih, zih)) {
                    close_term_ff(ff_diff(xh, xl, xih, xil), ff_diff(yh, yl, yih, yil),
                                  ff_diff(zh, zl, zih, zil), q, wf, p, cx, cy, cz);
                } else {
                    const size_t NP = (size_t)npad_total;
                    const double rx = c64[ig] - c64[jg], ry = c64[NP + ig] - c64[NP + jg],
                                 rz = c64[2 * NP + ig] - c64[2 * NP + jg];
                    const double w = c64[3 * NP + jg] * inv_r3_fp64(rx * rx + ry * ry + rz * rz);
                    const double c[3] = {w * rx / sc - (double)wf * (double)p.dx,
                                         w * ry / sc - (double)wf * (double)p.dy,
                                         w * rz / sc - (double)wf * (double)p.dz};
                    cx.h = (float)c[0];
                    cx.l = (float)(c[0] - (double)cx.h);
                    cy.h = (float)c[1];
                    cy.l = (float)(c[1] - (double)cy.h);
                    cz.h = (float)c[2];
                    cz.l = (float)(c[2] - (double)cz.h);
                }
            }
        }
        unsigned m = __ballot_sync(0xffffffffu, close);
        while (m) {
            const int from = __ffs(m) - 1;
            m &= m - 1;
            ff a, b, c;
            a.h = __shfl_sync(0xffffffffu, cx.h, from);
            a.l = __shfl_sync(0xffffffffu, cx.l, from);
            b.h = __shfl_sync(0xffffffffu, cy.h, from);
            b.l = __shfl_sync(0xffffffffu, cy.l, from);
            c.h = __shfl_sync(0xffffffffu, cz.h, from);
            c.l = __shfl_sync(0xffffffffu, cz.l, from);
            if (lane == src) {
                a = ff_add({corr[0][li], corr[3][li]}, a);
                b = ff_add({corr[1][li], corr[4][li]}, b);
                c = ff_add({corr[2][li], corr[5][li]}, c);
                corr[0][li] = a.h;
                corr[1][li] = b.h;
                corr[2][li] = c.h;
                corr[3][li] = a.l;
                corr[4][li] = b.l;
                corr[5][li] = c.l;
            }
        }
    }
    // non-negative floats order as their bit patterns
    return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(ym)));
}

// The conditioning estimate's strongest FP32 term of the j-ions [jb, je) just summed
// (fmx), and their close pairs: one flagged ion at a time by the whole warp.  y3max: per
// ion the largest 1/r^3 of these j-ions, the self pair left out; reset here.  LI(k): the
// thread's k-th ion in the corrections array.
template <int IPT, int TL, int NI, typename LI>
__device__ __forceinline__ void fold_close(const float (*tl)[TL], int jb, int je, int j0,
                                           const int* ipad, const f2* xh, const f2* yh,
                                           const f2* zh, const f2* xl, const f2* yl, const f2* zl,
                                           float wc, double sc, const double* __restrict__ c64,
                                           int npad_total, float (*corr)[NI], float* y3max,
                                           float* fmx, LI li) {
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        const bool hit = y3max[k] > wc;
        if (!hit) fmx[k] = fmaxf(fmx[k], y3max[k]);
        y3max[k] = 0.f;
        unsigned m = __ballot_sync(0xffffffffu, hit && ipad[k] >= 0);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            float a, dummy;
            upk(xh[k], a, dummy);
            const float xih = __shfl_sync(0xffffffffu, a, src);
            upk(yh[k], a, dummy);
            const float yih = __shfl_sync(0xffffffffu, a, src);
            upk(zh[k], a, dummy);
            const float zih = __shfl_sync(0xffffffffu, a, src);
            upk(xl[k], a, dummy);
            const float xil = __shfl_sync(0xffffffffu, a, src);
            upk(yl[k], a, dummy);
            const float yil = __shfl_sync(0xffffffffu, a, src);
            upk(zl[k], a, dummy);
            const float zil = __shfl_sync(0xffffffffu, a, src);
            const int igs = __shfl_sync(0xffffffffu, ipad[k], src);
            const float ymx = close_pairs_warp<TL, NI>(tl, jb, je, j0, igs, xih, yih, zih, xil, yil,
                                                       zil, wc, sc, c64, npad_total, src, corr,
                                                       li(k));
            if ((threadIdx.x & 31) == src) fmx[k] = fmaxf(fmx[k], ymx);
        }
    }
}

// One ion's partial sums of a slot: the float-float sum hi x, y, z, lo x, y, z of the
// Kahan accumulator and the close-pair corrections in frame units, and the conditioning
// estimate s2.  No FP64: converting and scaling here cost every warp ~25 FP64
// instructions of 64 cycles per slot; the reduction does it once per ion.
template <int NI>
__device__ __forceinline__ void store_partial(float* __restrict__ P, size_t NP, int ig,
                                              const float* ks, const float* kc,
                                              float (*corr)[NI], int li, float s2, float fmx) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const ff v = ff_add({ks[c], -kc[c]}, {corr[c][li], corr[3 + c][li]});
        P[c * NP + ig] = v.h;
        P[(3 + c) * NP + ig] = v.l;
    }
    P[6 * NP + ig] = conditioning_s2(s2, fmx);
}

// Main loop over one shared-memory j-tile for the IPT ions of a thread: packed FP32x2
// over consecutive j pairs.  DIAG: the tile contains the thread's own ions, whose self
// pair must not raise the close-pair flag.
template <int IPT, bool DIAG, bool NOQ = false, int NU = 2>
__device__ __forceinline__ void tile_pairs(const float* tx, const float* ty, const float* tz,
                                           const float* tq, const float* txl, const float* tyl,
                                           const float* tzl, int jb, int je, int j0,
                                           const int* ipad,
                                           const f2* xh, const f2* yh, const f2* zh,
                                           const f2* xl, const f2* yl, const f2* zl, f2 tiny2,
                                           float wc, f2* ax, f2* ay, f2* az, float* y3max) {
#pragma unroll NU
    for (int jj = jb; jj < je; jj += 2) {
        const f2 Xj = *reinterpret_cast<const f2*>(tx + jj);
        const f2 Yj = *reinterpret_cast<const f2*>(ty + jj);
        const f2 Zj = *reinterpret_cast<const f2*>(tz + jj);
        const f2 Qj = NOQ ? 0ull : *reinterpret_cast<const f2*>(tq + jj);
        const f2 XLj = *reinterpret_cast<const f2*>(txl + jj);
        const f2 YLj = *reinterpret_cast<const f2*>(tyl + jj);
        const f2 ZLj = *reinterpret_cast<const f2*>(tzl + jj);
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const f2 dx = add2(sub2(Xj, xh[k]), sub2(XLj, xl[k]));
            const f2 dy = add2(sub2(Yj, yh[k]), sub2(YLj, yl[k]));
            const f2 dz = add2(sub2(Zj, zh[k]), sub2(ZLj, zl[k]));
            f2 r2 = fma2(dx, dx, tiny2);
            r2 = fma2(dy, dy, r2);
            r2 = fma2(dz, dz, r2);
            float ra, rb;
            upk(r2, ra, rb);
            const f2 y = pk(rsqrt_approx(ra), rsqrt_approx(rb));
            const f2 y3 = mul2(mul2(y, y), y);
            float ua, ub;
            upk(y3, ua, ub);
            if (DIAG) {
                const float ma = (j0 + jj == ipad[k]) ? 0.f : ua;
                const float mb = (j0 + jj + 1 == ipad[k]) ? 0.f : ub;
                y3max[k] = fmaxf(y3max[k], fmaxf(ma, mb));
            } else {
                y3max[k] = fmaxf(y3max[k], fmaxf(ua, ub));
            }
            const f2 wy = pk(fminf(ua, wc), fminf(ub, wc));
            const f2 w = NOQ ? wy : mul2(Qj, wy);
            ax[k] = fma2(w, dx, ax[k]);
            ay[k] = fma2(w, dy, ay[k]);
            az[k] = fma2(w, dz, az[k]);
        }
    }
}


// Squared distance between two tile bounding boxes (frame units).
__device__ __forceinline__ float box_dist2(const float* a, const float* b) {
    float d2 = 0.f;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float g = fmaxf(0.f, fmaxf(b[c] - a[3 + c], a[c] - b[3 + c]));
        d2 = fmaf(g, g, d2);
    }
    return d2;
}

// Far tiles: packed FP32x2 over j pairs, high parts only, no close pairs possible.
// FU: j pairs unrolled (0: 4 for one ion per thread, else 2).
template <int IPT, bool NOQ = false, int FU = 0>
__device__ __forceinline__ void tile_pairs_far(const float* tx, const float* ty, const float* tz,
                                               const float* tq, int jb, int je, const f2* xh,
                                               const f2* yh, const f2* zh, f2 tiny2, f2* ax,
                                               f2* ay, f2* az) {
    constexpr int kFarUnroll = FU > 0 ? FU : (IPT == 1 ? 4 : 2);  // more j pairs in flight
#pragma unroll kFarUnroll
    for (int jj = jb; jj < je; jj += 2) {
        const f2 Xj = *reinterpret_cast<const f2*>(tx + jj);
        const f2 Yj = *reinterpret_cast<const f2*>(ty + jj);
        const f2 Zj = *reinterpret_cast<const f2*>(tz + jj);
        const f2 Qj = NOQ ? 0ull : *reinterpret_cast<const f2*>(tq + jj);
#pragma unroll
        for (int k = 0; k < IPT; k++) {
            const f2 dx = sub2(Xj, xh[k]);
            const f2 dy = sub2(Yj, yh[k]);
            const f2 dz = sub2(Zj, zh[k]);
            f2 r2 = fma2(dx, dx, tiny2);
            r2 = fma2(dy, dy, r2);
            r2 = fma2(dz, dz, r2);
            float ra, rb;
            upk(r2, ra, rb);
            const f2 y = pk(rsqrt_approx(ra), rsqrt_approx(rb));
            const f2 y3 = mul2(mul2(y, y), y);
            const f2 w = NOQ ? y3 : mul2(Qj, y3);
            ax[k] = fma2(w, dx, ax[k]);
            ay[k] = fma2(w, dy, ay[k]);
            az[k] = fma2(w, dz, az[k]);
        }
    }
}

// ---------------------------------------------------------------------------
// FP32c kernel.  Global layout: c32 = 7 float arrays of npad_total entries
// (x, y, z, q, xl, yl, zl in frame units); shared tile = the same 7 arrays of SG_TILE.
// ---------------------------------------------------------------------------
template <int NT, int IPT>
__global__ void __launch_bounds__(NT) coulomb_fp32c_kernel(const float* __restrict__ c32,
                                                            const double* __restrict__ c64,
                                                            const SgWorkItem* __restrict__ items,
                                                            const SgCloud* __restrict__ clouds,
                                                            const SgCtrl* __restrict__ ctrl,
                                                            double* __restrict__ part,
                                                            int npad_total, int* errword) {
    sg_griddep_wait();
    constexpr int T = SG_TILE;
    __shared__ __align__(128) float tile[SG_STAGES][7][T];
    __shared__ __align__(8) uint64_t full[SG_STAGES];
    __shared__ __align__(8) uint64_t never;  // the wait test's barrier
    __shared__ float corr[6][NT * IPT];

    const SgWorkItem it = items[blockIdx.x];
    const int wtest = errword ? errword[SG_FLAG_WAIT_TILE] : 0;
    if (ctrl != nullptr && (ctrl[it.cloud].done || ctrl[it.cloud].hold || ctrl[it.cloud].status != SG_OK)) return;
    const SgCloud& cl = clouds[it.cloud];
    const float wc = cl.wc;
    // uniform-charge clouds hold q_j / qscale (1 for ions, 0 for padding): tiles without
    // padding skip the charge product and the sums are scaled once at the end
    const double sc = cl.psc;
    const int j_real_end = cl.poff + cl.n;
    const int tid = threadIdx.x;
    const float* X = c32;
    const float* Y = c32 + npad_total;
    const float* Z = c32 + 2 * (size_t)npad_total;
    const float* XL = c32 + 4 * (size_t)npad_total;
    const float* YL = c32 + 5 * (size_t)npad_total;
    const float* ZL = c32 + 6 * (size_t)npad_total;

    // i-ions of this thread: it.i0 + tid + k*NT (clamped into the item for loads)
    int ipad[IPT];
    f2 xh[IPT], yh[IPT], zh[IPT], xl[IPT], yl[IPT], zl[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        int li = tid + k * NT;
        int ii = it.i0 + (li < it.ni ? li : 0);
        ipad[k] = li < it.ni ? ii : -1;
        float a = X[ii], b = Y[ii], c = Z[ii], d = XL[ii], e = YL[ii], f = ZL[ii];
        xh[k] = pk(a, a);
        yh[k] = pk(b, b);
        zh[k] = pk(c, c);
        xl[k] = pk(d, d);
        yl[k] = pk(e, e);
        zl[k] = pk(f, f);
#pragma unroll
        for (int c = 0; c < 6; c++) corr[c][li] = 0.f;
    }
    float ks[IPT][3], kc[IPT][3], s2[IPT], fmx[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        s2[k] = 0.f;
        fmx[k] = 0.f;
#pragma unroll
        for (int c = 0; c < 3; c++) ks[k][c] = kc[k][c] = 0.f;
    }

    const int ntiles = (it.nj + T - 1) / T;
    bool ok = true;
    if (tid == 0) {
        for (int s = 0; s < SG_STAGES; s++) mbar_init(&full[s], 1);
        mbar_init(&never, 1);
        fence_mbar_init();
    }
    __syncthreads();
    // prologue: fill the ring
    if (tid == 0) {
        for (int s = 0; s < SG_STAGES && s < ntiles; s++) {
            const int j0 = it.j0 + s * T;
            const int len = min(T, it.j0 + it.nj - j0);
            const uint32_t bytes = (uint32_t)len * 4u;
            mbar_arrive_tx(&full[s], 7u * bytes);
            for (int a = 0; a < 7; a++)
                bulk_g2s(&tile[s][a][0], c32 + (size_t)a * npad_total + j0, bytes, &full[s]);
        }
    }

    const f2 tiny2 = pk(kTiny, kTiny);
    // one ion per thread (the small-cloud shapes): four j pairs in flight per thread
    constexpr int kNU = IPT == 1 ? 4 : 2;
    // Small clouds fold partial sums every 16 j-ions so that the squared partial sums
    // still estimate sum_j |f_ij|^2 when the whole cloud is one or two tiles.
    const int flush_len = (cl.npad <= 2048) ? 16 : SG_TILE;
    for (int t = 0; t < ntiles; t++) {
        const int s = t % SG_STAGES;
        const uint32_t parity = (uint32_t)((t / SG_STAGES) & 1);
        const int j0 = it.j0 + t * T;
        const int len = min(T, it.j0 + it.nj - j0);
        bool arrived = mbar_wait(&full[s], parity);
        if (t + 1 == wtest) arrived = wait_test(&never, errword) && arrived;
        if (!__syncthreads_and(arrived)) {  // block-uniform decision
            ok = false;
            if (tid == 0) {
                atomicExch(errword, SG_TIMEOUT);
                // drain the copies still in flight (tiles t .. t+STAGES-1), bounded
                for (int u = t; u < ntiles && u < t + SG_STAGES; u++)
                    (void)mbar_wait(&full[u % SG_STAGES], (uint32_t)((u / SG_STAGES) & 1));
            }
            __syncthreads();
            break;
        }

        float y3max[IPT];
#pragma unroll
        for (int k = 0; k < IPT; k++) y3max[k] = 0.f;
        const float* tx = tile[s][0];
        const float* ty = tile[s][1];
        const float* tz = tile[s][2];
        const float* tq = tile[s][3];
        const float* txl = tile[s][4];
        const float* tyl = tile[s][5];
        const float* tzl = tile[s][6];
        // The tile holding this block's own ions takes the variant that keeps the self
        // pair (dx = 0, contributes nothing) out of the close-pair flag.
        const bool diag = (j0 < it.i0 + it.ni) && (j0 + len > it.i0);
        // no padding ions in this tile: their normalized charge 0 is the only one not 1
        const bool noq = cl.quniform && j0 + len <= j_real_end;
        for (int jb = 0; jb < len; jb += flush_len) {
            const int je = min(len, jb + flush_len);
            f2 ax[IPT], ay[IPT], az[IPT];
#pragma unroll
            for (int k = 0; k < IPT; k++) ax[k] = ay[k] = az[k] = 0ull;
            if (!diag && noq)
                tile_pairs<IPT, false, true, kNU>(tx, ty, tz, tq, txl, tyl, tzl, jb, je, j0, ipad, xh,
                                             yh, zh, xl, yl, zl, tiny2, wc, ax, ay, az, y3max);
            else if (!diag)
                tile_pairs<IPT, false, false, kNU>(tx, ty, tz, tq, txl, tyl, tzl, jb, je, j0, ipad, xh, yh, zh,
                                       xl, yl, zl, tiny2, wc, ax, ay, az, y3max);
            else
                tile_pairs<IPT, true, false, kNU>(tx, ty, tz, tq, txl, tyl, tzl, jb, je, j0, ipad, xh, yh, zh,
                                      xl, yl, zl, tiny2, wc, ax, ay, az, y3max);
            // fold the partial sums into the compensated accumulators
#pragma unroll
            for (int k = 0; k < IPT; k++) {
                float a, b;
                upk(ax[k], a, b);
                const float tx_ = __fadd_rn(a, b);
                upk(ay[k], a, b);
                const float ty_ = __fadd_rn(a, b);
                upk(az[k], a, b);
                const float tz_ = __fadd_rn(a, b);
                kahan_add(ks[k][0], kc[k][0], tx_);
                kahan_add(ks[k][1], kc[k][1], ty_);
                kahan_add(ks[k][2], kc[k][2], tz_);
                // sum of squared partial sums: estimates sum_j |f_ij|^2 (conditioning test)
                s2[k] = fmaf(tx_, tx_, fmaf(ty_, ty_, fmaf(tz_, tz_, s2[k])));
            }
            fold_close<IPT>(tile[s], jb, je, j0, ipad, xh, yh, zh, xl, yl, zl, wc, sc, c64,
                            npad_total, corr, y3max, fmx, [tid](int k) { return tid + k * NT; });
        }
        __syncthreads();  // every thread is done with ring slot s
        if (tid == 0 && t + SG_STAGES < ntiles) {
            fence_proxy_async();
            const int jn = it.j0 + (t + SG_STAGES) * T;
            const int ln = min(T, it.j0 + it.nj - jn);
            const uint32_t bytes = (uint32_t)ln * 4u;
            mbar_arrive_tx(&full[s], 7u * bytes);
            for (int a = 0; a < 7; a++)
                bulk_g2s(&tile[s][a][0], c32 + (size_t)a * npad_total + jn, bytes, &full[s]);
        }
    }
    if (!ok) return;
    const size_t NP = (size_t)npad_total;
    float* P = reinterpret_cast<float*>(part) + (size_t)it.slot * SG_PART_F32 * NP;
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        if (ipad[k] < 0) continue;
        store_partial(P, NP, ipad[k], ks[k], kc[k], corr, tid + k * NT, s2[k], fmx[k]);
        P[7 * NP + ipad[k]] = 0.f;  // no far tiles in this form
    }
}

// Adds packed partial sums (two interleaved FP32 sums per ion and component) into the
// compensated accumulators, and their squares into the conditioning estimate of the
// near tiles (s2: the pairs the FP64 fix-up re-evaluates) or of the far tiles (s2f: the
// hi-only pair terms, whose error grows with it; in k-d order a far tile's 32-ion sums
// are coherent, so s2f is kept apart rather than flagging ions through s2).
template <int IPT, bool S2F = true>
__device__ __forceinline__ void fold_partials(const f2* ax, const f2* ay, const f2* az,
                                              float (*ks)[3], float (*kc)[3], float* s2,
                                              float* s2f, bool near) {
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        float a, b;
        upk(ax[k], a, b);
        const float tx_ = __fadd_rn(a, b);
        upk(ay[k], a, b);
        const float ty_ = __fadd_rn(a, b);
        upk(az[k], a, b);
        const float tz_ = __fadd_rn(a, b);
        kahan_add(ks[k][0], kc[k][0], tx_);
        kahan_add(ks[k][1], kc[k][1], ty_);
        kahan_add(ks[k][2], kc[k][2], tz_);
        if (near)
            s2[k] = fmaf(tx_, tx_, fmaf(ty_, ty_, fmaf(tz_, tz_, s2[k])));
        else if (S2F)
            s2f[k] = fmaf(tx_, tx_, fmaf(ty_, ty_, fmaf(tz_, tz_, s2f[k])));
    }
}

// ---- k-d ordered clouds, leaf pairs once (shape 17) -----------------------------------
// Every unordered pair of 128-ion leaves is evaluated once, for both leaves, by one warp.
// A pair of leaves farther apart than d_far is summed from the high parts (far_warp); a near
// one, 5 % of the pairs of a 65,536-ion cloud and 36 % of a 4,000-ion one, keeps the
// float-float differences, the capped close pairs and the conditioning of the kernels
// above (near_warp).  Both sides' sums go to 64-bit fixed-point accumulators.

// The near leaves J >= I of every leaf I, in order (I itself first): one warp per leaf of
// the batch; lists[leaf] holds cap entries, counts[leaf] of them used.
__global__ void __launch_bounds__(128) near_list_kernel(const SgCloud* __restrict__ clouds,
                                                        const SgCtrl* __restrict__ ctrl,
                                                        const int* __restrict__ leaf_cloud,
                                                        int n_leaves, int cap,
                                                        const float* __restrict__ bbox,
                                                        int* __restrict__ counts,
                                                        unsigned short* __restrict__ lists,
                                                        int* __restrict__ fix_list) {
    sg_griddep_wait();
    // the fix-up lists of this call (a memset otherwise)
    if (blockIdx.x == 0 && threadIdx.x < 2) fix_list[threadIdx.x] = 0;
    const int leaf = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (leaf >= n_leaves) return;
    const int c = leaf_cloud[leaf];
    if (c < 0) return;
    if (ctrl != nullptr && (ctrl[c].done || ctrl[c].hold || ctrl[c].status != SG_OK)) return;
    const SgCloud& cl = clouds[c];
    const int nt = (cl.npad + SG_TILE - 1) / SG_TILE, own = leaf - cl.tile0;
    const float dfar2 = cl.dfar * cl.dfar;
    float ib[6];
    for (int q = 0; q < 6; q++) ib[q] = bbox[8 * (size_t)leaf + q];
    unsigned short* L = lists + (size_t)leaf * cap;
    int m = 0;
    for (int j0 = own; j0 < nt; j0 += 32) {
        // past the end: the last leaf again, not listed (every lane takes the same path)
        const int J = min(j0 + lane, nt - 1);
        float jb[6];
#pragma unroll
        for (int q = 0; q < 6; q++) jb[q] = bbox[8 * (size_t)(cl.tile0 + J) + q];
        const bool near = j0 + lane < nt && (J == own || !(box_dist2(ib, jb) > dfar2));
        const unsigned b = __ballot_sync(0xffffffffu, near);
        if (near) L[m + __popc(b & ((1u << lane) - 1u))] = (unsigned short)J;
        __syncwarp();
        m += __popc(b);
    }
    if (lane == 0) counts[leaf] = m;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ f2 shfl2(f2 v, int src) {
    return __shfl_sync(0xffffffffu, v, src);
}

// v (a float-float far sum in frame units) in the cloud's fixed point: round(v fs).  The
// bound on the far sums keeps |v fs| below 2^54 (far_scale in capi.cu), so the high part
// splits exactly at 2^30 and both halves are 32-bit conversions.
__device__ __forceinline__ long long far_fixed(float h, float l, float fs) {
    const float a = __fmul_rn(h, fs);                        // exact: a power of two
    const int hi = __float2int_rn(__fmul_rn(a, 9.31322574615478515625e-10f));  // a / 2^30
    const float rem = __fmaf_rn(-(float)hi, 1073741824.0f, a);  // exact
    const int lo = __float2int_rn(__fmaf_rn(l, fs, rem));
    return ((long long)hi << 30) + lo;
}

// Accumulators of a batch in shape 17, per padded ion; all zero between calls.
struct LeafAcc {
    unsigned long long* sum;  // [5][Npad]: x, y, z; s2 of the near leaves; s2f of the far ones
    int* fmx;                 // strongest near term (1/r^3 below the cap, float bits); kPoison
    int* n_close;             // close pairs of the ion, and the first kCloseCap partners
    int* close;               // [Npad][kCloseCap]
};
constexpr int kCloseCap = SG_CLOSE_CAP;
constexpr int kPoison = 0x7fffffff;  // a sum that is not finite: fixed point cannot hold it

// Float-float sum (h, l) of component c of ion ig into the accumulators.
__device__ __forceinline__ void leaf_add(const LeafAcc& A, size_t NP, int c, int ig, float h,
                                         float l, float fs) {
    if (!(fabsf(h) <= 3.402823466e38f)) A.fmx[ig] = kPoison;
    atomicAdd(A.sum + c * NP + ig, (unsigned long long)far_fixed(h, l, fs));
}

// The wait test (flags[SG_FLAG_WAIT_TILE] = t + 1) in a warp of the leaf kernel with more than
// t leaf pairs to take: it waits until the test's limit has passed, raises SG_TIMEOUT and adds
// nothing.  Its copies are cp.async groups, which have no wait that could run out.
__device__ __forceinline__ bool leaf_wait_test(int* flags, int pairs) {
    const int t = flags[SG_FLAG_WAIT_TILE];
    if (t == 0 || t > pairs) return false;
    const uint64_t limit = 1000ull * (uint64_t)max(flags[SG_FLAG_WAIT_US], 1), t0 = globaltimer();
    while (globaltimer() - t0 <= limit) {
    }
    if ((threadIdx.x & 31) == 0) atomicExch(flags, SG_TIMEOUT);
    return true;
}

// Far pairs of leaf I against up to 32 leaves J > I, by one warp, each unordered pair
// once, from the high parts.  Bound by the FMA pipe: 8 packed FP32x2 operations shared by
// the two ions and 3 for each, 7 lane operations per ordered pair where summing each
// ordered pair takes 11.
//
// Lane l keeps four ions of I (4 l ...) in registers with their sums; the ions of J
// pass through the lanes as packed pairs: at step s lane l meets j-pair (l + s) mod 32 of a
// 64-ion half-leaf, whose running sum it takes from lane l + 1, so no two lanes ever add
// to one j-ion.  Both sides' FP32 sums are folded into Kahan pairs in shared memory after
// chains of 32 terms.  The leaf sums of both
// sides are added to the cloud's far accumulators as 64-bit fixed point: integer
// additions commute, so the result does not depend on the order the warps run in, and
// there are no partial-sum slots to store and add up.
//
// Register reads bound it before the FMA pipe: a packed FMA of three distinct operands
// takes 3.1 - 3.6 cycles of its SM sub-partition, one of two 2.0 (measured), which makes
// the pair 17 cycles, not 14.  Near and far leaves of a 65,536-ion cloud: 1,245 us per
// call, 1,755 with the ordered pairs of shape 9; 500,009 ions 67.9 ms, 98.
constexpr int kFarFold = 8;  // steps between j-side folds
template <bool S2F>
struct __align__(16) FarWarpShared {
    float j[2][4][SG_TILE];   // x, y, z, q of leaf J, two in flight
    float S[3][SG_TILE], C[3][SG_TILE];    // leaf J's Kahan pairs
    float IS[3][SG_TILE], IC[3][SG_TILE];  // leaf I's
    float s2[S2F ? SG_TILE : 4];
};

template <bool NOQ, bool S2F>
__device__ __forceinline__ void far_leaf(const float (*tj)[SG_TILE], FarWarpShared<S2F>& sh,
                                         const f2 (*xi)[4], const float* __restrict__ qg,
                                         float* s2i) {
    const int lane = threadIdx.x & 31, next = (lane + 1) & 31;
    const f2 tiny2 = pk(kTiny, kTiny);
    f2 qi[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const float q = NOQ ? 0.f : qg[4 * lane + k];
        qi[k] = pk(q, q);
    }
#pragma unroll 1
    for (int half = 0; half < 4; half++) {  // sixteen steps of a 64-ion half-leaf
        const int sub = half >> 1, r0 = (half & 1) * 16;
        f2 a[3][4];
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int k = 0; k < 4; k++) a[c][k] = 0ull;
#pragma unroll 1
        for (int s8 = r0; s8 < r0 + 16; s8 += kFarFold) {
            f2 b[3];
#pragma unroll
            for (int u = 0; u < kFarFold; u++) {
                const int p = 64 * sub + 2 * ((lane + s8 + u) & 31);
                const f2 X = *reinterpret_cast<const f2*>(&tj[0][p]);
                const f2 Y = *reinterpret_cast<const f2*>(&tj[1][p]);
                const f2 Z = *reinterpret_cast<const f2*>(&tj[2][p]);
                const f2 Q = NOQ ? 0ull : *reinterpret_cast<const f2*>(&tj[3][p]);
                if (u > 0) {
#pragma unroll
                    for (int c = 0; c < 3; c++) b[c] = shfl2(b[c], next);
                }
                // the step's four j-side terms are summed first: chains of 4 and 8
                // additions instead of one of 32, and the shuffles off the critical path
                f2 t[3];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const f2 dx = sub2(X, xi[0][k]), dy = sub2(Y, xi[1][k]), dz = sub2(Z, xi[2][k]);
                    f2 r2 = fma2(dx, dx, tiny2);
                    r2 = fma2(dy, dy, r2);
                    r2 = fma2(dz, dz, r2);
                    float ra, rb;
                    upk(r2, ra, rb);
                    const f2 y = pk(rsqrt_approx(ra), rsqrt_approx(rb));
                    const f2 y3 = mul2(mul2(y, y), y);
                    const f2 w = NOQ ? y3 : mul2(Q, y3);
                    a[0][k] = fma2(w, dx, a[0][k]);
                    a[1][k] = fma2(w, dy, a[1][k]);
                    a[2][k] = fma2(w, dz, a[2][k]);
                    const f2 v = NOQ ? y3 : mul2(qi[k], y3);
                    t[0] = k ? fma2(v, dx, t[0]) : mul2(v, dx);
                    t[1] = k ? fma2(v, dy, t[1]) : mul2(v, dy);
                    t[2] = k ? fma2(v, dz, t[2]) : mul2(v, dz);
                }
#pragma unroll
                for (int c = 0; c < 3; c++) b[c] = u ? add2(b[c], t[c]) : t[c];  // subtracted in the end
            }
            // j-side fold: the pair this lane has now
            const int p = 64 * sub + 2 * ((lane + s8 + kFarFold - 1) & 31);
            if (S2F) {
                f2 e = s8 ? *reinterpret_cast<f2*>(&sh.s2[p]) : 0ull;
                e = fma2(b[0], b[0], fma2(b[1], b[1], fma2(b[2], b[2], e)));
                *reinterpret_cast<f2*>(&sh.s2[p]) = e;
            }
#pragma unroll
            for (int c = 0; c < 3; c++) {
                f2* S = reinterpret_cast<f2*>(&sh.S[c][p]);
                f2* C = reinterpret_cast<f2*>(&sh.C[c][p]);
                if (s8 == 0) {  // every pair's first fold
                    *S = b[c];
                    *C = 0ull;
                } else {
                    const f2 s = *S, y = sub2(b[c], *C), t = add2(s, y);
                    *C = sub2(sub2(t, s), y);
                    *S = t;
                }
            }
            __syncwarp();  // the pair moves on to another lane
        }
        // i-side fold: two chains of 16 terms per component and ion
        float t[3][4];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float4* S = reinterpret_cast<float4*>(sh.IS[c]) + lane;
            float4* C = reinterpret_cast<float4*>(sh.IC[c]) + lane;
            float4 s4 = *S, c4 = *C;
            float* sp = &s4.x;
            float* cp = &c4.x;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                float lo, hi;
                upk(a[c][k], lo, hi);
                t[c][k] = __fadd_rn(lo, hi);
                kahan_add(sp[k], cp[k], t[c][k]);
            }
            *S = s4;
            *C = c4;
        }
        if (S2F)
#pragma unroll
            for (int k = 0; k < 4; k++)
                s2i[k] = fmaf(t[0][k], t[0][k], fmaf(t[1][k], t[1][k], fmaf(t[2][k], t[2][k], s2i[k])));
    }
}

template <bool S2F>
__device__ __forceinline__ void far_warp(const float* __restrict__ c32, const SgFarItem& it,
                                         const SgCloud& cl, const LeafAcc& acc, int npad_total,
                                         const float* __restrict__ bbox, int* flags,
                                         FarWarpShared<S2F>& sh) {
    const int lane = threadIdx.x & 31;
    const size_t NP = (size_t)npad_total;
    // far leaves of the item: a lane each
    unsigned m;
    {
        float ib[6], jb[6];
        const int J = it.j0 + (lane < it.n ? lane : 0);
        for (int q = 0; q < 6; q++) ib[q] = bbox[8 * (size_t)(cl.tile0 + it.leaf) + q];
        for (int q = 0; q < 6; q++) jb[q] = bbox[8 * (size_t)(cl.tile0 + J) + q];
        m = __ballot_sync(0xffffffffu, lane < it.n && box_dist2(ib, jb) > cl.dfar * cl.dfar);
    }
    if (m == 0 || leaf_wait_test(flags, __popc(m))) return;
    // leaf I is whole: only the last leaf of a cloud may not be, and I < J
    const int i0 = cl.poff + it.leaf * SG_TILE;
    f2 xi[3][4];
    float s2i[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const float x = c32[c * NP + i0 + 4 * lane + k];
            xi[c][k] = pk(x, x);
            sh.IS[c][lane + 32 * k] = sh.IC[c][lane + 32 * k] = 0.f;
        }
        s2i[k] = 0.f;
    }
    const float* qg = c32 + 3 * NP + i0;
    const float fs = cl.far_fs, fs2 = cl.far_fs2;
    auto fetch = [&](int J, int slot) {
        const int j0 = cl.poff + J * SG_TILE, len = min(SG_TILE, cl.poff + cl.npad - j0);
        float(*t)[SG_TILE] = sh.j[slot];
#pragma unroll
        for (int a = 0; a < 4; a++) {
            if (4 * lane < len)
                cp_async16(&t[a][4 * lane], c32 + a * NP + j0 + 4 * lane);
            else  // a cloud's last leaf: far away, no charge
#pragma unroll
                for (int q = 0; q < 4; q++) t[a][4 * lane + q] = a < 3 ? sg_leaf_fill(false) : 0.f;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int slot = 0;
    __syncwarp();
    fetch(it.j0 + __ffs(m) - 1, 0);
    while (m) {
        const int J = it.j0 + __ffs(m) - 1;
        m &= m - 1;
        if (m) {
            fetch(it.j0 + __ffs(m) - 1, slot ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        const int j0 = cl.poff + J * SG_TILE;
        if (cl.quniform && j0 + SG_TILE <= cl.poff + cl.n)
            far_leaf<true, S2F>(sh.j[slot], sh, xi, qg, s2i);
        else
            far_leaf<false, S2F>(sh.j[slot], sh, xi, qg, s2i);
        // leaf J's sums, their sign the pair's other side's
#pragma unroll 1
        for (int k = 0; k < 4; k++) {
            const int p = lane + 32 * k, jg = j0 + p;
            if (jg >= cl.poff + cl.n) continue;
#pragma unroll
            for (int c = 0; c < 3; c++) leaf_add(acc, NP, c, jg, -sh.S[c][p], sh.C[c][p], fs);
            if (S2F) leaf_add(acc, NP, 4, jg, sh.s2[p], 0.f, fs2);
        }
        __syncwarp();
        slot ^= 1;
    }
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int p = lane + 32 * k;
#pragma unroll
        for (int c = 0; c < 3; c++) leaf_add(acc, NP, c, i0 + p, sh.IS[c][p], -sh.IC[c][p], fs);
        if (S2F) leaf_add(acc, NP, 4, i0 + 4 * lane + k, s2i[k], 0.f, fs2);
    }
}

// Half a near leaf I (64 ions, two per lane) against near leaves J >= I, by one warp, each
// unordered pair once: the j-pairs pass through the lanes as in far_leaf.  Per packed pair
// of j-ions and i-ion 14 FP32x2 operations serve both sides and 3 each side, where the
// ordered pairs of the plain kernels take 17 each.  60 clouds of 4,096 ions (36 % of their
// pairs near): 485 us with ordered near pairs, 400 so.
//
// A close pair enters both sums capped (1/r^3 <= wc) and is noted in the lists of both ions:
// the sums' reduction adds its exact term minus the capped one, in the order of the
// partners' indices.  An ion with more close pairs than a list holds gets its FP64 row.
struct __align__(16) NearWarpShared {
    float j[2][7][SG_TILE];              // leaf J: x, y, z, q, low parts; two in flight
    float S[3][SG_TILE], C[3][SG_TILE];  // leaf J's Kahan pairs
    float s2[SG_TILE], M[SG_TILE];       // ... conditioning: sum of squares, strongest term
};
constexpr int kNearStep = 8;  // steps per FP32 partial sum: 16 terms on either side

struct NearSide {
    f2 x[6][2], q[2];  // the lane's two ions, each value twice
    float ks[2][3], kc[2][3], s2[2], fmx[2];
};

template <bool NOQ, bool TWO>
__device__ __forceinline__ void near_leaf(const float (*tj)[SG_TILE], NearWarpShared& sh,
                                          NearSide& w, float wc, int i0, int j0, int end,
                                          const LeafAcc& acc) {
    const int lane = threadIdx.x & 31, next = (lane + 1) & 31;
    const f2 tiny2 = pk(kTiny, kTiny);
#pragma unroll 1
    for (int g = 0; g < 64; g += kNearStep) {
        const int sub = g >> 5, s0 = g & 31;  // half-leaf of J, first step in it
        f2 a[3][2], b[3];
#pragma unroll
        for (int c = 0; c < 3; c++) a[c][0] = a[c][1] = b[c] = 0ull;
        float jm0 = 0.f, jm1 = 0.f;
        unsigned close = 0u;
#pragma unroll
        for (int u = 0; u < kNearStep; u++) {
            const int p = 64 * sub + 2 * ((lane + s0 + u) & 31);
            const f2 X = *reinterpret_cast<const f2*>(&tj[0][p]);
            const f2 Y = *reinterpret_cast<const f2*>(&tj[1][p]);
            const f2 Z = *reinterpret_cast<const f2*>(&tj[2][p]);
            const f2 Q = NOQ ? 0ull : *reinterpret_cast<const f2*>(&tj[3][p]);
            const f2 XL = *reinterpret_cast<const f2*>(&tj[4][p]);
            const f2 YL = *reinterpret_cast<const f2*>(&tj[5][p]);
            const f2 ZL = *reinterpret_cast<const f2*>(&tj[6][p]);
            if (TWO && u > 0) {
#pragma unroll
                for (int c = 0; c < 3; c++) b[c] = shfl2(b[c], next);
                jm0 = __shfl_sync(0xffffffffu, jm0, next);
                jm1 = __shfl_sync(0xffffffffu, jm1, next);
            }
            f2 t[3];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                const f2 dx = add2(sub2(X, w.x[0][k]), sub2(XL, w.x[3][k]));
                const f2 dy = add2(sub2(Y, w.x[1][k]), sub2(YL, w.x[4][k]));
                const f2 dz = add2(sub2(Z, w.x[2][k]), sub2(ZL, w.x[5][k]));
                f2 r2 = fma2(dx, dx, tiny2);
                r2 = fma2(dy, dy, r2);
                r2 = fma2(dz, dz, r2);
                float ra, rb, ua, ub;
                upk(r2, ra, rb);
                const f2 y = pk(rsqrt_approx(ra), rsqrt_approx(rb));
                upk(mul2(mul2(y, y), y), ua, ub);
                // the self pair (dx = 0) counts as close: no term, not listed
                const bool ca = ua > wc, cb = ub > wc;
                if (ca) close |= 1u << (4 * u + 2 * k);
                if (cb) close |= 2u << (4 * u + 2 * k);
                const float m0 = ca ? 0.f : ua, m1 = cb ? 0.f : ub;
                w.fmx[k] = fmaxf(w.fmx[k], fmaxf(m0, m1));
                const f2 cap = pk(fminf(ua, wc), fminf(ub, wc));
                const f2 wi = NOQ ? cap : mul2(Q, cap);
                a[0][k] = fma2(wi, dx, a[0][k]);
                a[1][k] = fma2(wi, dy, a[1][k]);
                a[2][k] = fma2(wi, dz, a[2][k]);
                if (TWO) {
                    jm0 = fmaxf(jm0, m0);
                    jm1 = fmaxf(jm1, m1);
                    const f2 wj = NOQ ? cap : mul2(w.q[k], cap);
                    t[0] = k ? fma2(wj, dx, t[0]) : mul2(wj, dx);
                    t[1] = k ? fma2(wj, dy, t[1]) : mul2(wj, dy);
                    t[2] = k ? fma2(wj, dz, t[2]) : mul2(wj, dz);
                }
            }
            if (TWO)
#pragma unroll
                for (int c = 0; c < 3; c++) b[c] = u ? add2(b[c], t[c]) : t[c];  // subtracted in the end
        }
        if (TWO) {  // j-side fold: the pair this lane has now
            const int p = 64 * sub + 2 * ((lane + s0 + kNearStep - 1) & 31);
            f2* S2 = reinterpret_cast<f2*>(&sh.s2[p]);
            *S2 = fma2(b[0], b[0], fma2(b[1], b[1], fma2(b[2], b[2], s0 ? *S2 : 0ull)));
            sh.M[p] = s0 ? fmaxf(sh.M[p], jm0) : jm0;
            sh.M[p + 1] = s0 ? fmaxf(sh.M[p + 1], jm1) : jm1;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                f2* S = reinterpret_cast<f2*>(&sh.S[c][p]);
                f2* C = reinterpret_cast<f2*>(&sh.C[c][p]);
                if (s0 == 0) {  // every pair's first fold
                    *S = b[c];
                    *C = 0ull;
                } else {
                    const f2 s = *S, y = sub2(b[c], *C), t = add2(s, y);
                    *C = sub2(sub2(t, s), y);
                    *S = t;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 2; k++) {
            float t[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                float lo, hi;
                upk(a[c][k], lo, hi);
                t[c] = __fadd_rn(lo, hi);
                kahan_add(w.ks[k][c], w.kc[k][c], t[c]);
            }
            w.s2[k] = fmaf(t[0], t[0], fmaf(t[1], t[1], fmaf(t[2], t[2], w.s2[k])));
        }
        while (close) {
            const int bit = __ffs(close) - 1;
            close &= close - 1u;
            const int i = i0 + 2 * lane + ((bit >> 1) & 1);
            const int j = j0 + 64 * sub + 2 * ((lane + s0 + (bit >> 2)) & 31) + (bit & 1);
            if (!sg_lists_pair(i, j, end)) continue;
            int at = atomicAdd(acc.n_close + i, 1);
            if (at < kCloseCap) acc.close[(size_t)i * kCloseCap + at] = j;
            if (!TWO) continue;
            at = atomicAdd(acc.n_close + j, 1);
            if (at < kCloseCap) acc.close[(size_t)j * kCloseCap + at] = i;
        }
        __syncwarp();  // the j-pair moves on to another lane
    }
}

// Near item: leaf it.leaf >> 1, its half it.leaf & 1, entries it.j0, it.j0 + it.n, ... of the
// leaf's near list.
__device__ __forceinline__ void near_warp(const float* __restrict__ c32, const SgFarItem& it,
                                          const SgCloud& cl, const LeafAcc& acc, int npad_total,
                                          const int* __restrict__ counts,
                                          const unsigned short* __restrict__ lists, int cap,
                                          int* flags, NearWarpShared& sh) {
    const int lane = threadIdx.x & 31;
    const size_t NP = (size_t)npad_total;
    const int leaf = it.leaf >> 1, i0 = cl.poff + leaf * SG_TILE + (it.leaf & 1) * (SG_TILE / 2);
    const int end = cl.poff + cl.n, pend = cl.poff + cl.npad;
    const int count = counts[cl.tile0 + leaf];
    if (i0 >= end || it.j0 >= count) return;
    if (leaf_wait_test(flags, (count - it.j0 + it.n - 1) / it.n)) return;
    const unsigned short* L = lists + (size_t)(cl.tile0 + leaf) * cap;
    NearSide w;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = i0 + 2 * lane + k;
        const bool in = i < pend;  // past a cloud's last leaf: far from everything, no charge
#pragma unroll
        for (int c = 0; c < 6; c++) {
            const float x = in ? c32[(c < 3 ? c : c + 1) * NP + i] : c < 3 ? sg_leaf_fill(true) : 0.f;
            w.x[c][k] = pk(x, x);
        }
        const float q = in ? c32[3 * NP + i] : 0.f;
        w.q[k] = pk(q, q);
        w.s2[k] = w.fmx[k] = 0.f;
#pragma unroll
        for (int c = 0; c < 3; c++) w.ks[k][c] = w.kc[k][c] = 0.f;
    }
    auto fetch = [&](int J, int slot) {
        const int j0 = cl.poff + J * SG_TILE, len = min(SG_TILE, pend - j0);
        float(*t)[SG_TILE] = sh.j[slot];
#pragma unroll
        for (int a = 0; a < 7; a++) {
            if (4 * lane < len)
                cp_async16(&t[a][4 * lane], c32 + a * NP + j0 + 4 * lane);
            else
#pragma unroll
                for (int q = 0; q < 4; q++) t[a][4 * lane + q] = a < 3 ? sg_leaf_fill(false) : 0.f;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int slot = 0;
    fetch(L[it.j0], 0);
    for (int e = it.j0; e < count; e += it.n) {
        const int J = L[e];
        if (e + it.n < count) {
            fetch(L[e + it.n], slot ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        const int j0 = cl.poff + J * SG_TILE;
        const bool noq = cl.quniform && j0 + SG_TILE <= end;
        if (J == leaf) {  // every ordered pair of the half, one side
            if (noq)
                near_leaf<true, false>(sh.j[slot], sh, w, cl.wc, i0, j0, end, acc);
            else
                near_leaf<false, false>(sh.j[slot], sh, w, cl.wc, i0, j0, end, acc);
        } else {
            if (noq)
                near_leaf<true, true>(sh.j[slot], sh, w, cl.wc, i0, j0, end, acc);
            else
                near_leaf<false, true>(sh.j[slot], sh, w, cl.wc, i0, j0, end, acc);
#pragma unroll 1
            for (int k = 0; k < 4; k++) {
                const int p = lane + 32 * k, jg = j0 + p;
                if (jg >= end) continue;
#pragma unroll
                for (int c = 0; c < 3; c++)
                    leaf_add(acc, NP, c, jg, -sh.S[c][p], sh.C[c][p], cl.far_fs);
                leaf_add(acc, NP, 3, jg, sh.s2[p], 0.f, cl.near_fs2);
                atomicMax(acc.fmx + jg, __float_as_int(sh.M[p]));
            }
        }
        __syncwarp();
        slot ^= 1;
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const int i = i0 + 2 * lane + k;
        if (i >= end) continue;
#pragma unroll
        for (int c = 0; c < 3; c++) leaf_add(acc, NP, c, i, w.ks[k][c], -w.kc[k][c], cl.far_fs);
        leaf_add(acc, NP, 3, i, w.s2[k], 0.f, cl.near_fs2);
        atomicMax(acc.fmx + i, __float_as_int(w.fmx[k]));
    }
}

// A near item or a far item per one-warp block: one launch, so that the far items fill the
// SMs as the near ones run out.  In blocks of four warps the slots of a block's finished
// warps waited for its longest item: 20,001 / 65,536 / 200,000 ions 160 / 1,302 / 11,682 us
// per call with four, 151 / 1,245 / 11,190 with one.
template <bool S2F>
__global__ void __launch_bounds__(32, 19) coulomb_leaf_kernel(
    const float* __restrict__ c32, const SgFarItem* __restrict__ near_items, int n_near,
    const SgFarItem* __restrict__ far_items, int n_far, const SgCloud* __restrict__ clouds,
    const SgCtrl* __restrict__ ctrl, LeafAcc acc, int npad_total, const float* __restrict__ bbox,
    const int* __restrict__ counts, const unsigned short* __restrict__ lists, int cap, int* flags) {
    sg_griddep_wait();
    typedef FarWarpShared<S2F> Far;
    constexpr size_t kWarp = sizeof(NearWarpShared) > sizeof(Far) ? sizeof(NearWarpShared) : sizeof(Far);
    __shared__ __align__(16) unsigned char raw[kWarp];
    const bool near = (int)blockIdx.x < n_near;
    const SgFarItem it = near ? near_items[blockIdx.x] : far_items[(int)blockIdx.x - n_near];
    if (ctrl != nullptr &&
        (ctrl[it.cloud].done || ctrl[it.cloud].hold || ctrl[it.cloud].status != SG_OK))
        return;
    if (near)
        near_warp(c32, it, clouds[it.cloud], acc, npad_total, counts, lists, cap, flags,
                  *reinterpret_cast<NearWarpShared*>(raw));
    else
        far_warp<S2F>(c32, it, clouds[it.cloud], acc, npad_total, bbox, flags,
                      *reinterpret_cast<Far*>(raw));
}

template <int NT, int IPT, int MINB, int STAGES, int TJ = SG_TILE, int FU = 0, bool S2F = true>
__global__ void __launch_bounds__(NT, MINB) coulomb_fp32c_sorted_kernel(const float* __restrict__ c32,
                                                            const double* __restrict__ c64,
                                                            const SgWorkItem* __restrict__ items,
                                                            const SgCloud* __restrict__ clouds,
                                                            const SgCtrl* __restrict__ ctrl,
                                                            double* __restrict__ part,
                                                            int npad_total, int* errword,
                                                            const float* __restrict__ bbox) {
    sg_griddep_wait();
    constexpr int T = TJ;  // j-tile: a multiple of the 128-ion leaves
    __shared__ __align__(128) float tile[STAGES][7][T];
    __shared__ __align__(8) uint64_t full[STAGES];
    __shared__ __align__(8) uint64_t never;  // the wait test's barrier
    __shared__ float corr[6][NT * IPT];

    const SgWorkItem it = items[blockIdx.x];
    const int wtest = errword ? errword[SG_FLAG_WAIT_TILE] : 0;
    if (ctrl != nullptr && (ctrl[it.cloud].done || ctrl[it.cloud].hold || ctrl[it.cloud].status != SG_OK)) return;
    const SgCloud& cl = clouds[it.cloud];
    const float wc = cl.wc;
    // uniform-charge clouds hold q_j / qscale (1 for ions, 0 for padding): tiles without
    // padding skip the charge product and the sums are scaled once at the end
    const double sc = cl.psc;
    const int j_real_end = cl.poff + cl.n;
    const int tid = threadIdx.x;
    const float* X = c32;
    const float* Y = c32 + npad_total;
    const float* Z = c32 + 2 * (size_t)npad_total;
    const float* XL = c32 + 4 * (size_t)npad_total;
    const float* YL = c32 + 5 * (size_t)npad_total;
    const float* ZL = c32 + 6 * (size_t)npad_total;

    // i-ions of this thread: it.i0 + tid + k*NT (clamped into the item for loads)
    int ipad[IPT];
    f2 xh[IPT], yh[IPT], zh[IPT], xl[IPT], yl[IPT], zl[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        int li = IPT * tid + k;  // contiguous: warp w holds the 128-ion tile w of the block
        int ii = it.i0 + (li < it.ni ? li : 0);
        ipad[k] = li < it.ni ? ii : -1;
        float a = X[ii], b = Y[ii], c = Z[ii], d = XL[ii], e = YL[ii], f = ZL[ii];
        xh[k] = pk(a, a);
        yh[k] = pk(b, b);
        zh[k] = pk(c, c);
        xl[k] = pk(d, d);
        yl[k] = pk(e, e);
        zl[k] = pk(f, f);
#pragma unroll
        for (int c = 0; c < 6; c++) corr[c][li] = 0.f;
    }
    float ks[IPT][3], kc[IPT][3], s2[IPT], s2f[IPT], fmx[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        s2[k] = 0.f;
        s2f[k] = 0.f;
        fmx[k] = 0.f;
#pragma unroll
        for (int c = 0; c < 3; c++) ks[k][c] = kc[k][c] = 0.f;
    }

    const int ntiles = (it.nj + T - 1) / T;
    bool ok = true;
    if (tid == 0) {
        for (int s = 0; s < STAGES; s++) mbar_init(&full[s], 1);
        mbar_init(&never, 1);
        fence_mbar_init();
    }
    __syncthreads();
    // prologue: fill the ring
    if (tid == 0) {
        for (int s = 0; s < STAGES && s < ntiles; s++) {
            const int j0 = it.j0 + s * T;
            const int len = min(T, it.j0 + it.nj - j0);
            const uint32_t bytes = (uint32_t)len * 4u;
            mbar_arrive_tx(&full[s], 7u * bytes);
            for (int a = 0; a < 7; a++)
                bulk_g2s(&tile[s][a][0], c32 + (size_t)a * npad_total + j0, bytes, &full[s]);
        }
    }

    const f2 tiny2 = pk(kTiny, kTiny);
    // bounds of this warp's 128 i-ions (a k-d tree leaf after sorting)
    float wbox[6];
    {
        // warps past the cloud's last ion read the last tile (their results are dropped)
        const int last = (cl.npad + 127) / 128 - 1;
        const int wt = cl.tile0 + min(last, (it.i0 - cl.poff) / 128 + (tid >> 5) * (32 * IPT) / 128);
        for (int q = 0; q < 6; q++) wbox[q] = bbox[8 * (size_t)wt + q];
    }
    const float dfar2 = cl.dfar * cl.dfar;
    // FP32 running sums restart every 32 j-ions (16 for small clouds): in k-d order the
    // terms of a tile point the same way, and a 128-term running sum would carry several
    // times the rounding error of the summands.
    const int flush_len = (cl.npad <= 2048) ? 16 : 32;
    for (int t = 0; t < ntiles; t++) {
        const int s = t % STAGES;
        const uint32_t parity = (uint32_t)((t / STAGES) & 1);
        const int j0 = it.j0 + t * T;
        const int len = min(T, it.j0 + it.nj - j0);
        bool arrived = mbar_wait(&full[s], parity);
        if (t + 1 == wtest) arrived = wait_test(&never, errword) && arrived;
        if (!__syncthreads_and(arrived)) {  // block-uniform decision
            ok = false;
            if (tid == 0) {
                atomicExch(errword, SG_TIMEOUT);
                // drain the copies still in flight (tiles t .. t+STAGES-1), bounded
                for (int u = t; u < ntiles && u < t + STAGES; u++)
                    (void)mbar_wait(&full[u % STAGES], (uint32_t)((u / STAGES) & 1));
            }
            __syncthreads();
            break;
        }

        float y3max[IPT];
#pragma unroll
        for (int k = 0; k < IPT; k++) y3max[k] = 0.f;
        const float* tx = tile[s][0];
        const float* ty = tile[s][1];
        const float* tz = tile[s][2];
        const float* tq = tile[s][3];
        const float* txl = tile[s][4];
        const float* tyl = tile[s][5];
        const float* tzl = tile[s][6];
        // Per 128-ion leaf of the tile: far from this block's leaf, or not.  The leaf holding
        // this block's own ions takes the variant that keeps the self pair (dx = 0,
        // contributes nothing) out of the close-pair flag.
        // no padding ions in this tile: their normalized charge 0 is the only one not 1
        const bool noq = cl.quniform && j0 + len <= j_real_end;
        for (int sub = 0; sub < len; sub += SG_TILE) {
            const int send = min(len, sub + SG_TILE);
            const int sj0 = j0 + sub;
            const bool diag = (sj0 < it.i0 + it.ni) && (j0 + send > it.i0);
            float jbox[6];
            const int jt = cl.tile0 + (sj0 - cl.poff) / 128;
            for (int q = 0; q < 6; q++) jbox[q] = bbox[8 * (size_t)jt + q];
            const bool far = !diag && box_dist2(wbox, jbox) > dfar2;  // uniform per warp
            // Each 32-ion FP32 partial goes straight into the compensated accumulators.
            // (Adding the partials of a tile first, in FP32, saved 3 % of the kernel time but
            // raised the worst ion's error on the 65,536-ion cloud from 5.7e-7 to 8.8e-7.)
            for (int jb = sub; jb < send; jb += flush_len) {
                const int je = min(send, jb + flush_len);
                f2 ax[IPT], ay[IPT], az[IPT];
#pragma unroll
                for (int k = 0; k < IPT; k++) ax[k] = ay[k] = az[k] = 0ull;
                if (far && noq)
                    tile_pairs_far<IPT, true, FU>(tx, ty, tz, tq, jb, je, xh, yh, zh, tiny2, ax, ay,
                                                  az);
                else if (far)
                    tile_pairs_far<IPT, false, FU>(tx, ty, tz, tq, jb, je, xh, yh, zh, tiny2, ax, ay,
                                                   az);
                else if (!diag && noq)
                    tile_pairs<IPT, false, true>(tx, ty, tz, tq, txl, tyl, tzl, jb, je, j0, ipad,
                                                 xh, yh, zh, xl, yl, zl, tiny2, wc, ax, ay, az,
                                                 y3max);
                else if (!diag)
                    tile_pairs<IPT, false>(tx, ty, tz, tq, txl, tyl, tzl, jb, je, j0, ipad, xh, yh,
                                           zh, xl, yl, zl, tiny2, wc, ax, ay, az, y3max);
                else
                    tile_pairs<IPT, true>(tx, ty, tz, tq, txl, tyl, tzl, jb, je, j0, ipad, xh, yh,
                                          zh, xl, yl, zl, tiny2, wc, ax, ay, az, y3max);
                fold_partials<IPT, S2F>(ax, ay, az, ks, kc, s2, s2f, !far);
                if (!far)
                    fold_close<IPT>(tile[s], jb, je, j0, ipad, xh, yh, zh, xl, yl, zl, wc, sc,
                                    c64, npad_total, corr, y3max, fmx,
                                    [tid](int k) { return IPT * tid + k; });
            }
        }
        __syncthreads();  // every thread is done with ring slot s
        if (tid == 0 && t + STAGES < ntiles) {
            fence_proxy_async();
            const int jn = it.j0 + (t + STAGES) * T;
            const int ln = min(T, it.j0 + it.nj - jn);
            const uint32_t bytes = (uint32_t)ln * 4u;
            mbar_arrive_tx(&full[s], 7u * bytes);
            for (int a = 0; a < 7; a++)
                bulk_g2s(&tile[s][a][0], c32 + (size_t)a * npad_total + jn, bytes, &full[s]);
        }
    }
    if (!ok) return;
    const size_t NP = (size_t)npad_total;
    float* P = reinterpret_cast<float*>(part) + (size_t)it.slot * SG_PART_F32 * NP;
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        if (ipad[k] < 0) continue;
        store_partial(P, NP, ipad[k], ks[k], kc[k], corr, IPT * tid + k, s2[k], fmx[k]);
        if (S2F) P[7 * NP + ipad[k]] = s2f[k];
    }
}

// ---------------------------------------------------------------------------
// FP64 kernels (plain form).  c64 = 4 double arrays (x, y, z, q) in SI units.
// ---------------------------------------------------------------------------

// Every unordered pair once (fp64_pairs.cuh): a work item is one 128-ion i-block against
// nj j-ions, or a part of a pair of 32-ion tiles (tile_pair).
__global__ void __launch_bounds__(SG_SYM_IB) coulomb_fp64_sym_kernel(
    const double* __restrict__ c64, const SgWorkItem* __restrict__ items,
    const SgCloud* __restrict__ clouds, const SgCtrl* __restrict__ ctrl,
    double* __restrict__ part, int npad_total) {
    sg_griddep_wait();
    __shared__ Fp64SymShared sh;
    const SgWorkItem it = items[blockIdx.x];
    if (ctrl != nullptr && (ctrl[it.cloud].done || ctrl[it.cloud].hold || ctrl[it.cloud].status != SG_OK)) return;
    const SgCloud& cl = clouds[it.cloud];
    const size_t NP = (size_t)npad_total;
    const double* c = c64 + cl.poff;
    const auto ld = [c, NP](int a, int k) { return c[a * NP + k]; };
    double *pi = part + (size_t)it.slot * 3 * NP + cl.poff, *pj = part + (size_t)it.jslot * 3 * NP + cl.poff;
    if (it.tile_pair)
        fp64_sym_tile_block<false>(ld, cl.n, it.i0 - cl.poff, it.j0 - cl.poff, it.tile_pair & 255,
                                   it.tile_pair >> 8, cl.quniform != 0, cl.qscale, 0.0, pi, pj, NP, sh);
    else
        fp64_sym_block<false>(ld, cl.n, cl.npad, it.i0 - cl.poff, it.j0 - cl.poff, it.nj,
                              cl.quniform != 0, cl.qscale, 0.0, pi, pj, NP, sh);
}

// Every ordered pair, for clouds whose symmetric partial sums would not fit
// (SG_SYM_MAX_IONS).
template <int NT, int IPT>
__global__ void __launch_bounds__(NT) coulomb_fp64_kernel(const double* __restrict__ c64,
                                                           const SgWorkItem* __restrict__ items,
                                                           const SgCtrl* __restrict__ ctrl,
                                                           double* __restrict__ part,
                                                           int npad_total) {
    sg_griddep_wait();
    constexpr int T = NT;
    __shared__ double tile[4][T];
    const SgWorkItem it = items[blockIdx.x];
    if (ctrl != nullptr && (ctrl[it.cloud].done || ctrl[it.cloud].hold || ctrl[it.cloud].status != SG_OK)) return;
    const int tid = threadIdx.x;
    const double* X = c64;
    const double* Y = c64 + npad_total;
    const double* Z = c64 + 2 * (size_t)npad_total;
    const double* Q = c64 + 3 * (size_t)npad_total;
    int ipad[IPT];
    double xi[IPT], yi[IPT], zi[IPT], ax[IPT], ay[IPT], az[IPT];
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        const int li = tid + k * NT;
        const int ii = it.i0 + (li < it.ni ? li : 0);
        ipad[k] = li < it.ni ? ii : -1;
        xi[k] = X[ii];
        yi[k] = Y[ii];
        zi[k] = Z[ii];
        ax[k] = ay[k] = az[k] = 0.0;
    }
    for (int j0 = it.j0; j0 < it.j0 + it.nj; j0 += T) {
        const int len = min(T, it.j0 + it.nj - j0);
        __syncthreads();
        if (tid < len) {
            tile[0][tid] = X[j0 + tid];
            tile[1][tid] = Y[j0 + tid];
            tile[2][tid] = Z[j0 + tid];
            tile[3][tid] = Q[j0 + tid];
        }
        __syncthreads();
        for (int jj = 0; jj < len; jj++) {
            const double xj = tile[0][jj], yj = tile[1][jj], zj = tile[2][jj], qj = tile[3][jj];
            const int jg = j0 + jj;
#pragma unroll
            for (int k = 0; k < IPT; k++) {
                const double rx = xi[k] - xj, ry = yi[k] - yj, rz = zi[k] - zj;
                double w = qj * inv_r3_fp64(rx * rx + ry * ry + rz * rz);
                w = (jg == ipad[k]) ? 0.0 : w;
                ax[k] = fma(w, rx, ax[k]);
                ay[k] = fma(w, ry, ay[k]);
                az[k] = fma(w, rz, az[k]);
            }
        }
    }
    double* P = part + (size_t)it.slot * 3 * npad_total;
#pragma unroll
    for (int k = 0; k < IPT; k++) {
        if (ipad[k] < 0) continue;
        P[ipad[k]] = ax[k];
        P[npad_total + ipad[k]] = ay[k];
        P[2 * (size_t)npad_total + ipad[k]] = az[k];
    }
}


// ---------------------------------------------------------------------------
// Sum of the partial-sum slots of every ion into out[3][N] (SI, m^-2).
//
// FP32c only: the conditioning test.  sqrt(s2) estimates sqrt(sum_j |f_ij|^2) of the
// FP32 terms; the rounding of those terms is random, so the error of P_i is about
// 2.5e-7 * sqrt(s2).  An ion whose FP32 terms cancel strongly (sqrt(s2) > 1.5 |P_i|,
// e.g. near the centre of a cloud, or a single term above 1.5 |P_i|) gets its whole row
// re-evaluated in FP64 (fixup_row), spread over work units for a large cloud.
//
// k-d ordered shapes: the far tile pairs were summed from the high FP32 parts only, an
// error of ~1e-7 per pair that averages out unless the ion's net force is small next to
// its far terms (the centre of a uniform cloud).  Its size tracks sqrt(s2f), the far
// tiles' conditioning estimate: on the 1M-ion spheroid and the 65,536-ion Gaussian cloud
// (numpy model of the kernel's arithmetic) the relative error of P_i stayed below
// 1.3e-6 sqrt(s2f)/|P_i|, the constant growing with the ion density.  An ion with
// s2f > SgCloud::kfar2 |P_i|^2 gets the exact first-order correction of every far pair
// term (fixup_ion), which leaves it at the near tiles' FP32 accuracy.
// ---------------------------------------------------------------------------
// kinds of fix-up of a flagged ion
constexpr int kFixNear = 1, kFixFar = 2;

// Blocks of the fix-up kernel, each with every grid-th work unit: three per SM are resident,
// and the more there are the better the units even out (512 clouds of 500 to 1,000 ions, us
// per attempt: 512 blocks 2,938, 2,048 2,768), but they all have to start (167 of <= 300: 335,
// 339).
inline int fixup_blocks(int n_total) { return std::min(2048, std::max(512, n_total / 128)); }
// batches up to this many ions fix their flagged ions inside the reduction's blocks
constexpr int kInBlockFixupMax = SG_FINISH_MAX_IONS;

// Error-free difference: a - b = s + err exactly, s = fl(a - b) (Knuth's two-sum).
__device__ __forceinline__ float two_diff_err(float a, float b, float s) {
    const float bv = __fsub_rn(s, a);
    const float av = __fsub_rn(s, bv);
    return __fadd_rn(__fsub_rn(a, av), __fsub_rn(-b, bv));
}

template <int NTH>
struct FixupShared {
    double wsum[NTH / 32][3];
};

struct Corr3 {
    double x, y, z;
};

// Block-wide sum of one value per thread and component; the result is thread 0's.
template <int NTH>
__device__ Corr3 block_sum3(double ax, double ay, double az, FixupShared<NTH>& sh) {
    static_assert(NTH == 256, "eight warps");
    const int li = threadIdx.x, warp = li >> 5, lane = li & 31;
    double v = warp_sum3(ax, ay, az);
    if (lane == 0) sh.wsum[warp][0] = v;
    if (lane == 16) sh.wsum[warp][1] = v;
    if (lane == 8) sh.wsum[warp][2] = v;
    __syncthreads();
    Corr3 r{0.0, 0.0, 0.0};
    if (warp == 0) {
        v = lane < 24 ? sh.wsum[lane & 7][lane >> 3] : 0.0;
        for (int o = 4; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o, 8);
        r.x = __shfl_sync(0xffffffffu, v, 0);
        r.y = __shfl_sync(0xffffffffu, v, 8);
        r.z = __shfl_sync(0xffffffffu, v, 16);
    }
    __syncthreads();
    return r;
}

// Row of a flagged ion in FP64, chunk c of nch (contiguous j-ranges of the cloud's padded
// range; the padding ions carry no charge), by the whole block of NTH threads: the sum
// of q_j (x_i - x_j) / r^3 over the chunk, from the SI coordinates (thread 0's result).
// Re-evaluating only the dominant pairs is not enough: an ion whose FP32 terms cancel
// keeps the rounding of every addition made while a dominant term was in its partial sum
// (~1e-7 |f_max|), so the flagged ion's sum is replaced by its exact row.
template <int NTH>
__device__ Corr3 fixup_row(const SgCloud& cl, int i, const double* __restrict__ c64,
                           int npad_total, int c, int nch, FixupShared<NTH>& sh) {
    const size_t NP = (size_t)npad_total;
    const int igk = cl.poff + (i - cl.off);
    const double xi = c64[igk], yi = c64[NP + igk], zi = c64[2 * NP + igk];
    const int len = (cl.npad + nch - 1) / nch;
    const int j0 = c * len, j1 = min(cl.npad, j0 + len);
    double ax = 0.0, ay = 0.0, az = 0.0;
    // independent pairs in flight: each one's 1/r is a chain of dependent FP64 operations
#pragma unroll 4
    for (int j = j0 + (int)threadIdx.x; j < j1; j += NTH) {
        const int jg = cl.poff + j;
        if (jg == igk) continue;
        const double rx = xi - c64[jg], ry = yi - c64[NP + jg], rz = zi - c64[2 * NP + jg];
        const double wq = c64[3 * NP + jg] * inv_r3_fp64(rx * rx + ry * ry + rz * rz);
        ax = fma(wq, rx, ax);
        ay = fma(wq, ry, ay);
        az = fma(wq, rz, az);
    }
    return block_sum3<NTH>(ax, ay, az, sh);
}

// Far fix-up of ion i, chunk c of nch: the warps take the 128-ion tiles t = (c + m nch) W
// + w (W warps per block) that the Coulomb kernel treated as far from the ion's own
// tile, and each pair term f(u) = q u / |u|^3 of the hi-part difference u = fl(hi_j - hi_i)
// gets
//     delta = q y3 (D - 3 y^2 (u.D) u),   D = (lo_j - lo_i) + (hi_j - hi_i - u),
// the exact first-order change to the float-float difference (|D|/|u| ~ 1e-7, so the
// second order is far below FP32 rounding); y and y3 are formed as the kernel formed
// them.  Summed in FP32 per thread (the terms are small), in FP64 across the block;
// returns the correction of P_i (SI, thread 0).
template <int NTH>
__device__ Corr3 fixup_far(const SgCloud& cl, int i, const float* __restrict__ c32,
                           int npad_total, const float* __restrict__ bbox, int c, int nch,
                           FixupShared<NTH>& sh) {
    constexpr int W = NTH / 32;
    const int li = threadIdx.x;
    const int warp = li >> 5, lane = li & 31;
    const size_t NP = (size_t)npad_total;
    const int igk = cl.poff + (i - cl.off);
    const float xih = c32[igk], yih = c32[NP + igk], zih = c32[2 * NP + igk];
    const float xil = c32[4 * NP + igk], yil = c32[5 * NP + igk], zil = c32[6 * NP + igk];
    const int nt = (cl.npad + 127) / 128, itile = (igk - cl.poff) / 128;
    const float* ibox = bbox + 8 * (size_t)(cl.tile0 + itile);
    const float dfar2 = cl.dfar * cl.dfar;
    float fx = 0.f, fy = 0.f, fz = 0.f;
    for (int t = c * W + warp; t < nt; t += nch * W) {
        // the Coulomb kernel's far test for this (leaf, tile) pair, uniform per warp
        if (t == itile || !(box_dist2(ibox, bbox + 8 * (size_t)(cl.tile0 + t)) > dfar2)) continue;
        for (int jj = lane; jj < 128; jj += 32) {
            const int j = t * 128 + jj;
            if (j >= cl.npad) break;
            const int jg = cl.poff + j;
            const float xjh = c32[jg], yjh = c32[NP + jg], zjh = c32[2 * NP + jg];
            const float q = c32[3 * NP + jg];
            const float ux = __fsub_rn(xjh, xih), uy = __fsub_rn(yjh, yih), uz = __fsub_rn(zjh, zih);
            float r2 = __fmaf_rn(ux, ux, kTiny);
            r2 = __fmaf_rn(uy, uy, r2);
            r2 = __fmaf_rn(uz, uz, r2);
            const float y = rsqrt_approx(r2);
            const float y3 = __fmul_rn(__fmul_rn(y, y), y);
            const float dx = __fadd_rn(__fsub_rn(c32[4 * NP + jg], xil), two_diff_err(xjh, xih, ux));
            const float dy = __fadd_rn(__fsub_rn(c32[5 * NP + jg], yil), two_diff_err(yjh, yih, uy));
            const float dz = __fadd_rn(__fsub_rn(c32[6 * NP + jg], zil), two_diff_err(zjh, zih, uz));
            const float ud = fmaf(ux, dx, fmaf(uy, dy, uz * dz));
            const float s3 = 3.f * y * y * ud;
            const float qy3 = q * y3;
            fx = fmaf(qy3, fmaf(-s3, ux, dx), fx);
            fy = fmaf(qy3, fmaf(-s3, uy, dy), fy);
            fz = fmaf(qy3, fmaf(-s3, uz, dz), fz);
        }
    }
    Corr3 r = block_sum3<NTH>(fx, fy, fz, sh);
    // frame sums of q u / r^3 -> P (SI), as the kernel's epilogue scales them
    const double sc = -(cl.invL * cl.invL) * cl.qscale;
    r.x *= sc;
    r.y *= sc;
    r.z *= sc;
    return r;
}

// Whole fix-up of one flagged ion by one block: kFixNear replaces its sum by the exact
// FP64 row (which also covers its far terms); kFixFar alone adds the far correction
// (k-d ordered shapes).  Written to out by thread 0.  The j-ions are taken in a fixed
// order, so the result does not depend on which block runs it or when.
template <int NTH>
__device__ void fixup_ion(const SgCloud& cl, int i, int kind, const float* __restrict__ c32,
                          const double* __restrict__ c64, int npad_total,
                          double* __restrict__ out, int n_total, const float* __restrict__ bbox,
                          FixupShared<NTH>& sh) {
    if (kind & kFixNear) {
        const Corr3 r = fixup_row<NTH>(cl, i, c64, npad_total, 0, 1, sh);
        if (threadIdx.x == 0) {
            out[i] = r.x;
            out[(size_t)n_total + i] = r.y;
            out[2 * (size_t)n_total + i] = r.z;
        }
    } else if (bbox != nullptr) {
        const Corr3 r = fixup_far<NTH>(cl, i, c32, npad_total, bbox, 0, 1, sh);
        if (threadIdx.x == 0) {
            out[i] += r.x;
            out[(size_t)n_total + i] += r.y;
            out[2 * (size_t)n_total + i] += r.z;
        }
    }
    __syncthreads();
}

// Shape 17's accumulators (sum null for the other shapes) and the s2f of the last call that
// estimated it.
struct LeafSums {
    LeafAcc acc;
    float* s2f;
    int estimate;
};

// A fixed-point sum in units of 1 / fs as a float-float, by 24-bit pieces.
__device__ __forceinline__ ff far_value(long long v, float fs) {
    const float inv = 1.0f / fs;  // a power of two
    const float h = (float)(int)(v >> 30);            // up to 2^25 or so: may round
    const long long r = v - ((long long)(int)h << 30);
    const int r1 = (int)(r >> 8);                      // |r| <= 2^31
    const float m = (float)(r1 >> 8), l = (float)(int)(r - ((long long)(r1 >> 8) << 16));
    const ff a = ff_two_sum(__fmul_rn(h, 1073741824.0f * inv), __fmul_rn(m, 65536.0f * inv));
    return ff_add(a, {__fmul_rn(l, inv), 0.f});
}

// The listed close pairs of ion ig (m of them, at most kCloseCap): the exact term minus the
// capped FP32 one of each, in the order of the partners (the lists fill in any order);
// returns the strongest capped term.
__device__ float close_list_terms(const SgCloud& cl, int ig, int m, const int* __restrict__ list,
                                  const float* __restrict__ c32, const double* __restrict__ c64,
                                  size_t NP, ff& px, ff& py, ff& pz) {
    const float xih = c32[ig], yih = c32[NP + ig], zih = c32[2 * NP + ig];
    const float xil = c32[4 * NP + ig], yil = c32[5 * NP + ig], zil = c32[6 * NP + ig];
    float fmx = 0.f;
    int done = -1;
    for (int k = 0; k < m; k++) {
        int j = 0x7fffffff;
        for (int q = 0; q < m; q++) {
            const int l = list[q];
            if (l > done && l < j) j = l;
        }
        done = j;
        const float xjh = c32[j], yjh = c32[NP + j], zjh = c32[2 * NP + j], q = c32[3 * NP + j];
        const float xjl = c32[4 * NP + j], yjl = c32[5 * NP + j], zjl = c32[6 * NP + j];
        if (q == 0.f) continue;
        const PairF pr = pair_f32(xjh, yjh, zjh, xjl, yjl, zjl, xih, yih, zih, xil, yil, zil);
        fmx = fmaxf(fmx, capped_term_y3(pr.y3, cl.wc));
        const float wf = __fmul_rn(q, cl.wc);
        ff dx, dy, dz;
        if (!very_close(pr.y3, xih, yih, zih)) {
            close_term_ff(ff_diff(xjh, xjl, xih, xil), ff_diff(yjh, yjl, yih, yil),
                          ff_diff(zjh, zjl, zih, zil), q, wf, pr, dx, dy, dz);
        } else {
            const double rx = c64[ig] - c64[j], ry = c64[NP + ig] - c64[NP + j],
                         rz = c64[2 * NP + ig] - c64[2 * NP + j];
            const double w = c64[3 * NP + j] * inv_r3_fp64(rx * rx + ry * ry + rz * rz) / cl.psc;
            const double c0 = w * rx - (double)wf * (double)pr.dx,
                         c1 = w * ry - (double)wf * (double)pr.dy,
                         c2 = w * rz - (double)wf * (double)pr.dz;
            dx.h = (float)c0;
            dx.l = (float)(c0 - (double)dx.h);
            dy.h = (float)c1;
            dy.l = (float)(c1 - (double)dy.h);
            dz.h = (float)c2;
            dz.l = (float)(c2 - (double)dz.h);
        }
        px = ff_add(px, dx);
        py = ff_add(py, dy);
        pz = ff_add(pz, dz);
    }
    return fmx;
}

// The G threads of a row (thread li sums slots li / R, li / R + G, ... of row li % R, R
// rows in the block): their parts combined in a fixed order by the row's first thread.
struct SlotShared {
    float v[SG_ROWS][8];  // FP32c: hi x, y, z, lo x, y, z, s2, s2f
};
struct SlotShared64 {
    double v[SG_ROWS][3];
};

// Sums the partial-sum slots of each ion into out[3][N] (SI, m^-2), R rows per block with
// SG_ROWS / R threads each.
//
// FP32c: the slots hold float-float sums in frame units (store_partial); they are added
// in float-float and converted once.  An ion whose near terms cancel strongly
// (sqrt(s2) > 1.5 |P|, > |P| in clouds of up to SG_SMALL_ROW ions, batches of shape 17:
// sum_kappa in capi.cu) or whose far terms are
// large next to |P| (s2f > SgCloud::kfar2 |P|^2) is fixed up (fixup_ion): INBLOCK, by this
// block right away (small batches, where a second launch costs more than the work);
// otherwise its work units are put on the list of coulomb_fixup_kernel (ion index; cloud |
// kind << 28; unit and their count; first unit), or the ion whole once that is full.
//
// Latency-bound for small clouds: an FP64 addition takes a warp 64 cycles, so one thread
// per row over 32 slots of five FP64 values spent ~5 us on additions alone.  Batches of
// up to kInBlockFixupMax ions, and those with more than 24 slots, take 16 rows a block, 16
// threads each; the others 64 rows of 4 threads.
template <bool F32, bool INBLOCK>
__global__ void __launch_bounds__(SG_ROWS) coulomb_reduce_kernel(
    const SgRowBlock* __restrict__ rows, const SgCloud* __restrict__ clouds,
    const SgCtrl* __restrict__ ctrl, const double* __restrict__ part, int npad_total,
    double* __restrict__ out, int n_total, int* __restrict__ counters,
    int* __restrict__ fix_list, const float* __restrict__ c32,
    const double* __restrict__ c64, const float* __restrict__ bbox, float* __restrict__ risk,
    int* __restrict__ ran, const SgCheck* __restrict__ chk, int split, LeafSums leaf) {
    sg_griddep_wait();
    // this block's share of its row block: cap / split rows; leaf sums have no slots to
    // share, so the first block of a leaf cloud's row block takes all of it, a thread per row
    SgRowBlock rb = rows[blockIdx.x / split];
    if (F32 && !INBLOCK && clouds[rb.cloud].leafs) {
        if (blockIdx.x % split) return;
        split = 1;
    }
    const int R = rb.cap / split, G = SG_ROWS / R;  // powers of two
    const int first = (int)(blockIdx.x % split) * R;
    rb.i0 += first;
    rb.n = min(rb.n - first, R);
    if (rb.n <= 0) return;
    if (ctrl != nullptr &&
        (ctrl[rb.cloud].done || ctrl[rb.cloud].hold || ctrl[rb.cloud].status != SG_OK))
        return;
    const SgCloud& cl = clouds[rb.cloud];
    if (!(cl.fp.flags & SG_F_COULOMB)) return;
    const int li = threadIdx.x;
    const int row = li & (R - 1), g = li / R;
    const size_t NP = (size_t)npad_total;
    const int ig = cl.poff + (rb.i0 - cl.off) + row;  // padded index (row < rb.n)
    int kind = 0;
    const int i = rb.i0 + li;
    if constexpr (F32) {
        __shared__ SlotShared ss;
        ff px{0.f, 0.f}, py{0.f, 0.f}, pz{0.f, 0.f};
        float s2 = 0.f, s2f = 0.f;
        if (row < rb.n) {
            const float* P = reinterpret_cast<const float*>(part) + ig;
#pragma unroll 4
            for (int sl = g; sl < cl.nslots; sl += G) {
                const float* Q = P + (size_t)sl * SG_PART_F32 * NP;
                px = ff_add(px, {Q[0], Q[3 * NP]});
                py = ff_add(py, {Q[NP], Q[4 * NP]});
                pz = ff_add(pz, {Q[2 * NP], Q[5 * NP]});
                s2 += Q[6 * NP];
                s2f += Q[7 * NP];
            }
        }
        if (G > 1) {
            float* v = ss.v[li];
            v[0] = px.h;
            v[1] = py.h;
            v[2] = pz.h;
            v[3] = px.l;
            v[4] = py.l;
            v[5] = pz.l;
            v[6] = s2;
            v[7] = s2f;
            __syncthreads();
        }
        if (li < rb.n) {
            for (int q = 1; q < G; q++) {
                const float* v = ss.v[li + q * R];
                px = ff_add(px, {v[0], v[3]});
                py = ff_add(py, {v[1], v[4]});
                pz = ff_add(pz, {v[2], v[5]});
                s2 += v[6];
                s2f += v[7];
            }
            const double sc = cl.psc;
            bool many = false;
            if (cl.leafs) {
                // the leaf pairs' sums: taken and cleared for the next call
                unsigned long long* A = leaf.acc.sum + ig;
                px = far_value((long long)A[0], cl.far_fs);
                py = far_value((long long)A[NP], cl.far_fs);
                pz = far_value((long long)A[2 * NP], cl.far_fs);
                s2 = far_value((long long)A[3 * NP], cl.near_fs2).h;
                A[0] = A[NP] = A[2 * NP] = A[3 * NP] = 0ull;
                if (leaf.estimate) {
                    leaf.s2f[ig] = far_value((long long)A[4 * NP], cl.far_fs2).h;
                    A[4 * NP] = 0ull;
                }
                s2f = leaf.s2f[ig];
                const int fm = leaf.acc.fmx[ig], m = leaf.acc.n_close[ig];
                leaf.acc.fmx[ig] = 0;
                leaf.acc.n_close[ig] = 0;
                float fmx = __int_as_float(fm);
                many = m > kCloseCap;
                if (m > 0)
                    fmx = fmaxf(fmx, close_list_terms(cl, ig, min(m, kCloseCap),
                                                      leaf.acc.close + (size_t)ig * kCloseCap, c32,
                                                      c64, NP, px, py, pz));
                s2 = conditioning_s2(s2, fmx);
                if (fm == kPoison) px = py = pz = {__int_as_float(kPoison), 0.f};
            }
            out[i] = sc * ((double)px.h + (double)px.l);
            out[(size_t)n_total + i] = sc * ((double)py.h + (double)py.l);
            out[2 * (size_t)n_total + i] = sc * ((double)pz.h + (double)pz.l);
            // |P|^2 in frame units (a threshold test: FP32)
            const float pf2 = fmaf(px.h, px.h, fmaf(py.h, py.h, pz.h * pz.h));
            // the far threshold: the prior of the frame set-up, or the measured one
            const float kf2 = chk ? fminf(cl.kfar2, chk[rb.cloud].kfar2) : cl.kfar2;
            const float kap2 = cl.kappa2;
            kind = (many || s2 > kap2 * pf2 ? kFixNear : 0) | (s2f > kf2 * pf2 ? kFixFar : 0);
            if (risk != nullptr) {
                const float pf = sqrtf(pf2);
                risk[i] = kind ? -1.f : sqrtf(s2f) / pf;
                risk[(size_t)n_total + i] = kind ? -1.f : sqrtf(s2) / pf;
            }
        }
    } else {
        __shared__ SlotShared64 ss;
        double px = 0.0, py = 0.0, pz = 0.0;
        if (row < rb.n) {
            const int ns = cl.sym_k ? sg_sym_slots(cl, ig - cl.poff) : cl.nslots;
            const double* P = part + ig;
#pragma unroll 4
            for (int sl = g; sl < ns; sl += G) {
                const double* Q = P + (size_t)sl * 3 * NP;
                px += Q[0];
                py += Q[NP];
                pz += Q[2 * NP];
            }
        }
        // pairwise over the G parts: log2(G) dependent FP64 additions
        for (int h = G / 2; h > 0; h /= 2) {
            if (g >= h && g < 2 * h) {
                ss.v[li][0] = px;
                ss.v[li][1] = py;
                ss.v[li][2] = pz;
            }
            __syncthreads();
            if (g < h) {
                px += ss.v[li + h * R][0];
                py += ss.v[li + h * R][1];
                pz += ss.v[li + h * R][2];
            }
        }
        if (li < rb.n) {
            out[i] = px;
            out[(size_t)n_total + i] = py;
            out[2 * (size_t)n_total + i] = pz;
        }
    }
    if (F32 && ran != nullptr && li == 0) ran[rb.cloud] = 1;
    if (!F32) return;
    if (!INBLOCK) {
        if (kind) {
            // the ion's work units; past the list's end, the ion whole
            const int U = sg_fix_units(cl.npad), at = atomicAdd(fix_list, U);
            int4* units = reinterpret_cast<int4*>(fix_list + 4);
            const int ck = rb.cloud | kind << 28;
            const bool fits = at + U <= SG_FIX_CAP;
            for (int c = 0; c < U && at + c < SG_FIX_CAP; c++)
                units[at + c] = make_int4(fits ? i : -1, ck, c | U << 16, at);
            if (!fits) {
                int* whole = fix_list + 4 + 4 * SG_FIX_CAP + 2 * (size_t)atomicAdd(fix_list + 1, 1);
                whole[0] = i;
                whole[1] = ck;
            }
            if (counters != nullptr) atomicAdd(counters, 1);
        }
        return;
    }
    __shared__ FixupShared<SG_ROWS> sh;
    __shared__ int nflag;
    __shared__ int flist[SG_ROWS];
    __shared__ int fkind[SG_ROWS];
    if (li == 0) nflag = 0;
    __syncthreads();
    if (kind) {
        const int at = atomicAdd(&nflag, 1);
        flist[at] = i;
        fkind[at] = kind;
        if (counters != nullptr) atomicAdd(counters, 1);
    }
    __syncthreads();  // also orders this block's writes of out before the corrections
    const int nf = nflag;
    for (int k = 0; k < nf; k++)
        fixup_ion(cl, flist[k], fkind[k], c32, c64, npad_total, out, n_total, bbox, sh);
}

// The flagged ions of a whole batch: re-evaluated rows (kFixNear) and far corrections, in
// units of ~1,024 j-ions (sg_fix_units).  Each unit of an ion leaves its part in fix_part and
// the last of them (counted in fix_done) adds the parts in unit order -- writing the row,
// or adding the far correction -- so the result does not depend on the order the units
// ran in.  Ions that found the list full are one unit each.  FP64-bound: rows of up to
// 4,096 ions as units of their own left the device waiting for the longest (128 clouds of
// 64 to 8,192 ions, 596 rows a call: 84 us, 68 so).
constexpr int kFixupThreads = 256;
__global__ void __launch_bounds__(kFixupThreads, 3) coulomb_fixup_kernel(
    const SgCloud* __restrict__ clouds, const float* __restrict__ c32,
    const double* __restrict__ c64, int npad_total, double* __restrict__ out, int n_total,
    const int* __restrict__ fix_list, const float* __restrict__ bbox,
    double* __restrict__ fix_part, int* __restrict__ fix_done) {
    sg_griddep_wait();
    __shared__ FixupShared<kFixupThreads> sh;
    __shared__ int last;
    const int units = min(fix_list[0], SG_FIX_CAP), whole = fix_list[1];
    const int4* list = reinterpret_cast<const int4*>(fix_list + 4);
    for (int u = blockIdx.x; u < units + whole; u += gridDim.x) {
        if (u >= units) {
            const int* w = fix_list + 4 + 4 * SG_FIX_CAP + 2 * (size_t)(u - units);
            fixup_ion<kFixupThreads>(clouds[w[1] & 0x0FFFFFFF], w[0], w[1] >> 28, c32, c64,
                                     npad_total, out, n_total, bbox, sh);
            continue;
        }
        const int4 it = list[u];
        const int i = it.x, c = it.z & 0xffff, U = it.z >> 16, base = it.w;
        if (i < 0) continue;  // of an ion that did not fit
        const SgCloud& cl = clouds[it.y & 0x0FFFFFFF];
        const bool row = (it.y >> 28) & kFixNear;
        Corr3 r{0.0, 0.0, 0.0};
        if (row)
            r = fixup_row<kFixupThreads>(cl, i, c64, npad_total, c, U, sh);
        else if (bbox != nullptr)
            r = fixup_far<kFixupThreads>(cl, i, c32, npad_total, bbox, c, U, sh);
        if (threadIdx.x == 0) {
            last = U == 1;
            if (U > 1) {
                double* fp = fix_part + 3 * (size_t)u;
                fp[0] = r.x;
                fp[1] = r.y;
                fp[2] = r.z;
                __threadfence();
                last = atomicAdd(&fix_done[base], 1) == U - 1;
            }
        }
        __syncthreads();
        if (last && threadIdx.x < 32) {
            if (U > 1) {
                __threadfence();
                const volatile double* vp = fix_part + 3 * (size_t)base;
                r = {0.0, 0.0, 0.0};
                for (int q = threadIdx.x; q < U; q += 32) {
                    r.x += vp[3 * q];
                    r.y += vp[3 * q + 1];
                    r.z += vp[3 * q + 2];
                }
                const double v = warp_sum3(r.x, r.y, r.z);
                r.x = v;
                r.y = __shfl_sync(0xffffffffu, v, 16);
                r.z = __shfl_sync(0xffffffffu, v, 8);
                if (threadIdx.x == 0) fix_done[base] = 0;  // ready for the next call
            }
            if (threadIdx.x == 0) {
                double* o = out + i;
                const size_t N = (size_t)n_total;
                o[0] = row ? r.x : o[0] + r.x;
                o[N] = row ? r.y : o[N] + r.y;
                o[2 * N] = row ? r.z : o[2 * N] + r.z;
            }
        }
        __syncthreads();
    }
}

}  // namespace

// Launch shapes of the FP32c kernel (threads per block, ions per thread); the work
// planner sizes i-blocks as threads x ions.  Variant 0 is the default.
static const int kC32Shapes[SG_C32_VARIANTS][2] = {{128, 4}, {128, 2}, {256, 2}, {64, 4},
                                                   {128, 4}, {64, 2}, {32, 4}, {32, 4},
                                                   {64, 2}, {128, 1}, {32, 2}, {32, 1},
                                                   {128, 1}, {64, 2}, {64, 2}, {32, 4},
                                                   {64, 2}, {128, 1}};

int sg_coulomb_fp32c_ib(int variant) {
    if (variant < 0 || variant >= SG_C32_VARIANTS) variant = 0;
    return kC32Shapes[variant][0] * kC32Shapes[variant][1];
}

cudaError_t sg_launch_coulomb_fp32c(const SgCoulombArgs& a, cudaStream_t s) {
    if (a.n_items <= 0 && a.n_near <= 0) return cudaSuccess;
    switch (a.variant) {
        case 1:
            sg_launch(coulomb_fp32c_kernel<128, 2>, a.n_items, 128, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
            break;
        case 2:
            sg_launch(coulomb_fp32c_kernel<256, 2>, a.n_items, 256, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
            break;
        case 3:
            sg_launch(coulomb_fp32c_kernel<64, 4>, a.n_items, 64, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
            break;
        case 5:
            sg_launch(coulomb_fp32c_kernel<64, 2>, a.n_items, 64, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
            break;
        case 6:
            sg_launch(coulomb_fp32c_kernel<32, 4>, a.n_items, 32, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
            break;
        case SG_C32_SORTED:
            sg_launch(coulomb_fp32c_sorted_kernel<128, 4, 4, SG_STAGES>, a.n_items, 128, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case SG_C32_SORTED_LEAF:
            // one k-d leaf per block: warps never wait for a slower (near) neighbour
            sg_launch(coulomb_fp32c_sorted_kernel<32, 4, 16, 3>, a.n_items, 32, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case 8:
            // one leaf per block split over two warps (same far/near decisions)
            sg_launch(coulomb_fp32c_sorted_kernel<64, 2, 12, 3>, a.n_items, 64, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case 9:
            if (a.far_estimate)
                sg_launch(coulomb_fp32c_sorted_kernel<128, 1, 8, 3>, a.n_items, 128, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            else
                sg_launch(coulomb_fp32c_sorted_kernel<128, 1, 8, 3, SG_TILE, 0, false>, a.n_items, 128, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case 12:
            // as 9 with 256-ion j-tiles: half the ring waits and barriers per pair
            if (a.far_estimate)
                sg_launch(coulomb_fp32c_sorted_kernel<128, 1, 8, 3, 256>, a.n_items, 128, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            else
                sg_launch(coulomb_fp32c_sorted_kernel<128, 1, 8, 3, 256, 0, false>, a.n_items, 128, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case 13:
            if (a.far_estimate)
                sg_launch(coulomb_fp32c_sorted_kernel<64, 2, 9, 3, 256>, a.n_items, 64, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            else
                sg_launch(coulomb_fp32c_sorted_kernel<64, 2, 9, 3, 256, 0, false>, a.n_items, 64, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case 14:
            // as 13 with four j pairs in flight per ion on far tiles
            if (a.far_estimate)
                sg_launch(coulomb_fp32c_sorted_kernel<64, 2, 9, 3, 256, 4>, a.n_items, 64, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            else
                sg_launch(coulomb_fp32c_sorted_kernel<64, 2, 9, 3, 256, 4, false>, a.n_items, 64, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case 15:
            // the leaf in one warp (4 ions per thread), 256-ion j-tiles
            sg_launch(coulomb_fp32c_sorted_kernel<32, 4, 16, 3, 256>, a.n_items, 32, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case 16:
            // as 13 with a 4-stage ring
            sg_launch(coulomb_fp32c_sorted_kernel<64, 2, 8, 4, 256>, a.n_items, 64, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword, a.bbox);
            break;
        case SG_C32_FAR_ONCE:
            if (a.n_items > 0)
                sg_launch(coulomb_fp32c_kernel<64, 2>, a.n_items, 64, 0, s, 
                    a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
            if (a.n_near <= 0) break;
            sg_launch(near_list_kernel, (a.n_leaves + 3) / 4, 128, 0, s, a.clouds, a.ctrl, a.leaf_cloud,
                      a.n_leaves, a.near_cap, a.bbox, a.near_count, a.near_list, a.fix_list);
            {
                const LeafAcc acc{a.leaf_sum, a.leaf_fmx, a.leaf_n_close, a.leaf_close};
                sg_launch(a.far_estimate ? coulomb_leaf_kernel<true> : coulomb_leaf_kernel<false>,
                          a.n_near + a.n_far, 32, 0, s, a.c32, a.near_items, a.n_near, a.far_items,
                          a.n_far, a.clouds, a.ctrl, acc, a.npad_total, a.bbox,
                          (const int*)a.near_count, (const unsigned short*)a.near_list, a.near_cap,
                          a.errword);
            }
            break;
        case 10:
            sg_launch(coulomb_fp32c_kernel<32, 2>, a.n_items, 32, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
            break;
        case 11:
            sg_launch(coulomb_fp32c_kernel<32, 1>, a.n_items, 32, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
            break;
        default:
            sg_launch(coulomb_fp32c_kernel<128, 4>, a.n_items, 128, 0, s, 
                a.c32, a.c64, a.items, a.clouds, a.ctrl, a.part, a.npad_total, a.errword);
    }
    return cudaGetLastError();
}

cudaError_t sg_launch_coulomb_fp64(const SgCoulombArgs& a, cudaStream_t s) {
    if (a.n_items <= 0) return cudaSuccess;
    if (a.sym) {
        sg_launch(coulomb_fp64_sym_kernel, a.n_items, SG_SYM_IB, 0, s, a.c64, a.items, a.clouds,
                  a.ctrl, a.part, a.npad_total);
        return cudaGetLastError();
    }
    sg_launch(coulomb_fp64_kernel<SG_C64_THREADS, SG_C64_IPT>, a.n_items, SG_C64_THREADS, 0, s, 
        a.c64, a.items, a.ctrl, a.part, a.npad_total);
    return cudaGetLastError();
}

cudaError_t sg_launch_coulomb_reduce(const SgCoulombArgs& a, const SgRowBlock* rows, int n_rows,
                                     int row_cap, int fp32c, double* out, int n_total,
                                     int* counters, cudaStream_t s) {
    if (n_rows <= 0) return cudaSuccess;
    const int take = n_total <= kInBlockFixupMax || a.max_slots > 24 ? 16 : 64;
    const bool whole = fp32c && a.variant == SG_C32_FAR_ONCE && a.n_items <= 0 && n_total > kInBlockFixupMax;
    const int split = whole ? 1 : std::max(1, row_cap / take);
    if (fp32c) {
        const float* bbox = sg_variant_sorted(a.variant) ? a.bbox : nullptr;
        LeafSums leaf{};
        if (a.variant == SG_C32_FAR_ONCE)
            leaf = LeafSums{{a.leaf_sum, a.leaf_fmx, a.leaf_n_close, a.leaf_close}, a.far_s2f, a.far_estimate};
        if (n_total <= kInBlockFixupMax) {
            sg_launch(coulomb_reduce_kernel<true, true>, n_rows * split, SG_ROWS, 0, s, 
                rows, a.clouds, a.ctrl, a.part, a.npad_total, out, n_total, counters, nullptr,
                a.c32, a.c64, bbox, a.risk, a.ran, a.chk, split, leaf);
            return cudaGetLastError();
        }
        if (a.n_near <= 0) {  // near_list_kernel has cleared it otherwise
            cudaError_t e = cudaMemsetAsync(a.fix_list, 0, 2 * sizeof(int), s);
            if (e != cudaSuccess) return e;
        }
        // a plain launch: nothing programmatic may follow the memset
        coulomb_reduce_kernel<true, false><<<n_rows * split, SG_ROWS, 0, s>>>(
            rows, a.clouds, a.ctrl, a.part, a.npad_total, out, n_total, counters, a.fix_list,
            a.c32, a.c64, nullptr, a.risk, a.ran, a.chk, split, leaf);
        // a fixed grid that strides over however many work units there are (a batch of
        // small clouds can flag a few percent of its ions; unused blocks exit at once)
        const int grid = fixup_blocks(n_total);
        sg_launch(coulomb_fixup_kernel, grid, kFixupThreads, 0, s, 
            a.clouds, a.c32, a.c64, a.npad_total, out, n_total, a.fix_list, bbox,
            a.fix_part, a.fix_done);
    } else {
        sg_launch(coulomb_reduce_kernel<false, false>, n_rows * split, SG_ROWS, 0, s, 
            rows, a.clouds, a.ctrl, a.part, a.npad_total, out, n_total, counters, nullptr,
            nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, split, LeafSums{});
    }
    return cudaGetLastError();
}
