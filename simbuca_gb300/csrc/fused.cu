// fused.cu -- the small-cloud path: whole Dormand-Prince attempts of a cloud in one kernel.
//
// A cloud of a few hundred ions waits for latencies: launches, memory round trips, barriers
// and chains of FP64 instructions (64 cycles of their sub-partition each).  Here one
// thread-block cluster of up to 16 CTAs holds one cloud and runs its attempts back to back
// inside one launch.  CTA r owns the cloud's ions [r m, (r+1) m) in every phase:
//   * stage S (bin/ode.cpp:101-175): a thread per ion and component keeps y, the k_j and
//     the stage state in registers; the components of an ion meet in shared memory;
//   * exchange: each CTA stores its ions' new coordinates (SI and FP32 frame) into the
//     shared memory of every CTA of the cluster, then one cluster barrier (hardware
//     barriers of co-scheduled CTAs: no flag is spun on).  Two coordinate sets alternate
//     by stage, so a CTA may write stage S+1's while another still reads stage S's;
//   * between arriving at the barrier and waiting for it: the part of the next stage that
//     needs no Coulomb sum (field terms, the sum over earlier k_j);
//   * the Coulomb sum (bin/force.cpp:147-174): G threads sum each ion of the CTA against
//     interleaved G-ths of the cloud, in the FP32-compensated form of the tiled kernels
//     (float-float differences, SFU 1/r, 1/r^3 capped with float-float close pairs, partial
//     sums folded into Kahan accumulators every 16 j-ions, the G parts added in
//     float-float); an ion whose terms cancel strongly (s2 > kappa2 |P|^2, sg_kappa2_fused) gets its whole
//     row in FP64 instead, spread over the CTA's warps or (larger wide clouds) all CTAs;
//   * control: error partials go to every CTA, and every CTA decides alike
//     (error_succes and step(), sg_error_succes; bin/ode.cpp:426-494), so the commit
//     pos <- pos2, vel <- vel2 (bin/ode.cpp:488-489) needs no second barrier.
// Seven barriers per attempt.  State returns to the batch's global arrays when the
// launch ends, so every other entry point (upload, download, moments, the tiled path
// itself) sees it.
//
// A cloud of many hundred ions has more pairs than 16 SMs take quickly: the wide form spreads
// it over up to all SMs of the device (a cooperative launch).  There the coordinates go
// through the batch's two global sets and the barrier is a counter in global memory, waited
// for with a limit (SG_TIMEOUT); the rest is the same.  1,000 ions: 93 us per attempt, 124
// in a cluster of 16, 121 in the tiled kernels; 4,096 ions 193, 223 in the tiled kernels.
//
// Measured, one cloud, us per attempt (state, coordinates and sums through global memory
// with 15 barriers, close pairs found by a second scan, a flagged row per warp -> this
// form): 64 ions 70 -> 34, 300 131 -> 56, 512 155 -> 67.  What is left is the
// chain stage - barrier - pairs of dependent instructions.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "dp_stage.cuh"
#include "fp32c_math.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = SG_FUSED_THREADS;
constexpr int kWarps = kThreads / 32;
constexpr int kFold = 8;          // packed j-pairs per FP32 partial sum before the Kahan fold

// What the CTAs of a cluster tell each other at the end of an attempt, two attempts in
// turn: a CTA may be one barrier ahead of another's reads.
struct FusedNote {
    double err[SG_FUSED_MAX_CTAS];  // error partials
    double x0;                      // x of the caller's first ion
};

struct FusedShared {
    SgCtrl cs;
    SgFieldCoef fk[SG_MAX_STAGES];
    FusedNote note[2];
    int expired;  // wide: a wait ran out
    float part[kWarps][8];     // parts of the ions that several warps share
    double red[2][kWarps][3];  // parts of a flagged row; [0][w][0]: error partials
    double x0;
    int ew, wtest;  // at the launch
    int nflag;
};

// Dynamic shared memory: the cloud's coordinates in two sets, its normalized charges, and
// the CTA's own ions (mc of them at most): state, Coulomb sums, flagged ions.
struct FusedArrays {
    double* D;    // [2][3][npc] SI coordinates (wide: the batch's arrays hold them)
    float* C;     // [2][6][npc] frame coordinates: high parts x, y, z, low parts x, y, z (wide: [6][npc])
    float* Q;     // [npc]
    double* ST;   // [6][mc]
    float2* P;    // [3][mc] sums in frame units (float-float), or of a flagged ion SI (double)
    int* list;    // [mc] flagged ions
    int* flag;    // [mc]
    int npc, mc;
};
constexpr size_t smem_bytes(int npc, int mc, bool wide) {
    return (wide ? 7 * sizeof(float) : 13 * sizeof(float) + 6 * sizeof(double)) * (size_t)npc +
           (6 * sizeof(double) + 3 * sizeof(float2) + 2 * sizeof(int)) * (size_t)mc;
}
template <bool WIDE>
__device__ __forceinline__ FusedArrays carve(unsigned char* p, int npc, int mc) {
    FusedArrays s;
    s.D = reinterpret_cast<double*>(p);
    s.C = WIDE ? reinterpret_cast<float*>(p) : reinterpret_cast<float*>(s.D + 6 * npc);
    s.Q = s.C + (WIDE ? 6 : 12) * npc;
    s.ST = reinterpret_cast<double*>(s.Q + npc);  // npc is a multiple of 4: 16-byte aligned
    s.P = reinterpret_cast<float2*>(s.ST + 6 * mc);
    s.list = reinterpret_cast<int*>(s.P + 3 * mc);
    s.flag = s.list + mc;
    s.npc = npc;
    s.mc = mc;
    return s;
}
// Ions of a CTA: a multiple of 4, so that a CTA's rows of the coordinate arrays are whole
// 16-byte words.
__host__ __device__ constexpr int own_ions(int n, int ctas) {
    return ((n + ctas - 1) / ctas + 3) / 4 * 4;
}

// A thread's ions and components of the CTA's 6 m: slot t = thread + u kThreads is row
// t mod m of component t / m (packed: a stage costs an FP64 instruction per warp, whatever
// its lanes hold).
template <int PASSES>
struct Slots {
    int c[PASSES], row[PASSES];  // c = -1: none
    double y[PASSES];            // the step's initial value
    double st[PASSES];           // the stage's
    double k[PASSES][6];
    double p1[PASSES], p7[PASSES];  // Coulomb sums of stages 1 and 7 (acceleration components)
    double base[PASSES], part[PASSES];
    double qm[PASSES], kq[PASSES];
};

// What stage S needs besides its Coulomb sum: k_S of a coordinate or the field terms, and
// the sum over the earlier k_j for the next state or the error.
template <int S, int PASSES>
__device__ __forceinline__ void stage_before(const FusedArrays& s, const SgCloud& cl,
                                             const SgFieldCoef& fk, Slots<PASSES>& w) {
#pragma unroll
    for (int u = 0; u < PASSES; u++) {
        const int c = w.c[u];
        if (c < 0) continue;
        const double* st = s.ST + w.row[u];
        if (c < 3) {
            w.base[u] = st[(3 + c) * s.mc];
        } else {
            const int ax = c - 3, o = ax == 0 ? 1 : 0;
            w.base[u] = sg_field_axis(cl.fp, fk, w.qm[u], ax, st[ax * s.mc], st[c * s.mc],
                                      st[o * s.mc], st[(3 + o) * s.mc]);
        }
        double a = 0.0;
#pragma unroll
        for (int j = 1; j < S; j++) {
            if (S < 7)
                a += MethodDP::a(S + 1, j - 1) * w.k[u][j - 1];
            else if (j != 2)
                a += MethodDP::e(j) * w.k[u][j - 1];
        }
        w.part[u] = a;
    }
}

// k_S with the Coulomb sum of the ion, and the next stage's state; at S = 7 the squared
// scaled error (bin/ode.cpp:107-205).
template <int S, int PASSES>
__device__ __forceinline__ double stage_after(const FusedArrays& s, const SgCloud& cl, double h,
                                              double atol, double rtol, bool coul,
                                              Slots<PASSES>& w) {
    double acc2 = 0.0;
#pragma unroll
    for (int u = 0; u < PASSES; u++) {
        const int c = w.c[u];
        if (c < 0) continue;
        double kS = w.base[u];
        if (c >= 3) {
            double P = 0.0;
            if (S == 1) {
                P = w.p1[u];
            } else if (coul) {
                const float2* p = s.P + (c - 3) * s.mc + w.row[u];
                P = s.flag[w.row[u]] ? *reinterpret_cast<const double*>(p)
                                     : cl.psc * ((double)p->x + (double)p->y);
            }
            if (S == 7) w.p7[u] = P;
            kS = kS + w.kq[u] * P;
        }
        if constexpr (S < 7) {
            w.k[u][S - 1] = kS;
            w.st[u] = w.y[u] + h * (w.part[u] + MethodDP::a(S + 1, S - 1) * kS);
        } else {
            const double e = w.part[u] + MethodDP::e(7) * kS;
            const double m0 = fabs(w.y[u]), m1 = fabs(w.st[u]);
            const double sk = atol + rtol * ((m0 < m1) ? m1 : m0);
            const double r = h * e * stage_rcp(sk);
            acc2 += r * r;
        }
    }
    return acc2;
}

// The new state into shared memory, its coordinates into set `set`: of this CTA's shared
// memory, or (wide) of the batch's arrays.
template <bool WIDE, int PASSES>
__device__ __forceinline__ void store_state(const SgFusedArgs& f, const FusedArrays& s,
                                            const SgCloud& cl, int lo, int set,
                                            const Slots<PASSES>& w) {
    const size_t NP = (size_t)f.npad;
#pragma unroll
    for (int u = 0; u < PASSES; u++) {
        const int c = w.c[u];
        if (c < 0) continue;
        s.ST[c * s.mc + w.row[u]] = w.st[u];
        if (c < 3) {
            const int li = lo + w.row[u];
            const double v = (w.st[u] - (c == 0 ? cl.cx : c == 1 ? cl.cy : cl.cz)) * cl.invL;
            float hi, low;
            split_double(v, hi, low);
            if (WIDE) {
                float* C = f.c32 + set * 7 * NP + cl.poff + li;
                C[c * NP] = hi;
                C[(4 + c) * NP] = low;
                f.c64[(set * 4 + c) * NP + cl.poff + li] = w.st[u];
            } else {
                float* C = s.C + set * 6 * s.npc + li;
                C[c * s.npc] = hi;
                C[(3 + c) * s.npc] = low;
                s.D[(set * 3 + c) * s.npc + li] = w.st[u];
            }
        }
    }
}

// Wide: the cloud's frame coordinates of set `set`, written by every CTA of the cloud, from
// the batch's arrays (through L2).
__device__ __forceinline__ void load_coords(const SgFusedArgs& f, const FusedArrays& s,
                                            const SgCloud& cl, int set) {
    const size_t NP = (size_t)f.npad;
    const float4* src = reinterpret_cast<const float4*>(f.c32 + set * 7 * NP + cl.poff);
    const size_t row = NP / 4;  // rows of whole 16-byte words
#pragma unroll 2
    for (int v = threadIdx.x; v < s.npc / 4; v += kThreads) {
        float4 x[6];
#pragma unroll
        for (int a = 0; a < 6; a++) x[a] = __ldcg(src + (a < 3 ? a : a + 1) * row + v);
#pragma unroll
        for (int a = 0; a < 6; a++) reinterpret_cast<float4*>(s.C + a * s.npc)[v] = x[a];
    }
    __syncthreads();
}

// Wide: a cloud's CTAs and their barrier, a counter that each raises by one.  All of them are
// resident (cooperative launch); a wait gives up after SG_WAIT_NS.
struct WideGroup {
    int* count;   // arrivals, departures
    int R, r;     // CTAs of the cloud, this one's rank
    unsigned target;  // arrivals so far (modulo 2^32)
    int* flag_n;  // [2] flagged ions of the stage in either coordinate set ...
    double* flags;  // [2][SG_WIDE_FLAGS][4] ... x, y, z, index in the cloud
    bool share;   // flagged rows

    __device__ __forceinline__ void arrive() {
        __syncthreads();  // the CTA's stores come before its arrival
        target += (unsigned)R;
        if (threadIdx.x == 0)
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    }
    // past: arrivals beyond the last ones to wait for (the wait test)
    __device__ __forceinline__ bool wait(FusedShared& sh, unsigned past = 0,
                                         unsigned long long limit_ns = SG_WAIT_NS) {
        if (threadIdx.x == 0) {
            unsigned seen;
            unsigned long long t0 = 0, t;
            for (;;) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
                if (sg_reached(seen, target + past)) break;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                if (t0 == 0) t0 = t;
                if (t - t0 > limit_ns) {
                    sh.expired = 1;
                    break;
                }
            }
        }
        __syncthreads();
        return sh.expired == 0;
    }
};
// Wide clouds of more padded ions, or of more ions a CTA, share a flagged ion's FP64 row
// between all their CTAs: two more barriers a stage with a flagged ion and one without
// (~1.5 us each), where a row in one CTA takes 4 us per 1,000 ions, two in the same CTA twice
// that, and the others wait for it.  us per attempt, rows in one CTA / shared: 700 ions (5 a
// CTA) 78 / 90, 850 83 / 90, 1,200 136 / 96, 3,000 205 / 157; 2 clouds of 700 (10 a CTA) 75 / 82,
// 4 of 700 (19) 110 / 91, 8 of 600 (32) 113 / 90.
constexpr int kShareIons = 896, kShareOwn = 12;

// This CTA's rows [lo, lo + m) of set `set` into the other CTAs' shared memory, 16 bytes a
// store: 6 m / 4 words of frame coordinates and 3 m / 2 of SI ones for each.
__device__ __forceinline__ void push_coords(cg::cluster_group& cluster, const FusedArrays& s,
                                            int lo, int m, int set, int ctas, int r) {
    const int m4 = min(m, s.npc - lo) / 4, nv = 12 * m4;  // past the last ion: padding
    for (int q = threadIdx.x; q < nv * ctas; q += kThreads) {
        const int to = q / nv, v = q - to * nv;
        if (to == r) continue;
        float4* src;
        if (v < 6 * m4) {
            const int a = v / m4;
            src = reinterpret_cast<float4*>(s.C + (set * 6 + a) * s.npc + lo) + (v - a * m4);
        } else {
            const int a = (v - 6 * m4) / (2 * m4);
            src = reinterpret_cast<float4*>(s.D + (set * 3 + a) * s.npc + lo) +
                  (v - 6 * m4 - a * 2 * m4);
        }
        *cluster.map_shared_rank(src, to) = *src;
    }
}

// The sums of one thread: every G-th packed j-pair (j = 2p, 2p + 1) from pair q on against ion
// li, so that the G threads of an ion read consecutive 8-byte words of shared memory (no bank
// conflicts; the ions of a warp read the same words).  Every 8 pairs (16 j-ions) the FP32
// partial sums are folded into the Kahan accumulators.  GT: G where it is known.
//
// Bound by the issue and latency of a warp's instructions (18 packed FP32x2, 7 loads, ~6 ALU
// per packed pair, four warps a sub-partition): close pairs are looked for once per four
// packed pairs, and only the last ones of a cloud test for its end.  us per attempt, both
// tests for each pair / so: 300 ions 60 / 56, 1,000 72 / 67, 4,096 206 / 193.  Two ions a
// thread (half the loads per pair) spilled and gave 190 at 4,096, 65 at 300.
struct IonSums {
    ff x, y, z;
    float s2;
};
template <int GT, class Load>
__device__ __forceinline__ IonSums ion_pairs(const float* X, const float* Q, int npc, int q, int G0,
                                             int li, float wc, const double* SX, const double* SQ,
                                             size_t ND, double psc, const Load& ld) {
    const int G = GT ? GT : G0;
    const int npair = npc / 2;
    const float* Y = X + npc;
    const float* Z = X + 2 * npc;
    const float* XL = X + 3 * npc;
    const float* YL = X + 4 * npc;
    const float* ZL = X + 5 * npc;
    const float xih = X[li], yih = Y[li], zih = Z[li];
    const float xil = XL[li], yil = YL[li], zil = ZL[li];
    const f2 xh = pk(xih, xih), yh = pk(yih, yih), zh = pk(zih, zih);
    const f2 xl = pk(xil, xil), yl = pk(yil, yil), zl = pk(zil, zil);
    const f2 tiny2 = pk(kTiny, kTiny);
    float ks[3] = {0.f, 0.f, 0.f}, kc[3] = {0.f, 0.f, 0.f}, s2 = 0.f, fmx = 0.f;
    ff cx{0.f, 0.f}, cy{0.f, 0.f}, cz{0.f, 0.f};
    for (int b0 = q; b0 < npair; b0 += 2 * kFold * G) {
        // close pairs of these 32 j-ions, a bit each (the self pair, dx = 0, with them)
        unsigned close = 0u;
#pragma unroll
        for (int hb = 0; hb < 2; hb++) {
            f2 ax = 0ull, ay = 0ull, az = 0ull;
#pragma unroll
            for (int u0 = 0; u0 < kFold; u0 += 4) {
                const int p0 = b0 + (hb * kFold + u0) * G;
                if (p0 >= npair) break;
                float y3[8], m4 = 0.f;
                auto four = [&](auto tail) {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        // past the cloud's last pair: pair 0 again, with no weight
                        const bool ok = !decltype(tail)::value || p0 + u * G < npair;
                        const int jj = ok ? 2 * (p0 + u * G) : 0;
                        const f2 Xj = *reinterpret_cast<const f2*>(X + jj);
                        const f2 Yj = *reinterpret_cast<const f2*>(Y + jj);
                        const f2 Zj = *reinterpret_cast<const f2*>(Z + jj);
                        const f2 Qj = *reinterpret_cast<const f2*>(Q + jj);
                        const f2 XLj = *reinterpret_cast<const f2*>(XL + jj);
                        const f2 YLj = *reinterpret_cast<const f2*>(YL + jj);
                        const f2 ZLj = *reinterpret_cast<const f2*>(ZL + jj);
                        const f2 dx = add2(sub2(Xj, xh), sub2(XLj, xl));
                        const f2 dy = add2(sub2(Yj, yh), sub2(YLj, yl));
                        const f2 dz = add2(sub2(Zj, zh), sub2(ZLj, zl));
                        f2 r2 = fma2(dx, dx, tiny2);
                        r2 = fma2(dy, dy, r2);
                        r2 = fma2(dz, dz, r2);
                        float ra, rb, ua, ub;
                        upk(r2, ra, rb);
                        const f2 yv = pk(rsqrt_approx(ra), rsqrt_approx(rb));
                        upk(mul2(mul2(yv, yv), yv), ua, ub);
                        const f2 w = mul2(ok ? Qj : 0ull, pk(fminf(ua, wc), fminf(ub, wc)));
                        ax = fma2(w, dx, ax);
                        ay = fma2(w, dy, ay);
                        az = fma2(w, dz, az);
                        y3[2 * u] = ok ? ua : 0.f;
                        y3[2 * u + 1] = ok ? ub : 0.f;
                        m4 = fmaxf(m4, fmaxf(y3[2 * u], y3[2 * u + 1]));
                    }
                };
                if (p0 + 3 * G < npair)
                    four(std::false_type{});
                else
                    four(std::true_type{});
                if (m4 > wc) {
                    // which, and the strongest of the others (a capped one counts below)
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        if (y3[e] > wc)
                            close |= 1u << (2 * (hb * kFold + u0) + e);
                        else
                            fmx = fmaxf(fmx, y3[e]);
                    }
                } else {
                    fmx = fmaxf(fmx, m4);
                }
            }
            float a, b;
            upk(ax, a, b);
            const float tx = __fadd_rn(a, b);
            upk(ay, a, b);
            const float ty = __fadd_rn(a, b);
            upk(az, a, b);
            const float tz = __fadd_rn(a, b);
            kahan_add(ks[0], kc[0], tx);
            kahan_add(ks[1], kc[1], ty);
            kahan_add(ks[2], kc[2], tz);
            s2 = fmaf(tx, tx, fmaf(ty, ty, fmaf(tz, tz, s2)));
        }
        // close pairs: the exact term minus the capped FP32 one (close_term_ff; the
        // closest in FP64 from the SI coordinates); a capped term is a candidate for
        // the strongest
        while (close) {
            const int bit = __ffs(close) - 1;
            close &= close - 1u;
            const int jj = 2 * (b0 + (bit >> 1) * G) + (bit & 1);
            if (jj == li || Q[jj] == 0.f) continue;
            const PairF pr = pair_f32(X[jj], Y[jj], Z[jj], XL[jj], YL[jj], ZL[jj], xih, yih, zih, xil,
                                      yil, zil);
            fmx = fmaxf(fmx, capped_term_y3(pr.y3, wc));
            const float wf = __fmul_rn(Q[jj], wc);
            ff dx, dy, dz;
            if (!very_close(pr.y3, xih, yih, zih)) {
                close_term_ff(ff_diff(X[jj], XL[jj], xih, xil), ff_diff(Y[jj], YL[jj], yih, yil),
                              ff_diff(Z[jj], ZL[jj], zih, zil), Q[jj], wf, pr, dx, dy, dz);
            } else {
                const double rx = ld(SX + li) - ld(SX + jj),
                             ry = ld(SX + ND + li) - ld(SX + ND + jj),
                             rz = ld(SX + 2 * ND + li) - ld(SX + 2 * ND + jj);
                const double w = SQ[jj] * inv_r3_fp64(rx * rx + ry * ry + rz * rz) / psc;
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
            cx = ff_add(cx, dx);
            cy = ff_add(cy, dy);
            cz = ff_add(cz, dz);
        }
    }
    return IonSums{ff_add({ks[0], -kc[0]}, cx), ff_add({ks[1], -kc[1]}, cy),
                   ff_add({ks[2], -kc[2]}, cz), conditioning_s2(s2, fmx)};
}

// Coulomb sums of the CTA's mo ions (cloud indices lo ...) at coordinate set `set` into
// s.P, in the FP32-compensated form; risk: where the in-run check's inputs go (null: not
// written).
// One copy for the six stages of an attempt (inlined, they took minutes to compile).
template <bool WIDE>
__device__ __noinline__ bool coulomb_phase(const SgFusedArgs& f, const SgCloud& cl, int mc, int lo,
                                           int mo, int set, float* risk, FusedShared& sh,
                                           WideGroup& g) {
    extern __shared__ __align__(16) unsigned char dyn[];
    const FusedArrays s = carve<WIDE>(dyn, cl.npad, mc);
    const int tid = threadIdx.x;
    const int npc = s.npc;
    const float* X = s.C + (WIDE ? 0 : set * 6 * npc);
    const size_t ND = WIDE ? (size_t)f.npad : (size_t)npc;
    const double* SX = WIDE ? f.c64 + set * 4 * ND + cl.poff : s.D + set * 3 * npc;
    const double* SY = SX + ND;
    const double* SZ = SX + 2 * ND;
    // other CTAs write the global coordinates: through L2
    auto ld = [](const double* p) { return WIDE ? __ldcg(p) : *p; };
    const double* SQ = f.c64 + 3 * (size_t)f.npad + cl.poff;  // charges: never rewritten here
    // G threads per ion: as many as the CTA has, up to four warps of them
    int G = 1;
    while (2 * G * mo <= kThreads && 2 * G <= 128 && 4 * G <= npc) G *= 2;
    const int il = tid / G, q = tid - il * G;
    const int li = lo + il;  // index in the cloud's coordinate arrays
    IonSums p{{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, 0.f};
    if (il < mo) {
        switch (G) {
            case 128: p = ion_pairs<128>(X, s.Q, npc, q, G, li, cl.wc, SX, SQ, ND, cl.psc, ld); break;
            case 64: p = ion_pairs<64>(X, s.Q, npc, q, G, li, cl.wc, SX, SQ, ND, cl.psc, ld); break;
            case 32: p = ion_pairs<32>(X, s.Q, npc, q, G, li, cl.wc, SX, SQ, ND, cl.psc, ld); break;
            case 16: p = ion_pairs<16>(X, s.Q, npc, q, G, li, cl.wc, SX, SQ, ND, cl.psc, ld); break;
            default: p = ion_pairs<0>(X, s.Q, npc, q, G, li, cl.wc, SX, SQ, ND, cl.psc, ld);
        }
    }
    // the G parts of each ion, in a fixed order, still in float-float: first those of a warp
    // (consecutive lanes), then the warps'; the first thread of the G holds the ion
    ff px = p.x, py = p.y, pz = p.z;
    float ps2 = p.s2;
    for (int o = min(G, 32) / 2; o > 0; o >>= 1) {
        ff v;
        v.h = __shfl_down_sync(0xffffffffu, px.h, o);
        v.l = __shfl_down_sync(0xffffffffu, px.l, o);
        px = ff_add(px, v);
        v.h = __shfl_down_sync(0xffffffffu, py.h, o);
        v.l = __shfl_down_sync(0xffffffffu, py.l, o);
        py = ff_add(py, v);
        v.h = __shfl_down_sync(0xffffffffu, pz.h, o);
        v.l = __shfl_down_sync(0xffffffffu, pz.l, o);
        pz = ff_add(pz, v);
        ps2 += __shfl_down_sync(0xffffffffu, ps2, o);
    }
    if (G > 32) {
        float* v = sh.part[tid >> 5];
        if ((tid & 31) == 0) {
            v[0] = px.h;
            v[1] = px.l;
            v[2] = py.h;
            v[3] = py.l;
            v[4] = pz.h;
            v[5] = pz.l;
            v[6] = ps2;
        }
        __syncthreads();
        if (q == 0)
            for (int w = 1; w < G / 32; w++) {
                v += 8;
                px = ff_add(px, {v[0], v[1]});
                py = ff_add(py, {v[2], v[3]});
                pz = ff_add(pz, {v[4], v[5]});
                ps2 += v[6];
            }
    }
    // the conditioning test (frame units for a unit charge)
    if (il < mo && q == 0) {
        const float pf2 = fmaf(px.h, px.h, fmaf(py.h, py.h, pz.h * pz.h));
        const bool flagged = ps2 > sg_kappa2_fused(npc, f.loose) * pf2;
        s.flag[il] = flagged;
        if (flagged) {
            s.list[atomicAdd(&sh.nflag, 1)] = il;
            if (WIDE && g.share) {
                const int at = atomicAdd(g.flag_n + set, 1);
                if (at < SG_WIDE_FLAGS) {
                    double* e = g.flags + 4 * (set * SG_WIDE_FLAGS + at);
                    for (int c = 0; c < 3; c++) e[c] = s.ST[c * s.mc + il];
                    e[3] = (double)li;
                }
                s.flag[il] = at + 1;
            }
        } else {
            s.P[il] = make_float2(px.h, px.l);
            s.P[s.mc + il] = make_float2(py.h, py.l);
            s.P[2 * s.mc + il] = make_float2(pz.h, pz.l);
        }
        if (risk != nullptr) {
            const size_t i = (size_t)cl.off + li;
            risk[i] = flagged ? -1.f : 0.f;
            risk[(size_t)f.n + i] = flagged ? -1.f : sqrtf(ps2 / pf2);
        }
    }
    __syncthreads();
    if (WIDE && g.share) {
        // shared rows: every CTA of the cloud takes its j-ions of each flagged ion, a warp an
        // ion, and the owners add the parts in rank order
        const int warp = tid >> 5, lane = tid & 31;
        const int len = (npc / 32 + g.R - 1) / g.R * 32;
        const int j0 = g.r * len, j1 = min(npc, j0 + len);
        g.arrive();
        // this lane's first j-ion arrives while the barrier completes, the warp's first
        // flagged ion with their number
        double jx = 0.0, jy = 0.0, jz = 0.0, jq = 0.0;
        if (j0 < j1) {
            jx = ld(SX + j0 + lane);
            jy = ld(SY + j0 + lane);
            jz = ld(SZ + j0 + lane);
            jq = SQ[j0 + lane];
        }
        if (!g.wait(sh)) return false;
        const double2* flags = reinterpret_cast<const double2*>(g.flags + 4 * set * SG_WIDE_FLAGS);
        double2 e0 = __ldcg(flags + 2 * warp), e1 = __ldcg(flags + 2 * warp + 1);
        const int all = __ldcg(g.flag_n + set);
        if (all == 0) return true;
        if (all <= SG_WIDE_FLAGS) {
            double* parts = f.flag_part + (size_t)set * SG_WIDE_FLAGS * SG_FUSED_MAX_WIDE * 3;
            for (int k = warp; k < all; k += kWarps) {
                if (k != warp) {
                    e0 = __ldcg(flags + 2 * k);
                    e1 = __ldcg(flags + 2 * k + 1);
                }
                const int lf = (int)e1.y;
                double ax = 0.0, ay = 0.0, az = 0.0;
                for (int jj = j0 + lane; jj < j1; jj += 32) {
                    const bool first = jj == j0 + lane;
                    if (jj == lf) continue;
                    const double rx = e0.x - (first ? jx : ld(SX + jj)),
                                 ry = e0.y - (first ? jy : ld(SY + jj)),
                                 rz = e1.x - (first ? jz : ld(SZ + jj));
                    const double wq = (first ? jq : SQ[jj]) * inv_r3_fp64(rx * rx + ry * ry + rz * rz);
                    ax = fma(wq, rx, ax);
                    ay = fma(wq, ry, ay);
                    az = fma(wq, rz, az);
                }
                __syncwarp();
                const double v = j0 < j1 ? warp_sum3(ax, ay, az) : 0.0;
                if (lane == 0 || lane == 8 || lane == 16)
                    parts[((size_t)k * SG_FUSED_MAX_WIDE + blockIdx.x) * 3 +
                          (lane == 0 ? 0 : lane == 16 ? 1 : 2)] = v;
            }
            g.arrive();
            if (!g.wait(sh)) return false;
            for (int k = warp; k < sh.nflag; k += kWarps) {
                const int fi = s.list[k];
                const double* p = parts + ((size_t)(s.flag[fi] - 1) * SG_FUSED_MAX_WIDE +
                                           (blockIdx.x - g.r)) * 3;
                double ax = 0.0, ay = 0.0, az = 0.0;
                for (int q = lane; q < g.R; q += 32) {
                    ax += __ldcg(p + 3 * q);
                    ay += __ldcg(p + 3 * q + 1);
                    az += __ldcg(p + 3 * q + 2);
                }
                __syncwarp();
                const double v = warp_sum3(ax, ay, az);
                if (lane == 0 || lane == 8 || lane == 16)
                    *reinterpret_cast<double*>(s.P + (lane == 0 ? 0 : lane == 16 ? 1 : 2) * s.mc + fi) = v;
            }
            __syncthreads();
            return true;
        }
    }
    // Flagged ions: the whole row in FP64 from the SI coordinates, which replaces the ion's
    // sum (re-evaluating only its dominant pairs would keep the rounding of the FP32
    // additions made while they were in a partial sum).  The CTA's warps share a row by 32
    // j-ions: a row of 300 in one warp held up the whole cluster for 11,700 cycles.
    const int nf = sh.nflag;
    const int warp = tid >> 5, lane = tid & 31;
    for (int k = 0; k < nf; k++) {
        const int fi = s.list[k], lf = lo + fi;
        double(*red)[3] = sh.red[k & 1];
        if (32 * warp < npc) {
            double ax = 0.0, ay = 0.0, az = 0.0;
            const double xi = ld(SX + lf), yi = ld(SY + lf), zi = ld(SZ + lf);
            for (int jj = 32 * warp + lane; jj < npc; jj += kThreads) {
                if (jj == lf) continue;
                const double rx = xi - ld(SX + jj), ry = yi - ld(SY + jj), rz = zi - ld(SZ + jj);
                const double wq = SQ[jj] * inv_r3_fp64(rx * rx + ry * ry + rz * rz);
                ax = fma(wq, rx, ax);
                ay = fma(wq, ry, ay);
                az = fma(wq, rz, az);
            }
            __syncwarp();
            const double v = warp_sum3(ax, ay, az);
            if (lane == 0) red[warp][0] = v;
            if (lane == 16) red[warp][1] = v;
            if (lane == 8) red[warp][2] = v;
        }
        __syncthreads();
        if (tid < 96) {
            const int c = warp;
            double v = lane < kWarps && 32 * lane < npc ? red[lane][c] : 0.0;
            for (int o = kWarps / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) *reinterpret_cast<double*>(s.P + c * s.mc + fi) = v;
        }
    }
    if (nf > 0) __syncthreads();
    return true;
}

// Control of an attempt with error norm err (thread 0 of every CTA alike): error_succes,
// step() and the bookkeeping of dp_control_kernel for clouds without a recorder or
// operations.
__device__ __forceinline__ void control_phase(FusedShared& sh, const SgCloud& cl, const double* x0,
                                              double err) {
    SgCtrl& cs = sh.cs;
    cs.err = err;
    cs.print_due = 0;
    cs.force_evals += 7;
    cs.coulomb_evals += (cl.fp.flags & SG_F_COULOMB) ? 6 : 0;
    int accepted;
    if (sh.ew != 0) {
        cs.status = sh.ew;
        cs.done = 1;
        accepted = 0;
    } else {
        accepted = sg_error_succes(cs, err, x0);
    }
    if (accepted) {
        cs.h_last = cs.h;
        cs.t = cs.t + cs.h;
        cs.h = cs.hnext;
        cs.steps++;
        cs.stepped = 1;
        cs.rejects_here = 0;
        if (cs.t >= cs.t_end) cs.done = 1;
    }
    cs.accepted = accepted;
}

template <int PASSES, bool WIDE>
__global__ void __launch_bounds__(kThreads, 1) fused_attempts_kernel(const __grid_constant__ SgFusedArgs f,
                                                                     int mc) {
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ FusedShared sh;
    cg::cluster_group cluster = cg::this_cluster();
    const int R = WIDE ? f.ctas : (int)cluster.num_blocks();
    const int c = blockIdx.x / R;
    const int r = blockIdx.x - c * R;  // the rank in its cluster
    const int tid = threadIdx.x;
    const SgCloud& cl = f.clouds[c];
    const FusedArrays s = carve<WIDE>(dyn, cl.npad, mc);
    const int n = cl.n, npc = cl.npad;
    const int m = own_ions(n, R);
    const int lo = min(n, r * m), mo = min(n, (r + 1) * m) - lo;
    const int ctas = (n + m - 1) / m;  // CTAs with ions
    const bool coul = (cl.fp.flags & SG_F_COULOMB) != 0;
    const bool frozen = (cl.fp.flags & SG_F_FROZEN_T) != 0;
    const size_t N = (size_t)f.n, NP = (size_t)f.npad;
    if (tid == 0) {
        sh.cs = f.ctrl[c];
        if (f.one_step == 1) sh.cs.stepped = 0;
        sh.ew = f.flags[SG_FLAG_ERR];
        sh.wtest = f.flags[SG_FLAG_WAIT_TILE];
        sh.expired = 0;
    }
    // charges; the padding's coordinates, and for whole 16-byte words of the last CTA's rows
    // they are in both sets of every CTA
    for (int j = tid; j < npc; j += kThreads) s.Q[j] = f.c32[3 * NP + cl.poff + j];
    for (int j = n + tid; !WIDE && j < npc; j += kThreads)
        for (int set = 0; set < 2; set++)
            for (int a = 0; a < 3; a++) {
                float* C = s.C + (set * 6 + a) * npc + j;
                C[0] = f.c32[a * NP + cl.poff + j];
                C[3 * npc] = f.c32[(4 + a) * NP + cl.poff + j];
                s.D[(set * 3 + a) * npc + j] = f.c64[a * NP + cl.poff + j];
            }
    Slots<PASSES> w;
#pragma unroll
    for (int u = 0; u < PASSES; u++) {
        const int t = tid + u * kThreads;
        w.c[u] = t < 6 * mo ? t / mo : -1;
        w.row[u] = 0;
        w.y[u] = w.p1[u] = w.p7[u] = w.qm[u] = w.kq[u] = w.st[u] = 0.0;
        if (w.c[u] < 0) continue;
        w.row[u] = t - w.c[u] * mo;
        const size_t i = (size_t)cl.off + lo + w.row[u];
        w.y[u] = f.y[w.c[u] * N + i];
        if (w.c[u] >= 3) {
            w.qm[u] = f.qm[i];
            w.kq[u] = f.kq[i];
            if (coul) w.p1[u] = f.coul1[(w.c[u] - 3) * N + i];
        }
    }
    // wide: the cloud's barrier counter and notes
    WideGroup g{};
    double* notes = WIDE ? f.notes + (size_t)c * 2 * (SG_FUSED_MAX_WIDE + 1) : nullptr;
    bool ok = true;
    if (WIDE) {
        g.count = f.barrier + 2 * c;
        g.R = R;
        g.r = r;
        g.share = npc > kShareIons || m > kShareOwn;
        g.flag_n = f.flag_n + 2 * c;
        g.flags = f.flag_list + 8 * SG_WIDE_FLAGS * c;
        if (r == 0 && tid == 0) g.flag_n[0] = g.flag_n[1] = 0;
        g.arrive();
        ok = sh.wtest != 1 ? g.wait(sh)
                           : g.wait(sh, 1,  // the wait test: never
                                    1000ull * max(f.flags[SG_FLAG_WAIT_US], 1));
    } else {
        cluster.sync();  // every CTA runs, and has read the control block
    }
    int att = 0;
    for (; ok && att < f.max_attempts; att++) {
        if (sh.cs.done || sh.cs.hold || sh.cs.status != SG_OK || sh.ew != 0 ||
            (f.one_step && sh.cs.stepped))
            break;
        const double t0 = sh.cs.t, h = sh.cs.h, atol = sh.cs.atol, rtol = sh.cs.rtol;
        // every stage's field coefficients, a lane each
        if (tid < MethodDP::stages) {
            const int st = tid + 1;
            sh.fk[st] = sg_field_coef(cl.fp, frozen ? t0 : t0 + MethodDP::c(st) * h);
        }
#pragma unroll
        for (int u = 0; u < PASSES; u++)
            if (w.c[u] >= 0) {
                w.st[u] = w.y[u];
                s.ST[w.c[u] * mc + w.row[u]] = w.y[u];
            }
        __syncthreads();
        stage_before<1>(s, cl, sh.fk[1], w);
        stage_after<1>(s, cl, h, atol, rtol, coul, w);
        __syncthreads();  // the step's initial state has been read
        // the state of stage S+1 is in w: its Coulomb sum, then k_{S+1}
#define SG_FUSED_STAGE(S)                                                              \
    store_state<WIDE>(f, s, cl, lo, (S) & 1, w);                                       \
    if (tid == 0) sh.nflag = 0;                                                        \
    if (!coul) {                                                                       \
        __syncthreads();                                                               \
        stage_before<S>(s, cl, sh.fk[S], w);                                           \
        __syncthreads();                                                               \
    } else if (WIDE) {                                                                 \
        g.arrive();                                                                    \
        stage_before<S>(s, cl, sh.fk[S], w);                                           \
        ok = g.wait(sh);                                                               \
        if (!ok) break;                                                                \
        if (r == 0 && tid == 0) g.flag_n[((S) & 1) ^ 1] = 0;                           \
        load_coords(f, s, cl, (S) & 1);                                                \
        ok = coulomb_phase<WIDE>(f, cl, mc, lo, mo, (S) & 1, (S) == 7 ? f.risk : nullptr, sh, g); \
        if (!ok) break;                                                                \
    } else {                                                                           \
        __syncthreads();                                                               \
        if (mo > 0) push_coords(cluster, s, lo, m, (S) & 1, ctas, r);                  \
        auto token = cluster.barrier_arrive();                                         \
        stage_before<S>(s, cl, sh.fk[S], w);                                           \
        cluster.barrier_wait(std::move(token));                                        \
        coulomb_phase<WIDE>(f, cl, mc, lo, mo, (S) & 1, (S) == 7 ? f.risk : nullptr, sh, g); \
    }
        SG_FUSED_STAGE(2)
        stage_after<2>(s, cl, h, atol, rtol, coul, w);
        SG_FUSED_STAGE(3)
        stage_after<3>(s, cl, h, atol, rtol, coul, w);
        SG_FUSED_STAGE(4)
        stage_after<4>(s, cl, h, atol, rtol, coul, w);
        SG_FUSED_STAGE(5)
        stage_after<5>(s, cl, h, atol, rtol, coul, w);
        SG_FUSED_STAGE(6)
        stage_after<6>(s, cl, h, atol, rtol, coul, w);
        SG_FUSED_STAGE(7)
        double e = stage_after<7>(s, cl, h, atol, rtol, coul, w);
#undef SG_FUSED_STAGE
        // the CTA's error partial (warps without a component add nothing), to every CTA
        const int warp = tid >> 5, lane = tid & 31;
        const int nw = min(kWarps, (6 * mo + 31) / 32);  // warps with a component
        if (warp < nw) {
            for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
            if (lane == 0) sh.red[0][warp][0] = e;
        }
#pragma unroll
        for (int u = 0; u < PASSES; u++)
            if (w.c[u] == 0 && cl.off + lo + w.row[u] == cl.ion0) sh.x0 = w.y[u];
        __syncthreads();
        const bool own0 = cl.ion0 >= cl.off + lo && cl.ion0 < cl.off + lo + mo;
        if constexpr (WIDE) {
            double* nt = notes + (att & 1) * (SG_FUSED_MAX_WIDE + 1);
            if (tid < 32) {
                double v = lane < nw ? sh.red[0][lane][0] : 0.0;
                for (int o = kWarps / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) {
                    nt[r] = v;
                    if (own0) nt[SG_FUSED_MAX_WIDE] = sh.x0;
                }
            }
            g.arrive();
            ok = g.wait(sh);
            if (!ok) break;
            if (tid < 32) {
                double v = 0.0;
                for (int q = lane; q < R; q += 32) v += __ldcg(nt + q);
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) {
                    sh.x0 = __ldcg(nt + SG_FUSED_MAX_WIDE);
                    control_phase(sh, cl, &sh.x0, sqrt(v / (6 * n)));
                }
            }
        } else {
            FusedNote& nt = sh.note[att & 1];
            if (tid < 32) {
                double v = lane < nw ? sh.red[0][lane][0] : 0.0;
                for (int o = kWarps / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane < R) {
                    FusedNote* to = cluster.map_shared_rank(&nt, lane);
                    to->err[r] = v;
                    if (own0) to->x0 = sh.x0;
                }
            }
            cluster.sync();
            if (tid < 32) {
                double v = lane < R ? nt.err[lane] : 0.0;
                for (int o = SG_FUSED_MAX_CTAS / 2; o > 0; o >>= 1)
                    v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) control_phase(sh, cl, &nt.x0, sqrt(v / (6 * n)));
            }
        }
        __syncthreads();
        if (sh.cs.accepted) {
            // commit: pos <- pos2, vel <- vel2; the stage-7 sum is the next stage-1 sum
#pragma unroll
            for (int u = 0; u < PASSES; u++) {
                w.y[u] = w.st[u];
                w.p1[u] = w.p7[u];
            }
        }
    }
    if constexpr (WIDE) {
        // the last CTA to leave clears the counters for the next launch; a wait that ran out
        // stops the batch
        if (tid == 0) {
            if (!ok) {
                atomicExch(f.flags + SG_FLAG_ERR, SG_TIMEOUT);
                if (r == 0) {
                    f.ctrl[c].status = SG_TIMEOUT;
                    f.ctrl[c].done = 1;
                }
            }
            if (atomicAdd(g.count + 1, 1) == R - 1) {
                g.count[0] = 0;
                g.count[1] = 0;
            }
        }
        if (!ok) return;
    }
    if (att == 0) return;
    // state, stage sums and the last evaluation's coordinates back to the batch's arrays
    DpArgs a = {};
    a.c64 = f.c64;
    a.c32 = f.c32;
    a.npad = f.npad;
    a.fp32c = 1;
#pragma unroll
    for (int u = 0; u < PASSES; u++) {
        const int q = w.c[u];
        if (q < 0) continue;
        const int li = lo + w.row[u];
        const size_t i = (size_t)cl.off + li;
        f.y[q * N + i] = w.y[u];
        if (q < 3)
            write_coord(a, cl, q, cl.poff + li, w.st[u]);
        else if (coul) {
            f.coul1[(q - 3) * N + i] = w.p1[u];
            f.coulS[(q - 3) * N + i] = w.p7[u];
        }
    }
    if (r == 0 && tid == 0) {
        f.ctrl[c] = sh.cs;
        if (f.ran != nullptr && coul) f.ran[c] = 1;
    }
}

// The kernel with enough slots per thread for mc own ions.  Clusters: one slot covers clouds
// of up to 1,344 ions on 16 CTAs; the others keep more of them in registers (six: the
// largest clouds on 4 CTAs).
typedef void (*FusedKernel)(SgFusedArgs, int);
FusedKernel cluster_kernel(int mc) {
    return 6 * mc <= kThreads       ? fused_attempts_kernel<1, false>
           : 6 * mc <= 2 * kThreads ? fused_attempts_kernel<2, false>
                                    : fused_attempts_kernel<6, false>;
}

// Dynamic shared memory any launch asks for at most (clusters: 2,048 ions on 8 CTAs; wide:
// SG_FUSED_WIDE_IONS).  Every kernel is allowed it once and for all: a launch of one thread
// cannot lower another's.
constexpr size_t kMaxSmem = smem_bytes(SG_FUSED_MAX_IONS, SG_FUSED_MAX_IONS / 8, false);
constexpr size_t kMaxWide = smem_bytes(SG_FUSED_WIDE_IONS, kThreads / 6 / 4 * 4, true);

}  // namespace

int sg_fused_cluster_size(int max_npad, int n_clouds) {
    int found = 0;
    for (int R = SG_FUSED_MAX_CTAS; R >= 2; R /= 2) {
        const int mc = own_ions(max_npad, R);
        const size_t smem = smem_bytes(max_npad, mc, false);
        if (mc > kThreads || smem > kMaxSmem) continue;
        const FusedKernel kernel = cluster_kernel(mc);
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                cudaSuccess ||
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kMaxSmem) != cudaSuccess)
            continue;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(R);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = R;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int active = 0;
        if (cudaOccupancyMaxActiveClusters(&active, kernel, &cfg) != cudaSuccess || active <= 0)
            continue;
        found = R;
        if (active >= n_clouds) return R;
    }
    cudaGetLastError();
    return -found;
}

int sg_fused_wide_ctas(int max_npad, int n_clouds, int n_sm) {
    if (max_npad > SG_FUSED_WIDE_IONS) return 0;
    // no more CTAs than groups of four ions
    const int R = std::min({n_sm / n_clouds, max_npad / 4, SG_FUSED_MAX_WIDE});
    if (R < 1 || 6 * own_ions(max_npad, R) > kThreads) return 0;
    const size_t smem = smem_bytes(max_npad, own_ions(max_npad, R), true);
    int per_sm = 0;
    if (cudaFuncSetAttribute(fused_attempts_kernel<1, true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxWide) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fused_attempts_kernel<1, true>,
                                                      kThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return per_sm > 0 ? R : 0;
}

cudaError_t sg_fused_attempts(const SgFusedArgs& f, int ctas, int max_npad, cudaStream_t st) {
    const bool wide = f.ctas > 0;
    const int mc = own_ions(max_npad, ctas);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(f.n_clouds * ctas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_bytes(max_npad, mc, wide);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (wide) {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    } else {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = ctas;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, wide ? fused_attempts_kernel<1, true> : cluster_kernel(mc), f, mc);
}
