// fp64_pairs.cuh -- the FP64 pair sum over unordered pairs, shared by the resident and
// stand-alone Coulomb sums (coulomb.cu), the allocation-free entry point (noalloc.cu) and
// the CUNBODY slot (aux_kernels.cu).
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM sub-partition (2 lanes per
// clock and SM), so the sum is bound by its count of FP64 instructions alone: everything
// else -- shared-memory reads, shuffles, the SFU's 1/sqrt seed -- hides under them.  Taking
// each unordered pair once halves the differences, r^2 and 1/r^3: 12 instructions shared by
// the two ions, 3 per side, 1 more per side where the charges differ -- 9 (10) per ordered
// pair against 16 when every ordered pair is evaluated (and 19 in the form before, with
// its FP32 seed and conversions).
//
// A block of four warps, one per sub-partition, holds 128 i-ions, one per lane.  The ions
// of a 32-ion j-tile travel through the lanes: at step s lane l pairs its i-ion with j-ion
// (l + s) mod 32, whose running sum it gets from lane l + 1 by shuffle, so no two lanes
// ever add to the same j-ion and the order of every sum is fixed.  The four warps' j-side
// sums are added in warp order and stored to the i-block's own slot; the i-side sums stay
// in registers over the item's j-tiles.
//
// Measured: 1,000 ions 26.1 us (ordered pairs: 47.3), 5,003 ions 499 us (1,029).
//
// Small sets have too few such items for the device.  There a block takes one pair of
// 32-ion tiles, a quarter of the rotation steps in each warp, and adds the warps' parts
// before it stores them: an ion has npad / 32 + 1 slots (1,000 ions: 33, where eighths of a
// 128 x 32 item's steps as items of their own left it 264 slots to sum).  The smallest sets
// share a pair's steps between two or four blocks.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fp32c_math.cuh"
#include "sg_internal.cuh"

namespace {

struct Fp64SymShared {
    double tj[4][32];      // x, y, z, charge weight of the j-tile
    double sj[4][3][32];   // per warp: its sums for the j-tile's ions
    double si[4][3][32];   // (tile pairs) ... for the i-tile's
};

// One step's pair: i-side sums a, j-side sums b (subtracted: the pair's force changes
// sign).  SOFT: r^2 + eps2, and a coincident pair without softening contributes nothing.
template <bool NOQ, bool SOFT>
__device__ __forceinline__ void sym_pair(double xi, double yi, double zi, double qi, double xj,
                                         double yj, double zj, double qj, double eps2, bool jside,
                                         double& ax, double& ay, double& az, double& bx,
                                         double& by, double& bz) {
    const double dx = xi - xj, dy = yi - yj, dz = zi - zj;
    double r2 = SOFT ? fma(dx, dx, eps2) : dx * dx;
    r2 = fma(dz, dz, fma(dy, dy, r2));
    double w = inv_r3_fp64(r2);
    if (SOFT && !(r2 > 0.0)) w = 0.0;
    const double wi = NOQ ? w : w * qj;
    ax = fma(wi, dx, ax);
    ay = fma(wi, dy, ay);
    az = fma(wi, dz, az);
    if (jside) {
        const double wj = NOQ ? w : w * qi;
        bx = fma(-wj, dx, bx);
        by = fma(-wj, dy, by);
        bz = fma(-wj, dz, bz);
    }
}

// One 32-ion j-tile against the warp's 32 i-ions, rotation steps [s0, s1).  DIAG: the tile
// is the warp's own ions; steps 1..15 meet every unordered pair but those half a turn
// apart, which step 16 meets from both sides (i-side only), and step 0 is the self pair.
template <bool NOQ, bool SOFT, bool DIAG>
__device__ __forceinline__ void sym_tile(const double (*tj)[32], int s0, int s1, double xi,
                                         double yi, double zi, double qi, double eps2, double& ax,
                                         double& ay, double& az, double* sx, double* sy,
                                         double* sz) {
    const int lane = threadIdx.x & 31, next = (lane + 1) & 31;
    const int b0 = DIAG ? max(s0, 1) : s0, b1 = DIAG ? min(s1, 17) : s1;
    double bx = 0.0, by = 0.0, bz = 0.0;
#pragma unroll 2
    for (int s = b0; s < b1; s++) {
        const int j = (lane + s) & 31;
        sym_pair<NOQ, SOFT>(xi, yi, zi, qi, tj[0][j], tj[1][j], tj[2][j], NOQ ? 1.0 : tj[3][j],
                            eps2, !DIAG || s < 16, ax, ay, az, bx, by, bz);
        bx = __shfl_sync(0xffffffffu, bx, next);
        by = __shfl_sync(0xffffffffu, by, next);
        bz = __shfl_sync(0xffffffffu, bz, next);
    }
    const int j = (lane + max(b0, b1)) & 31;
    sx[j] = bx;
    sy[j] = by;
    sz[j] = bz;
}

// One work item by a block of 128 threads: i-ions [i0, i0 + 128) against j-ions
// [j0, j0 + nj) of a cloud, local padded indices (i0 a multiple of 128, j0 and nj of 32,
// j0 >= i0).  ld(a, k): x, y, z, q (a = 0..3) of local ion k; n real of npad ions (the
// padding ones carry charge 0).  uniform: every real ion has charge qs, and the sums are
// taken with weights 1 and scaled at the end.  pi, pj: the i-side and j-side slots,
// [3][ps] from the cloud's first padded ion.
template <bool SOFT, class Load>
__device__ __forceinline__ void fp64_sym_block(const Load& ld, int n, int npad, int i0, int j0,
                                               int nj, bool uniform, double qs, double eps2, double* __restrict__ pi,
                                               double* __restrict__ pj, size_t ps,
                                               Fp64SymShared& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int iw = i0 + 32 * warp;     // the warp's first ion
    const bool mine = iw < npad;       // npad is a multiple of 32: whole warps
    double xi = 0.0, yi = 0.0, zi = 0.0, qi = 0.0, ax = 0.0, ay = 0.0, az = 0.0;
    if (mine) {
        const int k = iw + lane;
        xi = ld(0, k);
        yi = ld(1, k);
        zi = ld(2, k);
        qi = ld(3, k);
        if (uniform) qi = qi != 0.0 ? 1.0 : 0.0;
    }
    for (int jt = j0; jt < j0 + nj; jt += 32) {
        __syncthreads();  // the previous tile's sums have been stored
        {
            double v = ld(warp, jt + lane);
            if (warp == 3 && uniform) v = v != 0.0 ? 1.0 : 0.0;
            sh.tj[warp][lane] = v;
        }
        __syncthreads();
        double(*sj)[32] = sh.sj[warp];
        // all weights 1: no padding ion on either side
        const bool noq = uniform && jt + 32 <= n && iw + 32 <= n;
        if (!mine || jt < iw) {
            sj[0][lane] = sj[1][lane] = sj[2][lane] = 0.0;
        } else if (jt == iw) {
            sym_tile<false, SOFT, true>(sh.tj, 0, 32, xi, yi, zi, qi, eps2, ax, ay, az, sj[0],
                                        sj[1], sj[2]);
        } else if (noq) {
            sym_tile<true, SOFT, false>(sh.tj, 0, 32, xi, yi, zi, qi, eps2, ax, ay, az, sj[0],
                                        sj[1], sj[2]);
        } else {
            sym_tile<false, SOFT, false>(sh.tj, 0, 32, xi, yi, zi, qi, eps2, ax, ay, az, sj[0],
                                         sj[1], sj[2]);
        }
        __syncthreads();
        if (warp < 3) {
            double v = sh.sj[0][warp][lane] + sh.sj[1][warp][lane];
            v += sh.sj[2][warp][lane];
            v += sh.sj[3][warp][lane];
            pj[warp * ps + (size_t)(jt + lane)] = uniform ? v * qs : v;
        }
    }
    if (mine) {
        const size_t k = (size_t)(iw + lane);
        pi[k] = uniform ? ax * qs : ax;
        pi[ps + k] = uniform ? ay * qs : ay;
        pi[2 * ps + k] = uniform ? az * qs : az;
    }
}

// Part `part` of `parts` (a power of two up to 4) of one pair of 32-ion tiles, i0 <= j0, by
// a block of 128 threads; arguments as above.
template <bool SOFT, class Load>
__device__ __forceinline__ void fp64_sym_tile_block(const Load& ld, int n, int i0, int j0,
                                                    int part, int parts, bool uniform, double qs, double eps2,
                                                    double* __restrict__ pi,
                                                    double* __restrict__ pj, size_t ps,
                                                    Fp64SymShared& sh) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double xi = ld(0, i0 + lane), yi = ld(1, i0 + lane), zi = ld(2, i0 + lane);
    double qi = ld(3, i0 + lane), ax = 0.0, ay = 0.0, az = 0.0;
    if (uniform) qi = qi != 0.0 ? 1.0 : 0.0;
    {
        double v = ld(warp, j0 + lane);
        if (warp == 3 && uniform) v = v != 0.0 ? 1.0 : 0.0;
        sh.tj[warp][lane] = v;
    }
    __syncthreads();
    double(*sj)[32] = sh.sj[warp];
    const int steps = 8 / parts, s0 = steps * (4 * part + warp), s1 = s0 + steps;
    if (j0 == i0)
        sym_tile<false, SOFT, true>(sh.tj, s0, s1, xi, yi, zi, qi, eps2, ax, ay, az, sj[0], sj[1],
                                    sj[2]);
    else if (uniform && j0 + 32 <= n)  // all weights 1
        sym_tile<true, SOFT, false>(sh.tj, s0, s1, xi, yi, zi, qi, eps2, ax, ay, az, sj[0], sj[1],
                                    sj[2]);
    else
        sym_tile<false, SOFT, false>(sh.tj, s0, s1, xi, yi, zi, qi, eps2, ax, ay, az, sj[0], sj[1],
                                     sj[2]);
    sh.si[warp][0][lane] = ax;
    sh.si[warp][1][lane] = ay;
    sh.si[warp][2][lane] = az;
    __syncthreads();
    if (warp < 3) {
        double v = (sh.si[0][warp][lane] + sh.si[1][warp][lane]) +
                   (sh.si[2][warp][lane] + sh.si[3][warp][lane]);
        double u = (sh.sj[0][warp][lane] + sh.sj[1][warp][lane]) +
                   (sh.sj[2][warp][lane] + sh.sj[3][warp][lane]);
        pi[warp * ps + (size_t)(i0 + lane)] = uniform ? v * qs : v;
        pj[warp * ps + (size_t)(j0 + lane)] = uniform ? u * qs : u;
    }
}

// Sets with fewer 128 x 32 blocks than this per SM take tile pairs.  A Dormand-Prince
// attempt, us, 128 x 32 items (in eighths where there are few) / tile pairs: 64 ions 78 / 64,
// 300 92 / 83, 1,000 231 / 187, 1,500 323 / 320, 2,000 567 / 503, 3,000 1,036 / 1,015, 4,000 1,749
// / 1,707, 5,003 2,615 / 2,670.
constexpr double kSymTilePairs = 16.0;
// Blocks that share a tile pair: what makes the last round of blocks over the SMs shortest,
// at 8 % a doubling for the slots it adds (a diagonal pair counts half).  us per attempt in one / two / four parts: 64 ions
// 91 / 73 / 64, 400 99 / 95 / 91, 600 128 / 116 / 114, 700 128 / 134 / 134, 1,000 198 / 187 /
// 204, 1,200 229 / 239 / 263, 32 clouds of 100 148 / 153 / 155.
inline int sym_parts(double tile_pairs, int n_sm) {
    int best = 1;
    double least = 1e300;
    for (int parts = 1; parts <= 4; parts *= 2) {
        const double cost = std::ceil(parts * tile_pairs / n_sm) / parts * (parts == 1 ? 1.0 : parts == 2 ? 1.08 : 1.17);
        if (cost < least) {
            least = cost;
            best = parts;
        }
    }
    return best;
}

// ---- one set of ions on its own (allocation-free entry point, CUNBODY slot) -----------
// Work items of one set of npad ions, in the order of their i-blocks: K j-tiles each, or
// (K = 0) pairs of 32-ion tiles in `parts` parts.
struct SymPlan {
    int K, parts, items, slots;
};

__host__ __device__ inline int sym_chunks(int npad, int b, int K) {
    return (npad / SG_SYM_JT - b * (SG_SYM_IB / SG_SYM_JT) + K - 1) / K;
}

// The plan for a device of n_sm SMs whose slots hold at most cap doubles: at least 4
// items per SM (as plan_sym in capi.cu), more j-tiles per item until the slots fit.
inline SymPlan sym_plan(int npad, int n_sm, size_t cap) {
    const int nb = (npad + SG_SYM_IB - 1) / SG_SYM_IB, nt = npad / SG_SYM_JT;
    double tiles = 0.0;
    for (int b = 0; b < nb; b++) tiles += sym_chunks(npad, b, 1);
    const int parts = sym_parts(0.5 * nt * nt, n_sm);
    if (tiles < kSymTilePairs * n_sm && (size_t)(nt + 1) * parts * 3 * npad <= cap)
        return SymPlan{0, parts, nt * (nt + 1) / 2 * parts, (nt + 1) * parts};
    SymPlan p{std::max(1, (int)(tiles / (16.0 * n_sm))), 1, 0, 0};
    for (;;) {
        p.items = p.slots = 0;
        for (int b = 0; b < nb; b++) {
            const int q = sym_chunks(npad, b, p.K);
            p.items += q;
            p.slots = std::max(p.slots, b + 1 + q);
        }
        if ((size_t)p.slots * 3 * npad <= cap || p.K >= nt) return p;
        p.K++;
    }
}

template <bool SOFT, class Load>
__global__ void __launch_bounds__(SG_SYM_IB) sym_set_kernel(Load ld, int n, int npad, SymPlan p,
                                                            bool uniform, double qs, double eps2,
                                                            double* part) {
    __shared__ Fp64SymShared sh;
    const size_t slot = (size_t)3 * npad;
    int it = blockIdx.x, b = 0;
    if (p.K == 0) {
        const int band = it % p.parts;
        it /= p.parts;
        int q = npad / SG_SYM_JT;
        while (it >= q) {
            it -= q--;
            b++;
        }
        fp64_sym_tile_block<SOFT>(ld, n, 32 * b, 32 * (b + it), band, p.parts, uniform, qs, eps2,
                                  part + ((b + it + 1) * p.parts + band) * slot,
                                  part + (b * p.parts + band) * slot, (size_t)npad, sh);
        return;
    }
    int q = sym_chunks(npad, 0, p.K);
    while (it >= q) {
        it -= q;
        q = sym_chunks(npad, ++b, p.K);
    }
    const int j0 = b * SG_SYM_IB + it * p.K * SG_SYM_JT;
    fp64_sym_block<SOFT>(ld, n, npad, b * SG_SYM_IB, j0, min(p.K * SG_SYM_JT, npad - j0), uniform,
                         qs, eps2, part + (b + 1 + it) * slot, part + b * slot, (size_t)npad, sh);
}

// out[i][c] = scale[i] (or f) times the sum of ion i's slots, [slot][3][npad]: R ions a
// block, 256 / R threads each (thread g takes slots g, g + 256 / R, ...), then pairwise.
// p.K == 0: every ion has p.slots slots.
template <int R>
__global__ void __launch_bounds__(256) sym_sum_kernel(const double* __restrict__ part, int n,
                                                             int npad, SymPlan p,
                                                             const double* __restrict__ scale,
                                                             double f, double* __restrict__ out) {
    constexpr int G = 256 / R;
    __shared__ double v[G][3][R + 1];
    const int r = threadIdx.x % R, g = threadIdx.x / R;
    const int i = blockIdx.x * R + r;
    double s[3] = {0.0, 0.0, 0.0};
    if (i < n) {
        const int b = i / SG_SYM_IB;
        const int ns = p.K ? b + 1 + sym_chunks(npad, b, p.K) : p.slots;
#pragma unroll 4
        for (int sl = g; sl < ns; sl += G)
#pragma unroll
            for (int c = 0; c < 3; c++) s[c] += part[((size_t)sl * 3 + c) * npad + i];
    }
    for (int h = G / 2; h > 0; h >>= 1) {
        if (g >= h && g < 2 * h)
            for (int c = 0; c < 3; c++) v[g][c][r] = s[c];
        __syncthreads();
        if (g < h)
            for (int c = 0; c < 3; c++) s[c] += v[g + h][c][r];
    }
    if (g == 0 && i < n) {
        const double w = scale ? scale[i] : f;
        for (int c = 0; c < 3; c++) out[3 * (size_t)i + c] = w * s[c];
    }
}

}  // namespace
