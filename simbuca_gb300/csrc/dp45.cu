// dp45.cu -- Dormand-Prince 5(4) stage, error-norm and step-control kernels of
// libsimgb (sm_103a), plus the O(N) helpers of the stand-alone force calls.
//
// Device layout (FP64, structure of arrays over all ions of all clouds, N ions):
//   y   [6][N]     state at the step start: x, y, z, vx, vy, vz  (IonCloud::pos/vel)
//   ys  [6][N]     stage state (IonCloud::pos2/vel2)
//   k   [7][6][N]  stage derivatives: stage velocity, stage acceleration (_ode_vars::k1..k7)
//   coul1, coul7 [3][N]  Coulomb sums P of stage 1 and stage 7
// The Coulomb inputs of the next stage are written by the stage kernel itself:
//   c64 [4][Npad] SI x, y, z, q;  c32 [7][Npad] frame hi x, y, z, q, lo x, y, z.
//
// One attempt = stage1, (coulomb, stage s) for s = 2..7, control, commit.  The stage-1
// Coulomb sum is never recomputed: after an accepted step the positions of stage 1
// are those of stage 7 (coul1 <- coul7), after a rejected one they are unchanged.
// The force count still follows the reference (7 per attempt, bin/ode.cpp:101-175).
#include <math.h>

#include <algorithm>

#include "dp_stage.cuh"

namespace {

__device__ __forceinline__ void write_coords(const DpArgs& a, const SgCloud& cl, int ig,
                                             double x, double y, double z, float* hu = nullptr) {
    a.c64[ig] = x;
    a.c64[a.npad + ig] = y;
    a.c64[2 * (size_t)a.npad + ig] = z;
    if (a.fp32c) {
        const double u = (x - cl.cx) * cl.invL, v = (y - cl.cy) * cl.invL,
                     w = (z - cl.cz) * cl.invL;
        const float uh = __double2float_rn(u), vh = __double2float_rn(v),
                    wh = __double2float_rn(w);
        a.c32[ig] = uh;
        a.c32[a.npad + ig] = vh;
        a.c32[2 * (size_t)a.npad + ig] = wh;
        a.c32[4 * (size_t)a.npad + ig] = __double2float_rn(u - (double)uh);
        a.c32[5 * (size_t)a.npad + ig] = __double2float_rn(v - (double)vh);
        a.c32[6 * (size_t)a.npad + ig] = __double2float_rn(w - (double)wh);
        if (hu) {
            hu[0] = uh;
            hu[1] = vh;
            hu[2] = wh;
        }
    }
}


// Bounds of the 128-ion tiles covered by a row block (256 ions = 2 tiles of the cloud):
// min/max of the FP32 frame coordinates of the block's real ions.
__device__ __forceinline__ void tile_bounds(const DpArgs& a, const SgCloud& cl,
                                            const SgRowBlock& rb, bool active, float u,
                                            float v, float w) {
    __shared__ float sb[SG_ROWS / 32][6];
    float b[6] = {active ? u : INFINITY, active ? v : INFINITY, active ? w : INFINITY,
                  active ? u : -INFINITY, active ? v : -INFINITY, active ? w : -INFINITY};
    for (int o = 16; o > 0; o >>= 1)
        for (int q = 0; q < 6; q++) {
            const float x = __shfl_xor_sync(0xffffffffu, b[q], o);
            b[q] = q < 3 ? fminf(b[q], x) : fmaxf(b[q], x);
        }
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
        for (int q = 0; q < 6; q++) sb[warp][q] = b[q];
    __syncthreads();
    if (threadIdx.x < 2) {
        const int h = threadIdx.x;                 // tile 0 or 1 of this row block
        float r[6];
        for (int q = 0; q < 6; q++) r[q] = sb[4 * h][q];
        for (int wv = 4 * h + 1; wv < 4 * h + 4; wv++)
            for (int q = 0; q < 6; q++) r[q] = q < 3 ? fminf(r[q], sb[wv][q]) : fmaxf(r[q], sb[wv][q]);
        const int local = rb.i0 - cl.off;          // multiple of SG_ROWS
        const int tile = local / 128 + h;
        if (local + 128 * h < cl.n) {
            float* B = a.bbox + 8 * (size_t)(cl.tile0 + tile);
            for (int q = 0; q < 6; q++) B[q] = r[q];
        }
    }
}

// ---- stage kernels -------------------------------------------------------------------
// A thread per ion and component: component slots of R threads each, R the rows of the
// block (a power of two >= 16); at R = 16 the slots are laid out so that the four warps,
// one per SM sub-partition, hold x and y, z, a_x and a_y, a_z.
//
// GB300 takes 64 cycles for every FP64 warp instruction, so a stage costs the FP64
// instructions of its longest warp, times the warps per sub-partition.  A thread per ion
// ran all six components' ~100 instructions on one warp of a block, behind one thread's
// drive cosines and divisions (a 1,000-ion stage: 8.4 - 15.1 us, 32 busy sub-partitions of
// 608); per component the longest chain is ~20 instructions (7.3 us), and the first
// stage computes every stage's field coefficients, a lane each.
// Field coefficients of stage S for the whole block.  The first stage of an attempt takes
// all of them, lane s - 1 of the first warp stage s, and leaves the others' in a.fcoef
// (`publish`: the cloud's first block).  Every thread of the block must call this.
template <int S, class M>
__device__ __forceinline__ SgFieldCoef stage_coef(const DpArgs& a, const SgCloud& cl,
                                                  const SgCtrl& cs, int cloud, bool publish) {
    if constexpr (S == 1) {
        __shared__ SgFieldCoef sk;
        if (threadIdx.x < M::stages) {
            const int s = threadIdx.x + 1;
            const bool frozen = (cl.fp.flags & SG_F_FROZEN_T) != 0;
            const SgFieldCoef k = sg_field_coef(cl.fp, frozen ? cs.t : cs.t + M::c(s) * cs.h);
            if (s == 1) sk = k;
            if (publish) a.fcoef[cloud * SG_MAX_STAGES + s] = k;
        }
        __syncthreads();
        return sk;
    } else {
        return a.fcoef[cloud * SG_MAX_STAGES + S];
    }
}

// Large batches: a thread per ion, all six components, R = 128 rows a block (one 128-ion
// tile of the k-d order).  Throughput-bound by the FP64 pipe, where a thread per component
// only adds barriers and loads (65,536 ions: 24 - 28 us a stage; this form 17 - 20 us).
template <int S, class M>
__global__ void __launch_bounds__(128) stage_wide_kernel(DpArgs a) {
    sg_griddep_wait();
    constexpr bool last = S == M::stages;
    SgRowBlock rb = a.rows[blockIdx.x / a.split];
    const int sub = blockIdx.x % a.split;
    rb.i0 += sub * 128;
    rb.n = min(rb.n - sub * 128, 128);
    const SgCtrl& cs = a.ctrl[rb.cloud];
    if (cs.done || cs.hold || cs.status != SG_OK) return;
    const SgCloud& cl = a.clouds[rb.cloud];
    const SgFieldCoef fk = stage_coef<S, M>(a, cl, cs, rb.cloud, rb.i0 == cl.off);
    const int row = threadIdx.x, i = rb.i0 + row;
    const bool active = row < rb.n;
    const size_t N = (size_t)a.n;
    double v[6], acc2 = 0.0;
    float hu[3] = {0.f, 0.f, 0.f};
    if (active) {
        double P[3] = {0.0, 0.0, 0.0};
        if (cl.fp.flags & SG_F_COULOMB) {
            const double* co = M::stages == 7 && S == 1 ? a.coul1 : a.coulS;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                P[c] = co[c * N + i];
                if (M::stages == 7 && last) a.coul7[c * N + i] = P[c];
            }
        }
#pragma unroll
        for (int c = 0; c < 6; c++) {
            double sol = 0.0;
            v[c] = stage_one<S, M>(a, cl, cs, fk, c, i, c < 3 ? 0.0 : P[c - 3], sol);
            if (last) acc2 += v[c];
            if (last && M::stages == 6) v[c] = sol;
        }
        if (!last || M::stages == 6)
#pragma unroll
            for (int c = 0; c < 6; c++) {
                a.ys[c * N + i] = v[c];
                if (!last && c < 3) hu[c] = write_coord(a, cl, c, cl.poff + (i - cl.off), v[c]);
            }
    }
    if constexpr (last) {
        acc2 = stage_block_sum(acc2);
        if (threadIdx.x == 0) a.err_part[blockIdx.x] = acc2;
    } else if (a.fp32c && a.bbox) {
        __shared__ float sb[4][6];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            float lo = active ? hu[c] : INFINITY, hi = active ? hu[c] : -INFINITY;
            for (int o = 16; o > 0; o >>= 1) {
                lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
                hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            }
            if ((threadIdx.x & 31) == 0) {
                sb[threadIdx.x >> 5][c] = lo;
                sb[threadIdx.x >> 5][3 + c] = hi;
            }
        }
        __syncthreads();
        if (threadIdx.x < 6 && rb.n > 0) {
            const int q = threadIdx.x;
            a.bbox[8 * (size_t)(cl.tile0 + (rb.i0 - cl.off) / 128) + q] =
                q < 3 ? fminf(fminf(sb[0][q], sb[1][q]), fminf(sb[2][q], sb[3][q]))
                      : fmaxf(fmaxf(sb[0][q], sb[1][q]), fmaxf(sb[2][q], sb[3][q]));
        }
    }
}

// Stage S of a block's rows, the Coulomb sums in coul1 (Dormand-Prince's first stage) or
// coulS.
template <int S, class M>
__global__ void __launch_bounds__(6 * 32) stage_kernel(DpArgs a) {
    sg_griddep_wait();
    constexpr bool last = S == M::stages;
    SgRowBlock rb = a.rows[blockIdx.x / a.split];
    const int R = rb.cap / a.split, sub = blockIdx.x % a.split;
    rb.i0 += sub * R;
    rb.n = min(rb.n - sub * R, R);
    const SgCtrl& cs = a.ctrl[rb.cloud];
    if (cs.done || cs.hold || cs.status != SG_OK) return;
    const SgCloud& cl = a.clouds[rb.cloud];
    const SgFieldCoef fk = stage_coef<S, M>(a, cl, cs, rb.cloud, rb.i0 == cl.off);
    const int row = threadIdx.x & (R - 1), c = stage_component(threadIdx.x / R, R);
    const bool active = row < rb.n && c >= 0;
    const size_t N = (size_t)a.n;
    const int i = rb.i0 + row;
    double v = 0.0, sol = 0.0;
    if (active) {
        double P = 0.0;
        if (c >= 3 && (cl.fp.flags & SG_F_COULOMB)) {
            P = (M::stages == 7 && S == 1 ? a.coul1 : a.coulS)[(c - 3) * N + i];
            if (M::stages == 7 && last) a.coul7[(c - 3) * N + i] = P;
        }
        v = stage_one<S, M>(a, cl, cs, fk, c, i, P, sol);
    }
    if (!last || M::stages == 6) {
        __syncthreads();  // this stage's state has been read
        if (active) {
            a.ys[c * N + i] = last ? sol : v;
            if (!last && c < 3) write_coord(a, cl, c, cl.poff + (i - cl.off), v);
        }
    }
    if constexpr (last) {
        v = stage_block_sum(active ? v : 0.0);
        if (threadIdx.x == 0) a.err_part[blockIdx.x] = v;
    }
}

// ---- Gear predictor-corrector, the reference's GearMethod (bin/ode.cpp:347-424) ----
// Fifth-order Nordsieck form with one force evaluation per step and a fixed step.
// Gear state in k, by column: acceleration of the last force call [0..2], b [3..5],
// c [6..8], d [9..11].  The e terms of the reference are never read there; left out.
#define SG_GEA0 (3.0 / 20.0)
#define SG_GEA1 (251.0 / 360.0)
#define SG_GEA3 (11.0 / 18.0)
#define SG_GEA4 (1.0 / 6.0)
#define SG_GEA5 (1.0 / 60.0)

// InitAcceleraction (bin/ode.cpp:36-59): constant seeds for every ion of a cloud but the
// last in the caller's order (left as allocated there, zero here); b = c = d = 0.
__global__ void __launch_bounds__(SG_ROWS) gear_init_kernel(DpArgs a, const int* __restrict__ perm) {
    sg_griddep_wait();
    const SgRowBlock rb = a.rows[blockIdx.x];
    const SgCloud& cl = a.clouds[rb.cloud];
    const int li = threadIdx.x;
    if (li >= rb.n) return;
    const int i = rb.i0 + li;
    const size_t N = (size_t)a.n;
    const int caller = perm ? perm[i] : i;
    const bool last = caller == cl.off + cl.n - 1;
    a.k[i] = last ? 0.0 : 1.6e9;
    a.k[N + i] = last ? 0.0 : 1.1e9;
    a.k[2 * N + i] = last ? 0.0 : -5e8;
#pragma unroll
    for (int c = 3; c < 12; c++) a.k[c * N + i] = 0.0;
}

template <int PHASE>
__global__ void __launch_bounds__(SG_ROWS) gear_kernel(DpArgs a) {
    sg_griddep_wait();
    const SgRowBlock rb = a.rows[blockIdx.x];
    const SgCtrl& cs = a.ctrl[rb.cloud];
    if (cs.done || cs.hold || cs.status != SG_OK) return;
    const SgCloud& cl = a.clouds[rb.cloud];
    const int li = threadIdx.x;
    const bool active = li < rb.n;
    const int i = rb.i0 + (active ? li : 0);
    const int ig = cl.poff + (i - cl.off);
    const size_t N = (size_t)a.n;
    const double h = cs.h;
    const double h2f = cs.hf[0], h3f = cs.hf[1], h4f = cs.hf[2], h5f = cs.hf[3];
    float hu[3] = {0.f, 0.f, 0.f};
    int bad = 0;
    if (active) {
        if (PHASE == 0) {
            // predictor: Taylor series of the Nordsieck vector (bin/ode.cpp:367-375)
            double p2[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const double ac = a.k[c * N + i], b = a.k[(3 + c) * N + i];
                const double cc = a.k[(6 + c) * N + i], d = a.k[(9 + c) * N + i];
                const double x = a.y[c * N + i], v = a.y[(3 + c) * N + i];
                p2[c] = x + v * h + ac * h2f + b * h3f + cc * h4f + d * h5f;
                a.ys[c * N + i] = p2[c];
                a.ys[(3 + c) * N + i] = v + ac * h + b * h2f + cc * h3f + d * h4f;
            }
            write_coords(a, cl, ig, p2[0], p2[1], p2[2], hu);
        } else {
            // corrector (bin/ode.cpp:396-420) with the force at the predicted state
            const bool frozen = (cl.fp.flags & SG_F_FROZEN_T) != 0;
            const double ts = frozen ? cs.t : cs.t + h;
            double st[6];
#pragma unroll
            for (int c = 0; c < 6; c++) st[c] = a.ys[c * N + i];
            double f[3];
            sg_field_accel(cl.fp, ts, a.qm[i], st[0], st[1], st[2], st[3], st[4], st[5], f[0],
                           f[1], f[2]);
            if (cl.fp.flags & SG_F_COULOMB) {
                const double kqi = a.kq[i];
#pragma unroll
                for (int c = 0; c < 3; c++) f[c] += kqi * a.coulS[c * N + i];
            }
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const double ac = a.k[c * N + i], b = a.k[(3 + c) * N + i];
                const double cc = a.k[(6 + c) * N + i], d = a.k[(9 + c) * N + i];
                const double sug = ac + b * h + cc * h2f + d * h3f;
                const double bn = b + cc * h + d * h2f;
                const double cn = cc + d * h;
                const double ad = h2f * (f[c] - sug);
                const double x = st[c] + SG_GEA0 * ad;
                const double v = st[3 + c] + SG_GEA1 * ad / h;
                a.ys[c * N + i] = x;
                a.ys[(3 + c) * N + i] = v;
                a.k[c * N + i] = f[c];
                a.k[(3 + c) * N + i] = bn + SG_GEA3 * ad / h3f;
                a.k[(6 + c) * N + i] = cn + SG_GEA4 * ad / h4f;
                a.k[(9 + c) * N + i] = d + SG_GEA5 * ad / h5f;
                bad |= !isfinite(x) || !isfinite(v);
            }
        }
    }
    if (PHASE == 0) {
        if (a.fp32c && a.bbox) tile_bounds(a, cl, rb, active, hu[0], hu[1], hu[2]);
    } else {
        // no error estimate: the partial is 0, or NaN when the step left finite numbers
        bad = __syncthreads_or(bad);
        if (threadIdx.x == 0) a.err_part[blockIdx.x] = bad ? __longlong_as_double(0x7ff8000000000000LL) : 0.0;
    }
}

// error_succes + step bookkeeping (bin/ode.cpp:426-494), one warp per cloud: its lanes
// sum the error partials, lane 0 decides.
// With flags[SG_FLAG_HOLD] set, a cloud that accepts holds (skips further attempts) until
// the host clears the hold: used to take exactly one step per cloud.
__global__ void dp_control_kernel(SgCloud* __restrict__ clouds, SgCtrl* __restrict__ ctrl,
                                  const double* __restrict__ err_part, int split,
                                  const double* __restrict__ y, int n_clouds,
                                  const int* __restrict__ flags, const SgOp* __restrict__ ops) {
    sg_griddep_wait();
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (c >= n_clouds) return;
    const SgCloud& cl = clouds[c];
    const int nb = cl.nrb * split;
    const double* ep = err_part + (size_t)cl.rb0 * split;
    double s = 0.0;
    for (int b = lane; b < nb; b += 32) s += ep[b];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane != 0) return;
    SgCtrl cs = ctrl[c];
    if (cs.done || cs.hold || cs.status != SG_OK) {
        ctrl[c].accepted = 0;
        ctrl[c].print_due = 0;
        return;
    }
    cs.print_due = 0;
    // Cash-Karp: the reference adds to the previous norm, odev.err is never reset there
    if (cs.method == 4) s += cs.err;
    const double err = sqrt(s / (6 * cl.n));
    cs.err = err;
    cs.force_evals += (cs.method == 4) ? 6 : (cs.method == 1 ? 1 : 7);
    cs.coulomb_evals += (cl.fp.flags & SG_F_COULOMB) ? (cs.method == 1 ? 1 : 6) : 0;
    int accepted = 1;
    if (flags[SG_FLAG_ERR] != 0) {
        // a kernel of this attempt gave up a bounded wait: its sums are incomplete, so
        // the attempt is neither accepted nor used for step control
        cs.status = flags[SG_FLAG_ERR];
        cs.done = 1;
        accepted = 0;
    } else {
        // IonCloud::pos[0][0] (bin/ode.cpp:482): x of the caller's first ion
        accepted = sg_error_succes(cs, err, y + cl.ion0);
    }
    if (accepted) {
        cs.h_last = cs.h;
        cs.t = cs.t + cs.h;
        cs.h = cs.hnext;
        cs.steps++;
        cs.rejects_here = 0;
        int print_now = 0;
        if (cs.n_ops > 0) {
            cs.dis_due = 0;
            if (cs.t >= cs.t_end) {
                // the operation has ended: print after it, start the next one
                print_now = ops[cs.op_index].print_after;
                print_now |= sg_start_ops(cs, clouds[c].fp, ops, cs.op_index + 1);
            } else if (ops[cs.op_index].kind == SG_OP_TRAP_RAMP) {
                // Vrf/Vdc for the next step (bin/ion_fly.cpp:95-99)
                const SgOp& op = ops[cs.op_index];
                const double ramp = (cs.t - cs.t_op_start) / (cs.t_end - cs.t_op_start);
                clouds[c].fp.Vrf = cs.old_vrf * (1 - ramp) + op.new_vrf * ramp;
                clouds[c].fp.Vdc = cs.old_vdc * (1 - ramp) + op.new_vdc * ramp;
            }
        } else if (cs.t >= cs.t_end) {
            cs.done = 1;
        }
        if (flags[SG_FLAG_HOLD]) cs.hold |= 1;
        // the reference prints after a step once (t - start) > interval * prints so far
        // (bin/ion_fly.cpp:103-108); the record goes to the next ring slot, and a full
        // ring holds the cloud until the host has drained it
        const bool rule = cs.print_interval > 0.0 &&
                          (cs.t - cs.t_print0) > cs.print_interval * (double)cs.n_print;
        if (cs.rec_cap > 0 && (rule || print_now)) {
            if (rule) cs.n_print++;
            if (cs.rec_count - cs.rec_drained < cs.rec_cap) {
                cs.print_due = 1;
                cs.rec_slot = (int)(cs.rec_count % cs.rec_cap);
                cs.rec_count++;
            }
            if (cs.rec_count - cs.rec_drained >= cs.rec_cap) cs.hold |= 2;
        }
    }
    cs.accepted = accepted;
    ctrl[c] = cs;
}

__global__ void clear_hold_kernel(SgCtrl* ctrl, int n_clouds) {
    sg_griddep_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < n_clouds) ctrl[c].hold &= ~1;
}

// Commit an accepted attempt: pos <- pos2, vel <- vel2 (bin/ode.cpp:488-489) and the
// stage-7 Coulomb sum becomes the next stage-1 sum.
__global__ void __launch_bounds__(SG_ROWS) dp_commit_kernel(DpArgs a) {
    sg_griddep_wait();
    const SgRowBlock rb = a.rows[blockIdx.x];
    if (!a.ctrl[rb.cloud].accepted) return;
    const int li = threadIdx.x;
    if (li >= rb.n) return;
    const int i = rb.i0 + li;
    const size_t N = (size_t)a.n;
#pragma unroll
    for (int c = 0; c < 6; c++) a.y[c * N + i] = a.ys[c * N + i];
#pragma unroll
    for (int c = 0; c < 3; c++) a.coul1[c * N + i] = a.coul7[c * N + i];
}

// Coulomb inputs of the state y (set-up and stand-alone calls); ghosts get q = 0.
__global__ void __launch_bounds__(SG_ROWS) coords_from_state_kernel(DpArgs a,
                                                                    const double* __restrict__ q) {
    sg_griddep_wait();
    const SgRowBlock rb = a.rows[blockIdx.x];
    const SgCloud& cl = a.clouds[rb.cloud];
    const int li = threadIdx.x;
    const size_t N = (size_t)a.n;
    // this block also covers the ghost tail of its cloud when it holds the cloud's last row
    const bool last = (rb.i0 + rb.n == cl.off + cl.n);
    float hu[3] = {0.f, 0.f, 0.f};
    if (li < rb.n) {
        const int i = rb.i0 + li;
        const int ig = cl.poff + (i - cl.off);
        write_coords(a, cl, ig, a.y[i], a.y[N + i], a.y[2 * N + i], hu);
        a.c64[3 * (size_t)a.npad + ig] = q[i];
        if (a.fp32c) a.c32[3 * (size_t)a.npad + ig] = (float)(q[i] / cl.qscale);
    }
    if (a.fp32c && a.bbox) tile_bounds(a, cl, rb, li < rb.n, hu[0], hu[1], hu[2]);
    if (last) {
        for (int g = cl.n + li; g < cl.npad; g += blockDim.x) {
            const int ig = cl.poff + g;
            // far away, no charge: contributes exactly zero as a j-ion
            const double far = 1.0e3 + 1.0e-3 * g;
            a.c64[ig] = far;
            a.c64[a.npad + ig] = far;
            a.c64[2 * (size_t)a.npad + ig] = far;
            a.c64[3 * (size_t)a.npad + ig] = 0.0;
            if (a.fp32c) {
                const float ff = sg_pad_frame(g);
                a.c32[ig] = ff;
                a.c32[a.npad + ig] = ff;
                a.c32[2 * (size_t)a.npad + ig] = ff;
                a.c32[3 * (size_t)a.npad + ig] = 0.f;
                a.c32[4 * (size_t)a.npad + ig] = 0.f;
                a.c32[5 * (size_t)a.npad + ig] = 0.f;
                a.c32[6 * (size_t)a.npad + ig] = 0.f;
            }
        }
    }
}

// Stand-alone force: out[i][c] (AoS) = field(t) + kq_i * sum_slots P (if Coulomb).
__global__ void __launch_bounds__(SG_ROWS) force_finish_kernel(DpArgs a, double t,
                                                               int with_field,
                                                               const int* __restrict__ perm,
                                                               double* __restrict__ out) {
    sg_griddep_wait();
    const SgRowBlock rb = a.rows[blockIdx.x];
    const SgCloud& cl = a.clouds[rb.cloud];
    const int li = threadIdx.x;
    if (li >= rb.n) return;
    const int i = rb.i0 + li;
    const size_t N = (size_t)a.n;
    double cx = 0.0, cy = 0.0, cz = 0.0;
    if (cl.fp.flags & SG_F_COULOMB) {
        cx = a.coulS[i];
        cy = a.coulS[N + i];
        cz = a.coulS[2 * N + i];
    }
    double fx = 0.0, fy = 0.0, fz = 0.0;
    if (with_field)
        sg_field_accel(cl.fp, t, a.qm[i], a.y[i], a.y[N + i], a.y[2 * N + i], a.y[3 * N + i],
                       a.y[4 * N + i], a.y[5 * N + i], fx, fy, fz);
    const double kqi = a.kq[i];
    const size_t o = 3 * (size_t)(perm ? perm[i] : i);
    out[o + 0] = fx + kqi * cx;
    out[o + 1] = fy + kqi * cy;
    out[o + 2] = fz + kqi * cz;
}

// AoS host layout -> SoA state (positions and velocities).
// y[c][k] = pos[perm[k]][c]: the caller's order into the device (sorted) order.
__global__ void aos_to_soa_kernel(const double* __restrict__ pos, const double* __restrict__ vel,
                                  const int* __restrict__ perm, double* __restrict__ y, int n) {
    sg_griddep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t N = (size_t)n;
    const size_t s = 3 * (size_t)(perm ? perm[i] : i);
    for (int c = 0; c < 3; c++) {
        y[c * N + i] = pos[s + c];
        y[(3 + c) * N + i] = vel ? vel[s + c] : 0.0;
    }
}

// pos[perm[k]][c] = y[c][k]: back to the caller's order.
__global__ void soa_to_aos_kernel(const double* __restrict__ y, const int* __restrict__ perm,
                                  double* __restrict__ pos, double* __restrict__ vel, int n) {
    sg_griddep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const size_t N = (size_t)n;
    const size_t d = 3 * (size_t)(perm ? perm[i] : i);
    for (int c = 0; c < 3; c++) {
        pos[d + c] = y[c * N + i];
        vel[d + c] = y[(3 + c) * N + i];
    }
}

__global__ void gather_kernel(const double* __restrict__ src, const int* __restrict__ perm,
                              double* __restrict__ dst, int n) {
    sg_griddep_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[perm ? perm[i] : i];
}

// Per-row-block moment partials: sum x, x^2 per axis, v^2 per axis, m(vx^2+vy^2), m vz^2.
__global__ void __launch_bounds__(SG_ROWS) moments_kernel(DpArgs a, const double* __restrict__ mass,
                                                          double* __restrict__ out) {
    sg_griddep_wait();
    __shared__ double red[11][SG_ROWS / 32];
    const SgRowBlock rb = a.rows[blockIdx.x];
    const int li = threadIdx.x;
    const size_t N = (size_t)a.n;
    double v[11];
    for (int q = 0; q < 11; q++) v[q] = 0.0;
    if (li < rb.n) {
        const int i = rb.i0 + li;
        for (int c = 0; c < 3; c++) {
            const double x = a.y[c * N + i], u = a.y[(3 + c) * N + i];
            v[c] = x;
            v[3 + c] = x * x;
            v[6 + c] = u * u;
        }
        v[9] = mass[i] * (v[6] + v[7]);
        v[10] = mass[i] * v[8];
    }
    for (int q = 0; q < 11; q++) {
        double s = v[q];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if ((li & 31) == 0) red[q][li >> 5] = s;
    }
    __syncthreads();
    if (li < 11) {
        double s = 0.0;
        for (int w = 0; w < SG_ROWS / 32; w++) s += red[li][w];
        out[(size_t)blockIdx.x * 11 + li] = s;
    }
}

}  // namespace

// ---- host-side launchers (called from capi.cu) ------------------------------------

// Blocks per row block: row blocks of 256 (large batches) take two of 128 rows, a thread
// per ion; the others blocks of 32 (a warp per component) or 16 rows.
int sg_stage_split(int cap) { return cap >= 256 ? 2 : std::max(1, cap / 32); }

template <int S, class M>
static void launch_stage_s(const SgDpArgs& a, int n_rows, int cap, cudaStream_t st) {
    const int R = cap / a.split;
    if (cap >= 256)
        sg_launch(stage_wide_kernel<S, M>, n_rows * a.split, 128, 0, st, a);
    else
        sg_launch(stage_kernel<S, M>, n_rows * a.split, R > 16 ? 6 * R : 8 * R, 0, st, a);
}

template <class M>
static cudaError_t launch_stage(const SgDpArgs& a, int stage, int n_rows, int cap, cudaStream_t st) {
    if (n_rows <= 0) return cudaSuccess;
    switch (stage) {
        case 1: launch_stage_s<1, M>(a, n_rows, cap, st); break;
        case 2: launch_stage_s<2, M>(a, n_rows, cap, st); break;
        case 3: launch_stage_s<3, M>(a, n_rows, cap, st); break;
        case 4: launch_stage_s<4, M>(a, n_rows, cap, st); break;
        case 5: launch_stage_s<5, M>(a, n_rows, cap, st); break;
        case 6: launch_stage_s<6, M>(a, n_rows, cap, st); break;
        case 7:
            if constexpr (M::stages == 7) launch_stage_s<7, M>(a, n_rows, cap, st);
            break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t sg_dp_stage(const SgDpArgs& a, int stage, int n_rows, int cap, cudaStream_t st) {
    return launch_stage<MethodDP>(a, stage, n_rows, cap, st);
}

cudaError_t sg_ck_stage(const SgDpArgs& a, int stage, int n_rows, int cap, cudaStream_t st) {
    return launch_stage<MethodCK>(a, stage, n_rows, cap, st);
}

cudaError_t sg_gear_stage(const SgDpArgs& a, int phase, int n_rows, cudaStream_t st) {
    if (n_rows <= 0) return cudaSuccess;
    if (phase == 0)
        sg_launch(gear_kernel<0>, n_rows, SG_ROWS, 0, st, a);
    else
        sg_launch(gear_kernel<1>, n_rows, SG_ROWS, 0, st, a);
    return cudaGetLastError();
}

cudaError_t sg_gear_init(const SgDpArgs& a, const int* perm, int n_rows, cudaStream_t st) {
    if (n_rows <= 0) return cudaSuccess;
    sg_launch(gear_init_kernel, n_rows, SG_ROWS, 0, st, a, perm);
    return cudaGetLastError();
}

cudaError_t sg_dp_control(SgCloud* clouds, SgCtrl* ctrl, const double* err_part,
                          int split, const double* y, int n_clouds, const int* flags,
                          const SgOp* ops, cudaStream_t st) {
    sg_launch(dp_control_kernel, (n_clouds + 3) / 4, 128, 0, st, clouds, ctrl, err_part, split, y,
              n_clouds, flags, ops);
    return cudaGetLastError();
}

cudaError_t sg_clear_hold(SgCtrl* ctrl, int n_clouds, cudaStream_t st) {
    sg_launch(clear_hold_kernel, (n_clouds + 127) / 128, 128, 0, st, ctrl, n_clouds);
    return cudaGetLastError();
}

cudaError_t sg_dp_commit(const SgDpArgs& a, int n_rows, cudaStream_t st) {
    sg_launch(dp_commit_kernel, n_rows, SG_ROWS, 0, st, a);
    return cudaGetLastError();
}

cudaError_t sg_coords_from_state(const SgDpArgs& a, const double* q, int n_rows, cudaStream_t st) {
    sg_launch(coords_from_state_kernel, n_rows, SG_ROWS, 0, st, a, q);
    return cudaGetLastError();
}

cudaError_t sg_force_finish(const SgDpArgs& a, double t, int with_field, const int* perm,
                            double* out, int n_rows, cudaStream_t st) {
    sg_launch(force_finish_kernel, n_rows, SG_ROWS, 0, st, a, t, with_field, perm, out);
    return cudaGetLastError();
}

cudaError_t sg_aos_to_soa(const double* pos, const double* vel, const int* perm, double* y, int n,
                          cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    sg_launch(aos_to_soa_kernel, (n + 255) / 256, 256, 0, st, pos, vel, perm, y, n);
    return cudaGetLastError();
}

cudaError_t sg_soa_to_aos(const double* y, const int* perm, double* pos, double* vel, int n,
                          cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    sg_launch(soa_to_aos_kernel, (n + 255) / 256, 256, 0, st, y, perm, pos, vel, n);
    return cudaGetLastError();
}

cudaError_t sg_gather(const double* src, const int* perm, double* dst, int n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    sg_launch(gather_kernel, (n + 255) / 256, 256, 0, st, src, perm, dst, n);
    return cudaGetLastError();
}

cudaError_t sg_moments(const SgDpArgs& a, const double* mass, double* out, int n_rows,
                       cudaStream_t st) {
    sg_launch(moments_kernel, n_rows, SG_ROWS, 0, st, a, mass, out);
    return cudaGetLastError();
}

