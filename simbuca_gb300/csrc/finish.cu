// finish.cu -- small batches: the slot sums, the flagged ions' FP64 rows and the
// Dormand-Prince stage in one launch after each pair kernel.
//
// Batches of up to SG_FINISH_MAX_IONS ions wait for launches and dependent chains, not for
// throughput: with the reduction (its flagged rows one after the other in the block that
// owns them) and the stage as launches of their own a 1,000-ion stage took 14.5 + 7.3 us;
// here 15.4 us.  A block owns 16 ions; 16 threads per ion sum its partial-sum slots;
// then a thread per ion and component takes the stage (dp_stage.cuh).
//
// Flagged ions (FP32c).  A row of n FP64 pairs is 16 instructions of 64 cycles per 32
// pairs on one of an SM's four sub-partitions: the eight blocks of a cluster take an
// eighth of every flagged row of the cluster each, through a list in the first block's
// shared memory, and the owner adds the eight parts in rank order.
//
// The rows read the coordinates of the current stage while other blocks already write
// the next stage's: stage S reads coordinate set S mod 2 and writes the other one.
#include <cooperative_groups.h>

#include "dp_stage.cuh"
#include "fp32c_math.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kRows = 16;                 // ions per block
constexpr int kThr = 256;
constexpr int kPer = kThr / kRows;        // threads per ion in the slot sums
constexpr int kCluster = 8;
constexpr int kList = kCluster * kRows;   // flagged ions of a cluster at most

struct FinishShared {
    union {
        float v[kThr][9];        // FP32c slot sums: hi x, y, z, lo x, y, z, s2 (8: padding)
        double v64[kThr][3];     // FP64 slot sums
        double row[3][kThr];     // a flagged row's partial sums
    };
    double P[3][kRows];          // Coulomb sums of the block's ions (SI)
    double part[kList][3];       // this block's eighth of each flagged row
    int list[kList][2];          // (first block) flagged ions: cloud, owner's rank << 8 | row
    int ig[kList];               // ... and padded index
    int nlist;
    int mine[kList][2], mig[kList];  // this block's copy of the list
};

// The slots of this block's rows into sh.P; FP32c: kind of fix-up of this thread's row
// (threads below kRows).
template <bool F32>
__device__ __forceinline__ bool slot_sums(const SgFinishArgs& f, const SgCloud& cl,
                                          const SgRowBlock& rb, FinishShared& sh) {
    const int tid = threadIdx.x, row = tid & (kRows - 1), g = tid / kRows;
    const size_t NP = (size_t)f.dp.npad;
    const int ig = cl.poff + (rb.i0 - cl.off) + row;
    bool flagged = false;
    if constexpr (F32) {
        ff p[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
        float s2 = 0.f;
        if (row < rb.n) {
            const float* Q0 = reinterpret_cast<const float*>(f.part) + ig;
#pragma unroll 2
            for (int sl = g; sl < cl.nslots; sl += kPer) {
                const float* Q = Q0 + (size_t)sl * SG_PART_F32 * NP;
#pragma unroll
                for (int c = 0; c < 3; c++) p[c] = ff_add(p[c], {Q[c * NP], Q[(3 + c) * NP]});
                s2 += Q[6 * NP];
            }
        }
        // the two ions' halves of a warp: lanes l and l + 16 hold parts of the same row
#pragma unroll
        for (int c = 0; c < 3; c++) {
            ff o;
            o.h = __shfl_down_sync(0xffffffffu, p[c].h, 16);
            o.l = __shfl_down_sync(0xffffffffu, p[c].l, 16);
            p[c] = ff_add(p[c], o);
        }
        s2 += __shfl_down_sync(0xffffffffu, s2, 16);
        if ((tid & 31) < 16) {
            float* v = sh.v[tid];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                v[c] = p[c].h;
                v[3 + c] = p[c].l;
            }
            v[6] = s2;
        }
        __syncthreads();
        // warp 0: lane (row, half) adds the even / odd warps' parts, then the halves meet
        if (tid < 32) {
            const int half = tid >> 4;
            p[0] = p[1] = p[2] = {0.f, 0.f};
            s2 = 0.f;
#pragma unroll
            for (int w = 0; w < kThr / 64; w++) {
                const float* v = sh.v[32 * (2 * w + half) + row];
#pragma unroll
                for (int c = 0; c < 3; c++) p[c] = ff_add(p[c], {v[c], v[3 + c]});
                s2 += v[6];
            }
#pragma unroll
            for (int c = 0; c < 3; c++) {
                ff o;
                o.h = __shfl_down_sync(0xffffffffu, p[c].h, 16);
                o.l = __shfl_down_sync(0xffffffffu, p[c].l, 16);
                p[c] = ff_add(p[c], o);
            }
            s2 += __shfl_down_sync(0xffffffffu, s2, 16);
            if (tid < rb.n) {
                const double sc = cl.psc;
#pragma unroll
                for (int c = 0; c < 3; c++) sh.P[c][tid] = sc * ((double)p[c].h + (double)p[c].l);
                const float pf2 = fmaf(p[0].h, p[0].h, fmaf(p[1].h, p[1].h, p[2].h * p[2].h));
                flagged = s2 > sg_kappa2(cl.npad) * pf2;
                if (f.risk != nullptr) {
                    const int i = rb.i0 + tid;
                    f.risk[i] = flagged ? -1.f : 0.f;
                    f.risk[(size_t)f.dp.n + i] = flagged ? -1.f : sqrtf(s2 / pf2);
                }
            }
        }
    } else {
        double p[3] = {0.0, 0.0, 0.0};
        if (row < rb.n) {
            const int ns = cl.sym_k ? sg_sym_slots(cl, ig - cl.poff) : cl.nslots;
            const double* Q0 = f.part + ig;
#pragma unroll 4
            for (int sl = g; sl < ns; sl += kPer) {
                const double* Q = Q0 + (size_t)sl * 3 * NP;
#pragma unroll
                for (int c = 0; c < 3; c++) p[c] += Q[c * NP];
            }
        }
#pragma unroll
        for (int c = 0; c < 3; c++) sh.v64[tid][c] = p[c];
        __syncthreads();
        // warp c sums component c: lane (row, half) eight parts, then the halves meet
        if (tid < 96) {
            const int c = tid >> 5, half = (tid >> 4) & 1;
            double s = sh.v64[half * kRows + row][c];
#pragma unroll
            for (int q = 1; q < kPer / 2; q++) s += sh.v64[(2 * q + half) * kRows + row][c];
            s += __shfl_down_sync(0xffffffffu, s, 16);
            if ((tid & 31) < rb.n) sh.P[c][row] = s;
        }
    }
    return flagged;
}

// This block's eighth of a flagged ion's row (padding ions carry no charge) into
// sh.part[k]: warp c adds up component c.
__device__ __forceinline__ void row_part(const SgFinishArgs& f, const SgCloud& cl, int ig, int rank,
                                         int k, FinishShared& sh) {
    const int tid = threadIdx.x;
    const size_t NP = (size_t)f.dp.npad;
    const double* c64 = f.c64r;
    const double xi = c64[ig], yi = c64[NP + ig], zi = c64[2 * NP + ig];
    const int len = (cl.npad / 32 + kCluster - 1) / kCluster * 32;  // whole warps of pairs
    const int j0 = rank * len, j1 = min(cl.npad, j0 + len);
    double ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll 2
    for (int j = j0 + tid; j < j1; j += kThr) {
        const int jg = cl.poff + j;
        if (jg == ig) continue;
        const double rx = xi - c64[jg], ry = yi - c64[NP + jg], rz = zi - c64[2 * NP + jg];
        const double w = c64[3 * NP + jg] * inv_r3_fp64(fma(rz, rz, fma(ry, ry, rx * rx)));
        ax = fma(w, rx, ax);
        ay = fma(w, ry, ay);
        az = fma(w, rz, az);
    }
    __syncthreads();  // the previous row's sums (or the slot sums) have been read
    sh.row[0][tid] = ax;
    sh.row[1][tid] = ay;
    sh.row[2][tid] = az;
    __syncthreads();
    if (tid < 96) {
        const int c = tid >> 5, lane = tid & 31;
        const int nw = min(kThr, max(j1 - j0, 0));
        double s = 0.0;
        for (int t = lane; t < nw; t += 32) s += sh.row[c][t];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) sh.part[k][c] = s;
    }
}

template <int S, bool F32>
__global__ void __launch_bounds__(kThr) finish_kernel(SgFinishArgs f) {
    sg_griddep_wait();
    __shared__ FinishShared sh;
    const DpArgs& a = f.dp;
    const bool exists = blockIdx.x < f.n_rows;  // the grid is padded to whole clusters
    const SgRowBlock rb = a.rows[exists ? blockIdx.x : 0];
    const SgCtrl& cs = a.ctrl[rb.cloud];
    const SgCloud& cl = a.clouds[rb.cloud];
    const bool live = exists && !(cs.done || cs.hold || cs.status != SG_OK);
    const bool coul = live && (cl.fp.flags & SG_F_COULOMB);
    const int tid = threadIdx.x;
    if constexpr (F32) {
        cg::cluster_group cluster = cg::this_cluster();
        const int rank = (int)cluster.block_rank();
        FinishShared* first = cluster.map_shared_rank(&sh, 0);
        if (tid == 0) sh.nlist = 0;
        auto token = cluster.barrier_arrive();
        bool flagged = false;
        if (coul) flagged = slot_sums<true>(f, cl, rb, sh);
        cluster.barrier_wait(std::move(token));  // the first block's list is ready
        if (flagged) {
            const int at = atomicAdd(&first->nlist, 1);
            first->list[at][0] = rb.cloud;
            first->list[at][1] = rank << 8 | tid;
            first->ig[at] = cl.poff + (rb.i0 - cl.off) + tid;
            if (f.counters != nullptr) atomicAdd(f.counters, 1);
        }
        cluster.sync();
        const int nf = first->nlist;
        if (nf > 0) {
            for (int k = tid; k < nf; k += kThr) {
                sh.mine[k][0] = first->list[k][0];
                sh.mine[k][1] = first->list[k][1];
                sh.mig[k] = first->ig[k];
            }
            __syncthreads();
            for (int k = 0; k < nf; k++)
                row_part(f, a.clouds[sh.mine[k][0]], sh.mig[k], rank, k, sh);
            cluster.sync();
            for (int q = tid; q < 3 * nf; q += kThr) {
                const int k = q / 3, c = q - 3 * k;
                if (sh.mine[k][1] >> 8 != rank) continue;
                double s = 0.0;
                for (int r = 0; r < kCluster; r++) s += cluster.map_shared_rank(&sh, r)->part[k][c];
                sh.P[c][sh.mine[k][1] & 255] = s;
            }
        }
        if (coul && f.ran != nullptr && tid == 0) f.ran[rb.cloud] = 1;
    } else {
        if (coul) slot_sums<false>(f, cl, rb, sh);
    }
    __syncthreads();
    if (live) {
        const SgFieldCoef fk = a.fcoef[rb.cloud * SG_MAX_STAGES + S];
        const int row = tid & (kRows - 1), c = tid < 8 * kRows ? stage_component(tid / kRows, kRows) : -1;
        const bool active = row < rb.n && c >= 0;
        const size_t N = (size_t)a.n;
        const int i = rb.i0 + row;
        double v = 0.0, sol = 0.0;
        if (active) {
            const double P = c >= 3 && coul ? sh.P[c - 3][row] : 0.0;
            v = stage_one<S, MethodDP>(a, cl, cs, fk, c, i, P, sol);
            if (S == 7 && c >= 3 && coul) {
                a.coul7[(c - 3) * N + i] = P;
                f.coulS[(c - 3) * N + i] = P;  // the in-run check's sums
            }
        }
        if constexpr (S == 7) {
            v = stage_block_sum(active ? v : 0.0);
            if (tid == 0) a.err_part[blockIdx.x] = v;
        } else {
            __syncthreads();  // this stage's state has been read
            if (active) {
                a.ys[c * N + i] = v;
                if (c < 3) write_coord(a, cl, c, cl.poff + (i - cl.off), v);
            }
        }
    }
    if constexpr (F32) cg::this_cluster().sync();  // other blocks may still read this one's parts
}

template <int S>
cudaError_t launch(const SgFinishArgs& f, int fp32c, cudaStream_t st) {
    if (!fp32c) return sg_launch(finish_kernel<S, false>, f.n_rows, kThr, 0, st, f);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((f.n_rows + kCluster - 1) / kCluster * kCluster);
    cfg.blockDim = dim3(kThr);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kCluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, finish_kernel<S, true>, f);
}

}  // namespace

cudaError_t sg_dp_finish(const SgFinishArgs& f, int stage, int fp32c, cudaStream_t st) {
    if (f.n_rows <= 0) return cudaSuccess;
    switch (stage) {
        case 2: return launch<2>(f, fp32c, st);
        case 3: return launch<3>(f, fp32c, st);
        case 4: return launch<4>(f, fp32c, st);
        case 5: return launch<5>(f, fp32c, st);
        case 6: return launch<6>(f, fp32c, st);
        case 7: return launch<7>(f, fp32c, st);
        default: return cudaErrorInvalidValue;
    }
}
