// proposer.cu -- the learned step-size proposer: per-cloud features, an MLP
// 16 -> 64 -> 64 -> 1 with SiLU activations, BF16 weights and FP32 accumulation, its
// training kernels (forward + backward + Adam), and the step-history log it learns from.
//
// After every Dormand-Prince attempt the proposer kernel (one warp per cloud):
//   * on an accepted step, appends (features of the step start, h of the previous
//     step, h and error norm of this step) to the cloud's log and recomputes the
//     features from the new state;
//   * when the proposer is on, replaces the controller's next step size h_c by
//     safety * h * exp(MLP(features)), clamped to [0.2, 10] x h and to [1/2, 2] x h_c:
//     the reference's controller stays the fallback, so features outside the training
//     range (a tiny error norm after tiny steps, say) cannot drive h down step after step.
// Rejected attempts keep the reference's reject rule (bin/ode.cpp:451-455): every step
// is still accepted or rejected by the embedded Dormand-Prince error estimate.
//
// Features (all O(1)):  0-2 centroid / L;  3-5 RMS spread / L - 1;  6-8 RMS velocity
// / v0 - 1 (L, v0: frame scale and RMS velocity at upload);  9 log10(h_last) + 8;
// 10 log10(err_last) (>= -8);  11 rejects of the last step;  12-13 cos/sin of the
// active drive's phase;  14 +1 quadrupole / -1 dipole / 0 none;  15 log10(h_last/h_prev).
// The target of a logged step is log(h_k err_k^-0.2 / h_{k-1}): the ratio to the
// previous step of the step size that would have met the tolerance exactly.
#include <cuda_bf16.h>

#include <algorithm>

#include "fp32c_math.cuh"
#include "sg_internal.cuh"

namespace {

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
    const float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// MLP forward of one feature vector by one warp; returns the output on every lane.
__device__ float mlp_warp(const __nv_bfloat16* __restrict__ w, const float* x) {
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* W1 = w + SG_MLP_W1;
    const __nv_bfloat16* B1 = w + SG_MLP_B1;
    const __nv_bfloat16* W2 = w + SG_MLP_W2;
    const __nv_bfloat16* B2 = w + SG_MLP_B2;
    const __nv_bfloat16* W3 = w + SG_MLP_W3;
    float h1[2], h2[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int u = lane + 32 * r;
        float z = __bfloat162float(B1[u]);
#pragma unroll
        for (int k = 0; k < SG_MLP_IN; k++) z = fmaf(__bfloat162float(W1[u * SG_MLP_IN + k]), x[k], z);
        h1[r] = silu(z);
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int u = lane + 32 * r;
        float z = __bfloat162float(B2[u]);
        for (int m = 0; m < SG_MLP_H; m++) {
            const float hm = __shfl_sync(0xffffffffu, h1[m >> 5], m & 31);
            z = fmaf(__bfloat162float(W2[u * SG_MLP_H + m]), hm, z);
        }
        h2[r] = silu(z);
    }
    float o = __bfloat162float(W3[lane]) * h2[0] + __bfloat162float(W3[lane + 32]) * h2[1];
    for (int off = 16; off > 0; off >>= 1) o += __shfl_xor_sync(0xffffffffu, o, off);
    return o + __bfloat162float(w[SG_MLP_B3]);
}

// Per-cloud features from the moment partials of moments_kernel.
__device__ void cloud_features(const SgCloud& cl, const SgCtrl& cs, const double* mom,
                               const SgProposerState& ps, float* f) {
    double s[11];
    for (int q = 0; q < 11; q++) s[q] = 0.0;
    for (int b = 0; b < cl.nmb; b++)
        for (int q = 0; q < 11; q++) s[q] += mom[(size_t)(cl.mb0 + b) * 11 + q];
    const double n = cl.n;
    const double L = cl.L, v0 = cl.vref > 0.0 ? cl.vref : 1.0;
    for (int c = 0; c < 3; c++) {
        const double m = s[c] / n;
        const double var = s[3 + c] / n - m * m;
        f[c] = (float)((m - (c == 0 ? cl.cx : c == 1 ? cl.cy : cl.cz)) / L);
        f[3 + c] = (float)((var > 0 ? sqrt(var) : 0.0) / L - 1.0);
        f[6 + c] = (float)(sqrt(s[6 + c] / n) / v0 - 1.0);
    }
    const double hl = cs.h_last > 0 ? cs.h_last : cs.h;
    f[9] = (float)(log10(hl) + 8.0);
    f[10] = (float)fmax(log10(fmax(cs.err, 1e-30)), -8.0);
    f[11] = (float)ps.rejects_in_step;
    const sg_field_params& fp = cl.fp;
    const double t = cs.t;
    double ph = 0.0, kind = 0.0;
    if ((fp.flags & SG_F_QUAD) && t >= fp.tq_on && t < fp.tq_off) {
        ph = 2.0 * SG_PI * fp.nu_q * t + fp.phi_q;
        kind = 1.0;
    } else if ((fp.flags & SG_F_DIPOLE) && t >= fp.td_on && t < fp.td_off) {
        ph = 2.0 * SG_PI * fp.nu_d * t + fp.phi_d;
        kind = -1.0;
    }
    f[12] = kind != 0.0 ? (float)cos(ph) : 0.f;
    f[13] = kind != 0.0 ? (float)sin(ph) : 0.f;
    f[14] = (float)kind;
    f[15] = ps.h_prev > 0 ? (float)log10(hl / ps.h_prev) : 0.f;
}

// One warp per cloud, after the commit of an attempt.
__global__ void proposer_kernel(const SgCloud* __restrict__ clouds, SgCtrl* __restrict__ ctrl,
                                const double* __restrict__ mom, SgProposerState* __restrict__ pst,
                                const __nv_bfloat16* __restrict__ w, float* __restrict__ log_feat,
                                double* __restrict__ log_num, int log_cap, int use_mlp,
                                double safety, int n_clouds) {
    sg_griddep_wait();
    const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (c >= n_clouds) return;
    SgCtrl cs = ctrl[c];
    SgProposerState ps = pst[c];
    const SgCloud& cl = clouds[c];
    // a fresh upload marks the state with init == 0: features of the first step
    if (!ps.init) {
        float f[SG_MLP_IN];
        cloud_features(cl, cs, mom, ps, f);
        if (lane == 0) {
            for (int k = 0; k < SG_MLP_IN; k++) pst[c].feat[k] = f[k];
            pst[c].init = 1;
        }
        return;
    }
    if (cs.status != SG_OK) return;
    if (!cs.accepted) {
        // a rejected attempt: remember it for the features; the reject rule stands
        if (lane == 0 && !cs.done && !cs.hold) pst[c].rejects_in_step = ps.rejects_in_step + 1;
        return;
    }
    // accepted: log (features at the step start, h_prev, h, err)
    if (lane == 0 && log_cap > 0 && ps.logged < log_cap) {
        const long long r = (long long)c * log_cap + ps.logged;
        for (int k = 0; k < SG_MLP_IN; k++) log_feat[r * SG_MLP_IN + k] = ps.feat[k];
        log_num[r * 4 + 0] = ps.h_prev;
        log_num[r * 4 + 1] = cs.h_last;
        log_num[r * 4 + 2] = cs.err;
        log_num[r * 4 + 3] = cs.t;
    }
    SgProposerState nps = ps;
    nps.logged = (log_cap > 0 && ps.logged < log_cap) ? ps.logged + 1 : ps.logged;
    nps.h_prev = cs.h_last;
    nps.rejects_in_step = 0;
    float f[SG_MLP_IN];
    cloud_features(cl, cs, mom, ps, f);
    if (use_mlp == 2 && !cs.done) {
        // the controller's rule with another safety factor (the ablation of the MLP)
        if (lane == 0) ctrl[c].h = safety * cs.h;
    } else if (use_mlp && !cs.done) {
        const float o = mlp_warp(w, f);
        const double lo = log(0.2), hi = log(10.0);
        const double r = fmin(fmax((double)o, lo), hi);
        const double h_ctrl = cs.h;  // the controller's next step (bin/ode.cpp:443-446)
        const double h_mlp = safety * cs.h_last * exp(r);
        if (lane == 0) ctrl[c].h = fmin(fmax(h_mlp, 0.5 * h_ctrl), 2.0 * h_ctrl);
    }
    if (lane == 0) {
        for (int k = 0; k < SG_MLP_IN; k++) nps.feat[k] = f[k];
        pst[c] = nps;
    }
}

// ---- training ----------------------------------------------------------------
// Forward + backward of a batch; block b takes samples [b*per, (b+1)*per) (of the
// index list idx), kTrainChunk at a time, and writes its gradient partial to
// gpart[b][SG_MLP_NP] and its squared-error sum to lpart[b].  MSE loss
// L = (1/B) sum (o - y)^2.
//
// Latency-bound: a minibatch of 256 is 4 M multiply-adds.  Each layer of a chunk is one
// product with a thread per (sample, unit), the weights (FP32 images of the BF16 values)
// and activations in shared memory, W2 with a row stride of 65 words so that both
// W2[u][m] over u (forward) and over m (backward) are conflict-free; each thread keeps
// the 16 + 4 weight gradients it owns in registers.  With one thread per whole sample
// and shared-memory atomics for every weight gradient (32 busy threads in each of 8
// blocks, activations in local memory) a minibatch of 256 took 7,347 us; this form, 64
// blocks of one chunk, takes 13.5 us.
constexpr int kTrainThreads = 256;
constexpr int kTrainChunk = 4;  // kTrainThreads / SG_MLP_H samples in flight per block
constexpr int kW2Stride = SG_MLP_H + 1;

struct TrainShared {
    float W1[SG_MLP_H][SG_MLP_IN + 1];
    float W2[SG_MLP_H * kW2Stride];
    float B1[SG_MLP_H], B2[SG_MLP_H], W3[SG_MLP_H];
    float x[kTrainChunk][SG_MLP_IN];
    float h1[kTrainChunk][SG_MLP_H], h2[kTrainChunk][SG_MLP_H];
    float gz1[kTrainChunk][SG_MLP_H], gz2[kTrainChunk][SG_MLP_H];
    float osum[kTrainThreads / 32];
    float go[kTrainChunk];
};

__global__ void __launch_bounds__(kTrainThreads) mlp_grad_kernel(
    const __nv_bfloat16* __restrict__ w, const float* __restrict__ X, const float* __restrict__ Y,
    const int* __restrict__ idx, int B, int per, float* __restrict__ gpart,
    float* __restrict__ lpart) {
    sg_griddep_wait();
    __shared__ TrainShared sh;
    const int tid = threadIdx.x;
    for (int k = tid; k < SG_MLP_H * SG_MLP_IN; k += kTrainThreads)
        sh.W1[k / SG_MLP_IN][k % SG_MLP_IN] = __bfloat162float(w[SG_MLP_W1 + k]);
    for (int k = tid; k < SG_MLP_H * SG_MLP_H; k += kTrainThreads)
        sh.W2[k / SG_MLP_H * kW2Stride + k % SG_MLP_H] = __bfloat162float(w[SG_MLP_W2 + k]);
    if (tid < SG_MLP_H) {
        sh.B1[tid] = __bfloat162float(w[SG_MLP_B1 + tid]);
        sh.B2[tid] = __bfloat162float(w[SG_MLP_B2 + tid]);
        sh.W3[tid] = __bfloat162float(w[SG_MLP_W3 + tid]);
    }
    const float b3 = __bfloat162float(w[SG_MLP_B3]);
    const int u = tid % SG_MLP_H, s = tid / SG_MLP_H;  // unit, sample of the chunk
    // this thread's weight gradients: W2[s*16 + r][u], W1[tid / 4][(tid % 4) * 4 + r]
    float g2[SG_MLP_H / kTrainChunk], g1[SG_MLP_H * SG_MLP_IN / kTrainThreads];
    float gb1 = 0.f, gb2 = 0.f, gw3 = 0.f, gb3 = 0.f, lerr = 0.f;
#pragma unroll
    for (int r = 0; r < SG_MLP_H / kTrainChunk; r++) g2[r] = 0.f;
#pragma unroll
    for (int r = 0; r < SG_MLP_H * SG_MLP_IN / kTrainThreads; r++) g1[r] = 0.f;
    const int s0 = blockIdx.x * per, s1 = min(B, s0 + per);
    for (int c0 = s0; c0 < s1; c0 += kTrainChunk) {
        const int nc = min(kTrainChunk, s1 - c0);
        __syncthreads();  // weights loaded; the previous chunk's arrays are free
        if (tid < kTrainChunk * SG_MLP_IN) {
            const int q = tid / SG_MLP_IN;
            const int at = q < nc ? (idx ? idx[c0 + q] : c0 + q) : -1;
            sh.x[q][tid % SG_MLP_IN] = at >= 0 ? X[(size_t)at * SG_MLP_IN + tid % SG_MLP_IN] : 0.f;
        }
        __syncthreads();
        float z1 = sh.B1[u];
#pragma unroll
        for (int k = 0; k < SG_MLP_IN; k++) z1 = fmaf(sh.W1[u][k], sh.x[s][k], z1);
        sh.h1[s][u] = silu(z1);
        __syncthreads();
        float z2 = sh.B2[u];
#pragma unroll 16
        for (int m = 0; m < SG_MLP_H; m++) z2 = fmaf(sh.W2[u * kW2Stride + m], sh.h1[s][m], z2);
        const float h2 = silu(z2);
        sh.h2[s][u] = h2;
        float o = sh.W3[u] * h2;
        for (int off = 16; off > 0; off >>= 1) o += __shfl_xor_sync(0xffffffffu, o, off);
        if ((tid & 31) == 0) sh.osum[tid >> 5] = o;
        __syncthreads();
        if (tid < kTrainChunk) {
            float go = 0.f;
            if (tid < nc) {
                const int at = idx ? idx[c0 + tid] : c0 + tid;
                const float d = sh.osum[2 * tid] + sh.osum[2 * tid + 1] + b3 - Y[at];
                lerr += d * d;
                go = 2.0f * d / (float)B;
            }
            sh.go[tid] = go;  // 0 past the batch: no gradient from there
            gb3 += go;
        }
        __syncthreads();
        sh.gz2[s][u] = sh.go[s] * sh.W3[u] * silu_grad(z2);
        __syncthreads();
        float gh = 0.f;
#pragma unroll 16
        for (int q = 0; q < SG_MLP_H; q++) gh = fmaf(sh.W2[q * kW2Stride + u], sh.gz2[s][q], gh);
        sh.gz1[s][u] = gh * silu_grad(z1);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kTrainChunk; q++) {
            const float hm = sh.h1[q][u];
#pragma unroll
            for (int r = 0; r < SG_MLP_H / kTrainChunk; r++)
                g2[r] = fmaf(sh.gz2[q][s * (SG_MLP_H / kTrainChunk) + r], hm, g2[r]);
            const float g = sh.gz1[q][tid / 4];
#pragma unroll
            for (int r = 0; r < SG_MLP_H * SG_MLP_IN / kTrainThreads; r++)
                g1[r] = fmaf(g, sh.x[q][(tid % 4) * 4 + r], g1[r]);
            if (s == 0) {
                gb1 += sh.gz1[q][u];
                gb2 += sh.gz2[q][u];
                gw3 = fmaf(sh.go[q], sh.h2[q][u], gw3);
            }
        }
    }
    float* gp = gpart + (size_t)blockIdx.x * SG_MLP_NP;
#pragma unroll
    for (int r = 0; r < SG_MLP_H / kTrainChunk; r++)
        gp[SG_MLP_W2 + (s * (SG_MLP_H / kTrainChunk) + r) * SG_MLP_H + u] = g2[r];
#pragma unroll
    for (int r = 0; r < SG_MLP_H * SG_MLP_IN / kTrainThreads; r++)
        gp[SG_MLP_W1 + (tid / 4) * SG_MLP_IN + (tid % 4) * 4 + r] = g1[r];
    if (s == 0) {
        gp[SG_MLP_B1 + u] = gb1;
        gp[SG_MLP_B2 + u] = gb2;
        gp[SG_MLP_W3 + u] = gw3;
    }
    if (tid < 32) {  // the chunk's per-sample threads are lanes 0-3 of this warp
        for (int off = 2; off > 0; off >>= 1) {
            lerr += __shfl_down_sync(0xffffffffu, lerr, off);
            gb3 += __shfl_down_sync(0xffffffffu, gb3, off);
        }
        if (tid == 0) {
            gp[SG_MLP_B3] = gb3;
            lpart[blockIdx.x] = lerr;
        }
    }
}

// Sum of the nb block partials p[b * stride], in order and compensated: 64 to 128 plain FP32
// additions added more rounding than the pass before them (relative l2 error of a gradient over
// 256 / 2,000 samples 1.4e-7 / 1.7e-7, so 0.7e-7 / 0.4e-7; 0.4 us of an iteration's 30).
__device__ __forceinline__ float block_partials(const float* __restrict__ p, int stride, int nb) {
    float s = 0.f, c = 0.f;  // the roundings of s in c, off its chain of additions
#pragma unroll 16
    for (int b = 0; b < nb; b++) {
        const ff t = ff_two_sum(s, p[(size_t)b * stride]);
        s = t.h;
        c += t.l;
    }
    return s + c;
}

// grad[k] = sum_b gpart[b][k] (fixed order); loss = sum_b lpart[b] / B.
__global__ void mlp_reduce_kernel(const float* __restrict__ gpart, const float* __restrict__ lpart,
                                  int nb, int B, float* __restrict__ grad, float* __restrict__ loss) {
    sg_griddep_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < SG_MLP_NP) {
        grad[k] = block_partials(gpart + k, SG_MLP_NP, nb);
    }
    if (k == 0) {
        *loss = block_partials(lpart, 1, nb) / (float)B;
    }
}

// One training iteration's end: the gradient (block partials in a fixed order), Adam on
// the FP32 master weights, the BF16 copy used by the next forward pass, and the loss into
// the iteration's history entry.  One launch: with the sums, Adam and the loss read-back
// apart, an iteration was 3 launches, a copy and a host wait.
__global__ void mlp_adam_kernel(float* __restrict__ wm, __nv_bfloat16* __restrict__ wb,
                                float* __restrict__ m1, float* __restrict__ m2,
                                const float* __restrict__ gpart, const float* __restrict__ lpart,
                                int nb, int B, float* __restrict__ loss, float lr, float b1,
                                float b2, float eps, int step) {
    sg_griddep_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < SG_MLP_NP) {
        const float g = block_partials(gpart + k, SG_MLP_NP, nb);
        const float a = b1 * m1[k] + (1.f - b1) * g;
        const float v = b2 * m2[k] + (1.f - b2) * g * g;
        m1[k] = a;
        m2[k] = v;
        const float ah = a / (1.f - powf(b1, (float)step));
        const float vh = v / (1.f - powf(b2, (float)step));
        const float nw = wm[k] - lr * ah / (sqrtf(vh) + eps);
        wm[k] = nw;
        wb[k] = __float2bfloat16_rn(nw);
    } else if (k == SG_MLP_NP) {  // a thread of its own
        *loss = block_partials(lpart, 1, nb) / (float)B;
    }
}

__global__ void mlp_to_bf16_kernel(const float* __restrict__ wm, __nv_bfloat16* __restrict__ wb) {
    sg_griddep_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < SG_MLP_NP) wb[k] = __float2bfloat16_rn(wm[k]);
}

// Inference of a batch: one warp per sample.
__global__ void mlp_forward_kernel(const __nv_bfloat16* __restrict__ w, const float* __restrict__ X,
                                   int n, float* __restrict__ out) {
    sg_griddep_wait();
    const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= n) return;
    float x[SG_MLP_IN];
#pragma unroll
    for (int k = 0; k < SG_MLP_IN; k++) x[k] = X[(size_t)s * SG_MLP_IN + k];
    const float o = mlp_warp(w, x);
    if ((threadIdx.x & 31) == 0) out[s] = o;
}

}  // namespace

cudaError_t sg_proposer_launch(const SgCloud* clouds, SgCtrl* ctrl, const double* mom,
                               SgProposerState* pst, const void* wbf, float* log_feat,
                               double* log_num, int log_cap, int use_mlp, double safety,
                               int n_clouds, cudaStream_t st) {
    const int warps = 4;
    sg_launch(proposer_kernel, (n_clouds + warps - 1) / warps, 32 * warps, 0, st, 
        clouds, ctrl, mom, pst, static_cast<const __nv_bfloat16*>(wbf), log_feat, log_num, log_cap,
        use_mlp, safety, n_clouds);
    return cudaGetLastError();
}

// Blocks of a forward + backward pass over B samples: one chunk of samples each while
// that fits the partial-gradient array (64 blocks for a minibatch of 256: one wave).
static int train_blocks(int B) {
    return std::max(1, std::min(SG_MLP_BLOCKS, (B + kTrainChunk - 1) / kTrainChunk));
}

cudaError_t sg_mlp_grad_launch(const void* wbf, const float* X, const float* Y, const int* idx,
                               int B, float* gpart, float* lpart, float* grad, float* loss,
                               cudaStream_t st) {
    const int nb = train_blocks(B);
    sg_launch(mlp_grad_kernel, nb, kTrainThreads, 0, st, static_cast<const __nv_bfloat16*>(wbf), X, Y, idx,
                                                  B, (B + nb - 1) / nb, gpart, lpart);
    sg_launch(mlp_reduce_kernel, (SG_MLP_NP + 255) / 256, 256, 0, st, gpart, lpart, nb, B, grad, loss);
    return cudaGetLastError();
}

cudaError_t sg_mlp_train_launch(float* wm, void* wbf, float* m1, float* m2, const float* X,
                                const float* Y, const int* idx, int B, float* gpart, float* lpart,
                                float* loss, float lr, int step, cudaStream_t st) {
    const int nb = train_blocks(B);
    __nv_bfloat16* wb = static_cast<__nv_bfloat16*>(wbf);
    sg_launch(mlp_grad_kernel, nb, kTrainThreads, 0, st, (const __nv_bfloat16*)wb, X, Y, idx, B,
              (B + nb - 1) / nb, gpart, lpart);
    sg_launch(mlp_adam_kernel, SG_MLP_NP / 128 + 1, 128, 0, st, wm, wb, m1, m2,
              (const float*)gpart, (const float*)lpart, nb, B, loss, lr, 0.9f, 0.999f, 1e-8f, step);
    return cudaGetLastError();
}

cudaError_t sg_mlp_to_bf16_launch(const float* wm, void* wbf, cudaStream_t st) {
    sg_launch(mlp_to_bf16_kernel, (SG_MLP_NP + 255) / 256, 256, 0, st, wm, static_cast<__nv_bfloat16*>(wbf));
    return cudaGetLastError();
}

cudaError_t sg_mlp_forward_launch(const void* wbf, const float* X, int n, float* out,
                                  cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    sg_launch(mlp_forward_kernel, (n + 3) / 4, 128, 0, st, static_cast<const __nv_bfloat16*>(wbf), X, n, out);
    return cudaGetLastError();
}
