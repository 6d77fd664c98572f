// noalloc.cu -- sg_coulomb_accel_noalloc: the FP64 Coulomb sum for callers that must
// not allocate device memory.
//
// Some callers of this library cannot call cudaMalloc: a host application that does
// all its device allocation up front and forbids it afterwards (real-time or
// memory-budgeted loops), or a plug-in that runs inside another framework's device
// memory pool and is only handed device pointers.  This entry point takes the
// caller's device buffers for inputs and outputs and keeps its own scratch -- the partial
// sums of the pair kernel -- in one file-scope device array of fixed size, so it creates
// no context, allocates nothing and frees nothing, and it copies nothing from host
// memory: each block derives its work item from its block index.
//
// Two launches: the pairs, each unordered pair once (fp64_pairs.cuh), straight from the
// caller's arrays, and the sums of the slots.  FP64-bound: 2,048 ions take 100 us, where
// the ordered pairs over 32 blocks of 128 threads (a fifth of the SMs) with a launch to
// transpose the positions took 705.
//
// Capacity: at most kNaMaxIons ions per call (larger n returns SG_TOO_LARGE before
// any work is queued).  The array is 13 MB and every GPU that loads this library
// holds it until the process exits.  All calls on a device share it and it keeps
// the last call's contents: every scratch entry a call reads is written earlier in
// the same call, so nothing has to start at zero, but calls that overlap on the GPU
// (different streams, or host threads without ordering) race on the array.
//
// Set-up: a __device__ array has one address per CUDA context.  The first call made
// in a context looks that address up (cudaGetSymbolAddress, with the context
// current) and keeps it under the context's unique id, so a caller that switches
// between contexts on one device, or destroys and re-creates one, never gets an
// address from another context.  That first call should come before any stream
// capture.
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "fp64_pairs.cuh"
#include "sg_internal.cuh"

namespace {

constexpr int kNaMaxIons = 8192;
constexpr int kNaMaxContexts = 64;
constexpr int kNaSms = 152;  // GB300

// the partial-sum slots: room for 66 at the largest size, which takes 65 (64 i-blocks, 128
// ions each, on the j side of the last one); smaller sets use more of them
constexpr size_t kNaSlotDoubles = (size_t)66 * 3 * kNaMaxIons;
constexpr size_t kScratchBytes = kNaSlotDoubles * sizeof(double);

static __device__ __align__(256) unsigned char g_na_scratch[kScratchBytes];

// The caller's device buffers; the padding ions past n sit far away with no charge.
struct NaLoad {
    const double *pos, *q;
    int n;
    __device__ __forceinline__ double operator()(int a, int k) const {
        if (k < n) return a < 3 ? pos[3 * (size_t)k + a] : q[k];
        return a < 3 ? 1.0e3 + 1.0e-3 * k : 0.0;
    }
};

// The current context's unique id, through the driver entry points the runtime hands
// out (no link against the driver library).
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

struct NaCtxEntry {
    unsigned long long id;
    void* addr;
};

std::mutex g_na_mu;
CtxGetCurrentFn g_get_current = nullptr;
CtxGetIdFn g_get_id = nullptr;
NaCtxEntry g_na_ctx[kNaMaxContexts];
int g_na_nctx = 0;

bool na_current_context_id(unsigned long long* id) {
    if (!g_get_current || !g_get_id) {
        void* f0 = nullptr;
        void* f1 = nullptr;
        cudaDriverEntryPointQueryResult q0, q1;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f0, 12000, cudaEnableDefault,
                                             &q0) != cudaSuccess ||
            q0 != cudaDriverEntryPointSuccess || !f0)
            return false;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f1, 12000, cudaEnableDefault,
                                             &q1) != cudaSuccess ||
            q1 != cudaDriverEntryPointSuccess || !f1)
            return false;
        g_get_current = reinterpret_cast<CtxGetCurrentFn>(f0);
        g_get_id = reinterpret_cast<CtxGetIdFn>(f1);
    }
    CUcontext ctx = nullptr;
    if (g_get_current(&ctx) != CUDA_SUCCESS || !ctx) return false;
    return g_get_id(ctx, id) == CUDA_SUCCESS;
}

// The scratch array's device address in the current context (set-up on first use in
// that context).  Returns null on failure.
void* na_scratch_address() {
    std::lock_guard<std::mutex> lk(g_na_mu);
    unsigned long long id = 0;
    const bool have_id = na_current_context_id(&id);
    if (have_id)
        for (int k = 0; k < g_na_nctx; k++)
            if (g_na_ctx[k].id == id) return g_na_ctx[k].addr;
    // In host code g_na_scratch names a host-side stand-in: the kernels get this
    // pointer, never the symbol itself.  With no context current, this runtime call
    // makes the current device's primary context current first.
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_na_scratch) != cudaSuccess || !p) return nullptr;
    if (!have_id && !na_current_context_id(&id)) return p;  // valid now, not kept
    if (g_na_nctx < kNaMaxContexts) {
        g_na_ctx[g_na_nctx++] = {id, p};
    } else {
        // more contexts than the table holds: replace the oldest entry
        std::rotate(g_na_ctx, g_na_ctx + 1, g_na_ctx + kNaMaxContexts);
        g_na_ctx[kNaMaxContexts - 1] = {id, p};
    }
    return p;
}

}  // namespace

extern "C" int sg_coulomb_accel_noalloc(int n, const double* pos, const double* q,
                                        const double* kq, double* acc, void* stream) {
    if (n < 0) return SG_BAD_ARG;
    if (n == 0) return SG_OK;
    if (!pos || !q || !kq || !acc) return SG_BAD_ARG;
    if (n > kNaMaxIons) return SG_TOO_LARGE;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return SG_NO_DEVICE;
    unsigned char* scratch = static_cast<unsigned char*>(na_scratch_address());
    if (!scratch) return SG_CUDA_ERR;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int npad = (n + SG_PAD - 1) / SG_PAD * SG_PAD;
    const SymPlan plan = sym_plan(npad, kNaSms, kNaSlotDoubles);
    double* part = reinterpret_cast<double*>(scratch);
    // Each launch's own return value: an error an earlier call left in the runtime's
    // last-error slot neither fails this call nor gets cleared by it.
    cudaLaunchConfig_t cfg = {};
    cfg.stream = st;
    cfg.gridDim = dim3(plan.items);
    cfg.blockDim = dim3(SG_SYM_IB);
    if (cudaLaunchKernelEx(&cfg, sym_set_kernel<false, NaLoad>, NaLoad{pos, q, n}, n, npad, plan,
                           false, 1.0, 0.0, part) != cudaSuccess)
        return SG_CUDA_ERR;
    cfg.gridDim = dim3((n + 15) / 16);
    cfg.blockDim = dim3(256);
    if (cudaLaunchKernelEx(&cfg, sym_sum_kernel<16>, (const double*)part, n, npad, plan, kq, 1.0,
                           acc) != cudaSuccess)
        return SG_CUDA_ERR;
    return SG_OK;
}
