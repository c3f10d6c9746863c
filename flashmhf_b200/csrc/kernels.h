// Internal launch interface between the C-ABI layer (api.cu) and the kernel translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/flashmhf.h"

namespace fmhf {

// Per-device control words and facts, resolved once per device (with that device current).
//   status    : 0, or the code of the first bounded wait that ran out since the host last read it
//   abort_seq : sequence number of the launch whose wait ran out; the other CTAs of THAT launch see it at
//               their start and return at once, later launches (other numbers) run normally
struct DeviceCtl {
    int *status = nullptr;
    unsigned *abort_seq = nullptr;
    int num_sms = 0;
    int device = -1;
};
const DeviceCtl *device_ctl();  // nullptr if the device query failed
unsigned next_launch_seq();     // process-wide, never 0
// SM count of the current device (the B200's 148 when no device can be queried, e.g. sizing a workspace on a CPU-only host).
inline int num_sms() {
    const DeviceCtl *c = device_ctl();
    return c ? c->num_sms : 148;
}

// What every tensor-core kernel needs for its bounded waits.
struct WaitArgs {
    int *status;
    unsigned *abort_seq;
    unsigned seq;
    long long limit_cycles;
};
constexpr long long kDefaultWaitLimitCycles = 3LL << 30;  // ~1.5 s at 1.4-1.9 GHz; a healthy kernel waits microseconds
inline WaitArgs wait_args(const DeviceCtl *c) {
    return WaitArgs{c->status, c->abort_seq, next_launch_seq(), kDefaultWaitLimitCycles};
}

// ---- fp32 check kernels (CUDA cores) -------------------------------------------------------
cudaError_t simt_forward(const flashmhf_fwd_params &p, cudaStream_t st, int *n_launch);
cudaError_t simt_backward(const flashmhf_bwd_params &p, cudaStream_t st, int *n_launch);

// ---- bf16 tensor-core kernels (tcgen05 / TMEM / TMA) ---------------------------------------
// Each returns a flashmhf_status (tensor-map encoding can fail with BAD_STRIDE / CUDA).
// `chained`: launched so that it may overlap the end of the kernel before it on the stream (see flashmhf_forward_chained)
int tc_forward(const flashmhf_fwd_params &p, cudaStream_t st, int *n_launch, bool chained);
size_t tc_forward_workspace_bytes(const flashmhf_dims &d);
int tc_backward(const flashmhf_bwd_params &p, cudaStream_t st, int *n_launch);
size_t tc_backward_workspace_bytes(const flashmhf_dims &d);          // all of it
size_t tc_backward_weights_workspace_bytes(const flashmhf_dims &d);  // what the dK/dU/dV part cannot do without
size_t tc_backward_inputs_workspace_bytes(const flashmhf_dims &d);   // what a call for dQ and dR alone can use (0: nothing)
// Sum of `nsplit` fp32 partial planes [B,H,S,Dh], in index order, as bf16 to `out` (strides multiples of 4 elements).
// Launched early; adds when the kernel before it is done.  `chained`: between two chained forward kernels.
cudaError_t launch_o_reduce(const float *part, const flashmhf_tensor &out, const flashmhf_dims &d, int nsplit, bool chained, int num_sms,
                            cudaStream_t st);
void tc_backward_plan(const flashmhf_dims &d, uint32_t parts, flashmhf_backward_plan_info *out);
int tc_backward_static_scratch(const flashmhf_bwd_params &p, cudaStream_t st, int *n_launch);

// ---- fused layer prologue (per-head RMSNorm + router weights), HBM-bound CUDA-core kernels --
// `bf16_params`: norm weight and router (and their gradients) are bf16 instead of fp32
int prologue_forward(const flashmhf_prologue_params &p, bool bf16_params, cudaStream_t st, int *n_launch);
size_t prologue_backward_workspace_bytes(const flashmhf_prologue_params &p);
int prologue_backward(const flashmhf_prologue_bwd_params &p, bool bf16_params, cudaStream_t st, int *n_launch);

// ---- helpers for the measurement LM: rotary embedding and hidden-size RMSNorm (lm_aux.cu) ----
int lm_rope(const void *x, void *y, const float *cos_t, const float *sin_t, long long tokens, int S, int heads, int hd,
            long long x_tok, long long y_tok, int transpose, cudaStream_t st, int *n_launch);
int lm_rope_pair(const void *q, void *yq, int heads_q, const void *k, void *yk, int heads_k, const float *cos_t, const float *sin_t,
                 long long tokens, int S, int hd, int transpose, cudaStream_t st, int *n_launch);
int lm_rmsnorm_forward(const void *x, const void *d, void *sum, const void *w, bool bf16_w, void *y, long long rows, int n, float eps,
                       cudaStream_t st, int *n_launch);
size_t lm_rmsnorm_backward_workspace_bytes(long long rows, int n);
int lm_rmsnorm_backward(const void *x, const void *w, bool bf16_w, const void *g, const void *gh, void *dx, void *dw, void *workspace,
                        size_t workspace_bytes, long long rows, int n, float eps, cudaStream_t st, int *n_launch);

// Launch.  `early`: with programmatic stream serialization, so that the kernel may start before the one ahead of it on the
// stream has ended (as soon as that one's CTAs have all asked for it, or exited).
// `cluster`: CTAs (along x) of a thread-block cluster.
template <typename... KArgs, typename... Args>
cudaError_t launch_kernel(bool early, int cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (early) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)cluster;
        at[n].val.clusterDim.y = 1;
        at[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t launch_kernel(bool early, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    return launch_kernel(early, 1, kernel, grid, block, smem, st, std::forward<Args>(args)...);
}

void set_cuda_error(cudaError_t e, const char *where);
int selftest_bounded_wait(long long limit_cycles, cudaStream_t st, int *n_launch);

// Kernel-boundary marks for the profiling aid (flashmhf_profile_begin/end): records an event on
// `st` tagged `tag` when profiling is on, does nothing otherwise.
enum { kMarkStart = 0, kMarkFwd = 1, kMarkBwdDq = 2, kMarkBwdDw = 3, kMarkBwdReduce = 4, kMarkFwdReduce = 5,
       kMarkPrologueFwd = 6, kMarkPrologueBwd = 7, kMarkPrologueReduce = 8 };
void prof_mark(cudaStream_t st, int tag);

}  // namespace fmhf
