// Chained launches: the kernels of a step (and of a plain transform) launched so that each
// may be set up, and read its constant tables, while the one before it still runs
// (programmatic stream serialization).  A kernel launched through chain_launch calls
//   chain_start()  before its last stores: the next kernel of the stream may be scheduled once
//                  every CTA of this one has come so far or ended;
//   chain_start(lead)  at its beginning, where lead (its last argument, from chain_launch) is the
//                  number of its CTAs that are resident at once: the CTAs after those do the same;
//   chain_wait()   before its first access to anything another kernel writes, and before its
//                  first write: returns when the kernel before it has completed and its writes
//                  are visible.  Every thread calls it, in every kernel of the chain, so the
//                  order of the stream holds across the whole chain.
// A chained kernel is resident while the one before it still stores, so none of its pointers but
// those of the constant tables is __restrict__: the qualifier on a const pointer promises data
// that nothing writes during the kernel, and allows its loads to move above the wait or to go
// through the non-coherent path.
// The launch gap of the small passes is what this removes: 1.6 us of a 5 us pass.  A next kernel that
// starts while most of this one's work is still to come has its CTAs packed onto the few
// multiprocessors with room left, and runs them there: with chain_start() at the beginning of every
// CTA 192x128x32 FP32 with noise took 42.5 us per step, unchained 37.7, so 28.2; 64x64x64 15.2,
// 20.1, 11.8; R2C of 1024^2 22.5, 17.4, 12.9.  In a grid of several waves the CTAs after the first
// wave start it early, so that the next kernel fills the last wave's gaps (192x160x192 68 us per
// step; with the late start alone 88).  Calls whose stream is being captured, and ensembles
// (captured, several branches), launch plainly.
#pragma once
#include <cuda_runtime.h>
#include <climits>
#include <cstdint>
#include "pfc_ctx.h"

namespace pfc {

__device__ __forceinline__ void chain_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_start(int lead) {
    if (blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z) >= (unsigned)lead) chain_start();
}
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_with(const cudaLaunchConfig_t& cfg, void (*kernel)(P...), A&&... args) {
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// args: the kernel's but the last, lead
template <class... P, class... A>
cudaError_t chain_launch(const pfc_ctx* c, void (*kernel)(P...), dim3 grid, int threads, size_t smem, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = c->chain ? 1 : 0;
    int lead = INT_MAX;
    if (c->chain && (int64_t)grid.x * grid.y * grid.z > 2 * (int64_t)c->num_sms) {
        int n = 0;  // (0.1 us of host time)
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem);
        if (e) return e;
        lead = n * c->num_sms;
    }
    return launch_with(cfg, kernel, args..., lead);
}

// Chains the launches of one API call on the context's stream.
struct ChainScope {
    pfc_ctx* c;
    explicit ChainScope(pfc_ctx* ctx) : c(ctx) {
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(c->stream, &st) != cudaSuccess) {
            cudaGetLastError();
            st = cudaStreamCaptureStatusActive;
        }
        c->chain = st == cudaStreamCaptureStatusNone && c->batch == 1;
    }
    ~ChainScope() { c->chain = false; }
    ChainScope(const ChainScope&) = delete;
    ChainScope& operator=(const ChainScope&) = delete;
};

}  // namespace pfc
