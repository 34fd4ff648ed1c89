// Chained launches: the kernels of a step (and of a plain transform) launched so that each
// may be set up, and read its constant tables, while the one before it still runs
// (programmatic stream serialization).  A kernel launched through chain_launch calls
//   chain_start()  at its beginning: the next kernel of the stream may be scheduled once every
//                  CTA of this one has started;
//   chain_wait()   before its first access to anything another kernel writes, and before its
//                  first write: returns when the kernel before it has completed and its writes
//                  are visible.  Every thread calls it, in every kernel of the chain, so the
//                  order of the stream holds across the whole chain.
// A chained kernel is resident while the one before it still stores, so none of its pointers but
// those of the constant tables is __restrict__: the qualifier on a const pointer promises data
// that nothing writes during the kernel, and allows its loads to move above the wait or to go
// through the non-coherent path.
// The launch gap of the small passes is what this removes: 1.6 us of a 5 us pass.  Calls whose
// stream is being captured, and ensembles (captured, several branches), launch plainly.
#pragma once
#include <cuda_runtime.h>
#include <utility>
#include "pfc_ctx.h"

namespace pfc {

__device__ __forceinline__ void chain_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

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
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
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
