// The general-length passes over the reference layout (x fastest; half spectrum of nx/2+1
// complex per row): whole lines of a tile in shared memory, transformed by the engine of
// genfft.cuh.  They serve the reference-shaped primitives (R2C, C2R) and the stepper wherever
// a length has no register kernel, in FP32 and FP64.  kern_gen*.cu instantiate them.
#pragma once
#include "genfft.cuh"
#include "pfc_ctx.h"

namespace pfc {

template <typename T> cudaError_t gen_attrs();
template <typename T> cudaError_t gen_cols(const pfc_ctx* c, int axis, int dir, const void* in, void* out, double scale);
enum { kR2C = 0, kC2R = 1, kNonlin = 2 };
template <typename T>
cudaError_t gen_rows(const pfc_ctx* c, int mode, const void* in, void* out, double mul, double C, double mu);
template <typename T> cudaError_t gen_zattrs();
template <typename T>
cudaError_t gen_zprop(const pfc_ctx* c, void* A, const void* B, const ZPropArgs& a, void* anext, bool carry, bool flat);

// Register budget of the general passes: FP32 64 (four CTAs of 256 threads per SM), FP64 80
// (six of 128; a radix-10 butterfly holds 40 of them, and its FP64 arithmetic needs more
// temporaries).  They are latency-bound: at 128 registers and radices up to 16 the passes of
// 240 x 200 x 180 FP32 took 0.025 / 0.049 / 0.088 ms (y, x, z) against 0.021 / 0.044 / 0.060.
// The column passes may take the whole register file with one CTA: 1024 threads (FP64 768) of the
// same registers, for fields with few tiles.  One body holds the radices 1 to 6 and 8 to 10, so the FP32
// kernels spill at 64 registers: k_cols 48 and 152 bytes (inverse, forward), k_rows 100 to 112,
// k_zprop 120 to 176; k_xpass has 80 registers and does not spill.  The kernels of plans with radix 7 or
// 11 to 31 are instantiated apart, with the points of a direct DFT in local memory.
template <typename T> constexpr int kGenCtas = sizeof(T) == 8 ? 3 : 4;
constexpr int kGenThreads = 256;
template <typename T> constexpr int kColThreads = sizeof(T) == 8 ? 768 : 1024;

// largest first radix of the stepper's paired x pass (two butterflies in registers)
constexpr int kPairRadix = 5;

// The columns of a CTA: 2^lg elements of one column (FP64, and FP32 with w = 1: the second line
// then holds zeros) or of two columns 2^lg apart (FP32, w = 2; consecutive threads then move
// consecutive columns of either half), of ni.
template <typename T> struct ColTile {
    int i0, n, second;
    __device__ __forceinline__ ColTile(int lg, int w, int ni) {
        i0 = blockIdx.x * (w << lg);
        n = min(ni - i0, w << lg);
        second = 1 << lg;
    }
    __device__ __forceinline__ bool ok(int i, int half) const { return i + half * second < n; }
    // the elements of position i at g (column i0 + i), step apart
    __device__ __forceinline__ auto get(const cx<T>* g, int i, int64_t step) const {
        const bool ok0 = ok(i, 0), ok1 = ok(i, 1);
        const cx<T>* h = g + second;
        return [=](int r) {
            const cx<T> z = mkc<T>(T(0), T(0));
            const cx<T> a = ok0 ? g[r * step] : z;
            return Elem<T>::pack(a, Elem<T>::lines > 1 && ok1 ? h[r * step] : z);
        };
    }
};

}  // namespace pfc
