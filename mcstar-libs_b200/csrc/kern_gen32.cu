// The general column and row passes in single precision.
#include "genpass_xy.cuh"

namespace pfc {
template cudaError_t gen_attrs<float>();
template cudaError_t gen_cols<float>(const pfc_ctx*, int, int, const void*, void*, double);
template cudaError_t gen_rows<float>(const pfc_ctx*, int, const void*, void*, double, double, double);
}  // namespace pfc
