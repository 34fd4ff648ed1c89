// The general column and row passes in double precision.
#include "genpass_xy.cuh"

namespace pfc {
template cudaError_t gen_attrs<double>();
template cudaError_t gen_cols<double>(const pfc_ctx*, int, int, const void*, void*, double);
template cudaError_t gen_rows<double>(const pfc_ctx*, int, const void*, void*, double, double, double);
}  // namespace pfc
