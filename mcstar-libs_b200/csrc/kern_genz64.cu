// The general z pass in double precision.
#include "genpass_z.cuh"

namespace pfc {
template cudaError_t gen_zattrs<double>();
template cudaError_t gen_zprop<double>(const pfc_ctx*, void*, const void*, const ZPropArgs&, void*, bool, bool);
}  // namespace pfc
