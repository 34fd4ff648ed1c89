// The general z pass in single precision.
#include "genpass_z.cuh"

namespace pfc {
template cudaError_t gen_zattrs<float>();
template cudaError_t gen_zprop<float>(const pfc_ctx*, void*, const void*, const ZPropArgs&, void*, bool, bool);
}  // namespace pfc
