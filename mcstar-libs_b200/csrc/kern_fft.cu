// Launchers of the general-length passes (genpass.cuh) by the context's precision.
#include "genpass.cuh"

namespace pfc {

cudaError_t set_fft_attributes(const pfc_ctx* c) {
    const bool d = c->dtype == PFC_F64;
    const cudaError_t e = d ? gen_attrs<double>() : gen_attrs<float>();
    return e ? e : d ? gen_zattrs<double>() : gen_zattrs<float>();
}

cudaError_t launch_cols(const pfc_ctx* c, int axis, int dir, const void* in, void* out, double scale) {
    return c->dtype == PFC_F64 ? gen_cols<double>(c, axis, dir, in, out, scale)
                               : gen_cols<float>(c, axis, dir, in, out, scale);
}

namespace {
cudaError_t rows(const pfc_ctx* c, int mode, const void* in, void* out, double mul, double C, double mu) {
    return c->dtype == PFC_F64 ? gen_rows<double>(c, mode, in, out, mul, C, mu)
                               : gen_rows<float>(c, mode, in, out, mul, C, mu);
}
cudaError_t zprop(const pfc_ctx* c, void* A, const void* B, const ZPropArgs& a, void* anext, bool carry, bool flat) {
    return c->dtype == PFC_F64 ? gen_zprop<double>(c, A, B, a, anext, carry, flat)
                               : gen_zprop<float>(c, A, B, a, anext, carry, flat);
}
}  // namespace

cudaError_t launch_rows_r2c(const pfc_ctx* c, const void* in, void* out) { return rows(c, kR2C, in, out, 1.0, 0.0, 0.0); }
cudaError_t launch_rows_c2r(const pfc_ctx* c, const void* in, void* out) { return rows(c, kC2R, in, out, 1.0, 0.0, 0.0); }
cudaError_t launch_rows_nonlin(const pfc_ctx* c, void* buf, double mul, double C, double mu) {
    return rows(c, kNonlin, buf, buf, mul, C, mu);
}

cudaError_t launch_zprop(const pfc_ctx* c, void* A, const void* B, const ZPropArgs& a) {
    return zprop(c, A, B, a, nullptr, false, false);
}
cudaError_t launch_zprop_carry(const pfc_ctx* c, void* kpsi, const void* B, void* anext, const ZPropArgs& a) {
    return zprop(c, kpsi, B, a, anext, true, c->nz == 1);
}

}  // namespace pfc
