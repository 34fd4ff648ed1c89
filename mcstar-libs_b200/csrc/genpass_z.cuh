// The general z pass of the stepper (genpass.cuh): kernel and launcher, instantiated per
// precision by kern_genz32.cu and kern_genz64.cu.
#pragma once
#include "chain.cuh"
#include "genpass.cuh"

namespace pfc {
namespace {

// ---------------------------------------------------------------------------------
// The stepper's z pass: along the columns of the last axis (z; y in a 2D field) the
// forward transform of the nonlinear term, the semi-implicit update (eom.hpp:60-72 with
// stabilisation C) with its noise, and the inverse transform for the next step.
// ---------------------------------------------------------------------------------
// 2 pi / L of an axis, in FP32 with its rounding: that is the same for all modes of the axis, and grows
// into the state step by step
template <typename T> struct Wave {
    T hi, lo;
    explicit Wave(double k) : hi((T)k), lo((T)(k - (double)(T)k)) {}
    // the wavenumber of index i of n (common.hpp:27-28)
    __device__ __forceinline__ T at(int i, int n) const {
        const T m = T(i < n / 2 + 1 ? i : i - n);
        return sizeof(T) == 4 ? fma(m, lo, m * hi) : m * hi;
    }
};

template <typename T>
struct ZArgsT {
    T dt, eps, C, namp_eff;
    Wave<T> ckx, cky, ckz;
    uint64_t seed, counter;
    const unsigned long long* dev_counter;  // read instead of counter when set
    int use_noise, final_step, prop;
    unsigned* maxc;                         // relaxations: max |psi^' - psi^| (float bits), or null
    const MemberArgs* margs;                // batched fields: per-field eps, noise amplitude, seed
    int ky0, nyg;                           // a ky-slab: the field's first row here and its row count
};

// The field of a batch this CTA steps (grid z): its noise counter and parameters.
template <typename T>
__device__ __forceinline__ void zmember(ZArgsT<T>& a) {
    if (a.dev_counter) a.counter = a.dev_counter[blockIdx.z];
    if (a.margs) {
        const MemberArgs m = a.margs[blockIdx.z];
        a.eps = (T)m.eps;
        a.namp_eff = (T)m.namp_eff;
        a.seed = m.seed;
    }
}

// What a kx column contributes to the modes of a CTA: its wavenumber and kx^2 + ky^2.
template <typename T> struct ZColumn {
    int kx;
    T kk0, kxy;
    __device__ __forceinline__ ZColumn(int kx_, int nx, T k1, const ZArgsT<T>& a)
        : kx(kx_), kk0(a.ckx.at(kx_, nx)), kxy(kk0 * kk0 + k1 * k1) {}
};

// The update of mode (kx, kyg, kz) from psi^ and N^ by propagator PROP with its noise; kk2 =
// the kz wavenumber, deps = 1 + C - eps.  At k = 0 the conserved propagators return psi^
// itself (dopx = 0).  The relaxations fold |psi^' - psi^| into mc.
template <typename T, int PROP>
__device__ __forceinline__ cx<T> zmode_of(cx<T> psi, cx<T> nl, const ZColumn<T>& col, int kyg, int kz, T kk2, int nx,
                                          int nz, T deps, const ZArgsT<T>& a, float& mc) {
    const int kx = col.kx;
    const T dopx = -(col.kxy + kk2 * kk2);
    cx<T> v;
    if constexpr (PROP == kPropConserved) {
        const T dopy = dopx * dopx;
        const T denom = T(1) - a.dt * (deps * dopx + T(2) * dopy + dopx * dopy);
        const T f = a.dt * dopx;
        cx<T> num = mkc<T>(psi.x + f * nl.x, psi.y + f * nl.y);
        if (a.use_noise) {
            const cx<T> xi = kspace_noise<T>(kx, kyg, kz, nx, a.nyg, nz, a.seed, a.counter);
            const T g = a.dt * a.namp_eff * sqrt(-dopx);
            num.x += g * xi.x;
            num.y += g * xi.y;
        }
        v = mkc<T>(num.x / denom, num.y / denom);
    } else {
        T ca, cb, cg;
        prop_coef<PROP, T>(dopx, a.dt, deps, ca, cb, cg);
        v = mkc<T>(ca * psi.x + cb * nl.x, ca * psi.y + cb * nl.y);
        if (prop_conserved<PROP>() && a.use_noise) {
            // (the anisotropic noise is for 2D fields, whose y axis is the columns' here)
            const cx<T> xi = PROP == kPropConservedHpfc
                                 ? hpfc_noise<T>(kx, kz, nx, nz, col.kk0, kk2, sqrt(-dopx), a.seed, a.counter)
                                 : kspace_noise<T>(kx, kyg, kz, nx, a.nyg, nz, a.seed, a.counter);
            v.x += a.namp_eff * cg * xi.x;
            v.y += a.namp_eff * cg * xi.y;
        }
        if (!prop_conserved<PROP>()) {
            const T dx = v.x - psi.x, dy = v.y - psi.y;
            mc = fmaxf(mc, (float)sqrt(dx * dx + dy * dy));
        }
    }
    return v;
}

// (the propagator is a run-time switch, the same for every mode: one kernel for all of them but the
// conserved step, PROP >= 0, whose instructions are then together: 240 x 200 x 180 FP32 with noise 166.9
// -> 161.3 us per step, 2400 x 2000 104.1 -> 100.1, 192^3 FP64 with noise 231.8 -> 228.8: more than the
// update's divisions cost against the reciprocal they replaced)
template <typename T, int PROP, class... A>
__device__ __forceinline__ cx<T> zmode(int prop, A&&... args) {
    if constexpr (PROP >= 0) return zmode_of<T, PROP>(args...);
    switch (prop) {
        case kPropConservedExp: return zmode_of<T, kPropConservedExp>(args...);
        case kPropRelax: return zmode_of<T, kPropRelax>(args...);
        case kPropRelaxExp: return zmode_of<T, kPropRelaxExp>(args...);
        case kPropConservedPoly: return zmode_of<T, kPropConservedPoly>(args...);
        case kPropConservedHpfc: return zmode_of<T, kPropConservedHpfc>(args...);
        default: return zmode_of<T, kPropConserved>(args...);
    }
}

// A tile of kx columns (2^lg elements of n modes, at one ky) per CTA, over the reference layout.
// CARRY true: psi^ itself is carried in A; N^ = FFT(B), the update writes psi^' over psi^, and
// A' = IFFT(psi^')/n goes to anext (which may be B: a CTA reads its columns before it writes
// them; not written on the final step; in a 2D field without the 1/n, which its x pass applies).  CARRY false (ky-slabs, and schedules that ask for
// it): A = IFFT(psi^)/n is carried; psi^ = FFT(A), N^ = FFT(B), the update, A' over A (psi^'
// on the final step), the k = 0 mode from its FP64 slot.  The N^ lines (and with CARRY false
// the psi^ lines beside them) stay in shared memory, digit-reversed, between the transforms.
template <typename T, bool CARRY, bool ODD, int PROP>
__global__ void __launch_bounds__(kColThreads<T>, 1)
    k_zprop(cx<T>* A, const cx<T>* B, int nx, int ny, const __grid_constant__ GPlan p, const el<T>* __restrict__ tw,
            const int* __restrict__ tab, int lg, int w, ZArgsT<T> a, const double2* k0, int* flag, int64_t ms,
            cx<T>* anext, double rn, int lead) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    el<T>* buf = reinterpret_cast<el<T>*>(smem_raw);
    chain_start(lead);
    chain_wait();
    zmember(a);
    const int nxh = nx / 2 + 1, n = p.n;
    const ColTile<T> tile{lg, w, nxh};
    const int i0 = tile.i0, ky = blockIdx.y;
    const int64_t es = (int64_t)ny * nxh;
    const int64_t base = blockIdx.z * ms + (int64_t)ky * nxh + i0;  // grid z: fields of a batch
    A += base;
    B += base;
    // the lines in shared memory: the tile's N^ lines, after its psi^ lines when they are
    // transformed too
    const ColLines<ODD> lay{CARRY ? lg : lg + 1};
    const int tmask = (1 << lg) - 1, nl0 = CARRY ? 0 : 1 << lg;
    stage_first<T, -1>(buf, p, lay, tw, [&](int i, int j, int m) {
        const int c = i & tmask;
        return tile.get((!CARRY && i <= tmask ? A : B) + c + j * es, c, m * es);
    });
    __syncthreads();
    stages_mid<T, -1>(buf, p, lay, tw);
    stage_inplace<T, -1, false, false>(buf, p, p.nst - 1, lay, tw);
    __syncthreads();
    // a ky-slab of a larger field: wavenumbers, the k = 0 mode and the noise keys of the field
    const int kyg = ky + a.ky0;
    const T k1 = a.cky.at(kyg, a.nyg);
    const T deps = T(1) + a.C - a.eps;
    float mc = 0.f;
    T bad = T(0);
    const int* rev = tab + p.rev;
    const bool conserved = a.prop != kPropRelax && a.prop != kPropRelaxExp;
    // a thread keeps to one element of the tile's columns (the threads of a CTA are a multiple of
    // the tile), so that what depends on kx alone is computed once
    const int i = threadIdx.x & tmask;
    const ZColumn<T> ca(i0 + i, nx, k1, a), cb(i0 + i + tile.second, nx, k1, a);
    const bool both = Elem<T>::lines > 1 && tile.ok(i, 1);
    const cx<T> zero = mkc<T>(T(0), T(0));
    for (int q = tile.ok(i, 0) ? threadIdx.x >> lg : n; q < n; q += blockDim.x >> lg) {
        const int b = fdiv(q, p.by_rl);
        const int kz = rev[b] + (q - b * p.rl) * p.kstep;
        const int at = q + (p.pad ? b : 0);
        cx<T>* g = A + i + kz * es;
        el<T>* slot = buf + lay.at(nl0 + i, at);
        const cx<T> psi_a = CARRY ? *g : zero, psi_b = CARRY && both ? g[tile.second] : zero;
        const el<T> psi = CARRY ? Elem<T>::pack(psi_a, psi_b) : buf[lay.at(i, at)];
        const el<T> nl = *slot;
        const T kk2 = a.ckz.at(kz, n);
        auto update = [&](cx<T> ps, cx<T> f, const ZColumn<T>& col) {
            if (!CARRY && conserved && col.kx == 0 && kyg == 0 && kz == 0)
                ps = mkc<T>((T)k0[blockIdx.z].x, (T)k0[blockIdx.z].y);
            const cx<T> v = zmode<T, PROP>(a.prop, ps, f, col, kyg, kz, kk2, nx, n, deps, a, mc);
            bad = bad + (v.x - v.x) + (v.y - v.y);  // zero while everything is finite
            return v;
        };
        const cx<T> va = update(Elem<T>::template line<0>(psi), Elem<T>::template line<0>(nl), ca);
        cx<T> vb = zero;
        if (both) vb = update(Elem<T>::template line<1>(psi), Elem<T>::template line<1>(nl), cb);
        if (CARRY || a.final_step) {
            *g = va;
            if (both) g[tile.second] = vb;
        }
        *slot = Elem<T>::pack(va, vb);
    }
    if (!conserved && a.maxc) fold_max_change(mc, a.maxc);
    if (__any_sync(0xffffffffu, !(bad == T(0))) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
    if (a.final_step) return;
    __syncthreads();
    // back to the columns of the tile (CARRY false: the psi^ lines ride along unused)
    stage_inplace<T, 1, true, false>(buf, p, p.nst - 1, lay, tw);
    __syncthreads();
    stages_back<T, 1>(buf, p, lay, tw);
    chain_start();
    cx<T>* dst = CARRY ? anext + base : A;
    // (rn: the entry transform's scale, so that a resumed run repeats the bits)
    const typename Elem<T>::real scale = Elem<T>::bc(rn);
    stage_out<T, 1>(buf, p, lay, tw, [&](int i, int j, int m) {
        const int c = i & tmask;
        const bool ok0 = i >= nl0 && tile.ok(c, 0), ok1 = i >= nl0 && tile.ok(c, 1);
        cx<T>* g = dst + c + j * es;
        cx<T>* h = g + tile.second;
        const int64_t step = m * es;
        return [=](int r, el<T> v) {
            v = Elem<T>::make(vmul(Elem<T>::re(v), scale), vmul(Elem<T>::im(v), scale));
            if (ok0) g[r * step] = Elem<T>::template line<0>(v);
            if (Elem<T>::lines > 1 && ok1) h[r * step] = Elem<T>::template line<1>(v);
        };
    });
}

// The z pass of a slab of a 2D field (nz = 1: the y transforms are the slab's xy part): no transform,
// so the update of every mode in place, one thread per mode.  (The column pass with lines of one
// point has a CTA per row and half of its threads idle: 2048 x 1536 FP64 209 us, so 13.)
template <typename T>
__global__ void __launch_bounds__(256) k_zflat(cx<T>* A, const cx<T>* B, int nx, int ny, FastDiv by_nxh, ZArgsT<T> a,
                                               const double2* k0, int* flag) {
    const int nxh = nx / 2 + 1, m = blockIdx.x * blockDim.x + threadIdx.x;
    float mc = 0.f;
    bool bad = false;
    if (m < nxh * ny) {
        const int ky = fdiv(m, by_nxh), kx = m - ky * nxh, kyg = ky + a.ky0;
        const ZColumn<T> col(kx, nx, a.cky.at(kyg, a.nyg), a);
        cx<T> psi = A[m];
        if (kx == 0 && kyg == 0 && a.prop != kPropRelax && a.prop != kPropRelaxExp) psi = mkc<T>((T)k0->x, (T)k0->y);
        const cx<T> v = zmode<T, -1>(a.prop, psi, B[m], col, kyg, 0, a.ckz.at(0, 1), nx, 1, T(1) + a.C - a.eps, a, mc);
        bad = !isfinite(v.x) || !isfinite(v.y);
        A[m] = v;
    }
    if ((a.prop == kPropRelax || a.prop == kPropRelaxExp) && a.maxc) fold_max_change(mc, a.maxc);
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1);
}

}  // namespace

// f(kernel) for the z pass of a plan and a propagator (`all`: for every one of them)
template <typename T, class F> cudaError_t by_zprop(bool carry, bool odd, int prop, bool all, F&& f) {
    cudaError_t e = cudaSuccess;
    auto take = [&](bool c, bool o, bool p, auto kernel) {
        if (!e && (all || (carry == c && odd == o && (prop == kPropConserved) == p))) e = f(kernel);
    };
    take(false, false, true, k_zprop<T, false, false, kPropConserved>);
    take(false, false, false, k_zprop<T, false, false, -1>);
    take(false, true, true, k_zprop<T, false, true, kPropConserved>);
    take(false, true, false, k_zprop<T, false, true, -1>);
    take(true, false, true, k_zprop<T, true, false, kPropConserved>);
    take(true, false, false, k_zprop<T, true, false, -1>);
    take(true, true, true, k_zprop<T, true, true, kPropConserved>);
    take(true, true, false, k_zprop<T, true, true, -1>);
    return e;
}

template <typename T> cudaError_t gen_zattrs() {
    return by_zprop<T>(false, false, 0, true, [](auto k) {
        return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynSmem);
    });
}

// flat: a 2D field, its y columns in the place of z (mode (kx, ky) of the field is mode (kx, 0,
// kz = ky) of the pass: the same linear index, so the same noise)
template <typename T>
cudaError_t gen_zprop(const pfc_ctx* c, void* A, const void* B, const ZPropArgs& a, void* anext, bool carry,
                      bool flat) {
    if (a.prop == kPropConservedHpfc && !flat) return cudaErrorNotSupported;
    const AxisPlan& ap = flat ? c->py2 : carry ? c->pzprop : c->pz2;
    const int ny = flat ? 1 : c->ny, tile = ap.w << ap.lg;
    const double tp = 6.283185307179586232;
    // (kz = 0 of a 2D field: zero, or not a number for an lz that gives none)
    const double kz0 = flat ? (double)(T(0) * (T)tp / (T)a.lz) : 0.0;
    dim3 grid((c->nxh + tile - 1) / tile, ny, c->batch);
    ZArgsT<T> t{(T)a.dt, (T)a.eps, (T)a.C, (T)a.namp_eff, Wave<T>(tp / a.lx + kz0), Wave<T>(flat ? 0.0 : tp / a.ly),
                Wave<T>(tp / (flat ? a.ly : a.lz)), a.seed, a.counter, a.dev_counter, a.use_noise, a.final_step, a.prop,
                a.maxc, a.margs, a.ky0, a.ny_global > 0 ? a.ny_global : ny};
    if (!flat && !carry && c->nz == 1 && c->batch == 1) {
        const int modes = c->nxh * c->ny;
        k_zflat<T><<<(modes + 255) / 256, 256, 0, c->stream>>>((cx<T>*)A, (const cx<T>*)B, c->nx, c->ny,
                                                               make_fastdiv(c->nxh), t, c->k0, c->flag);
        return cudaGetLastError();
    }
    return by_zprop<T>(carry, ap.plan.odd, a.prop, false, [&](auto k) {
        return chain_launch(c, k, grid, ap.threads, carry ? ap.smem : 2 * ap.smem, (cx<T>*)A, (const cx<T>*)B, c->nx,
                            ny, ap.plan, (const el<T>*)c->gtw, c->fft_tab, ap.lg, ap.w, t, c->k0, c->flag, c->mstride,
                            (cx<T>*)anext, flat ? 1.0 : 1.0 / (double)ap.plan.n);
    });
}

}  // namespace pfc
