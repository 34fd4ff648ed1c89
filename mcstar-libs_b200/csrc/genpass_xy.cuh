// The general column and row passes (genpass.cuh): kernels and launchers, instantiated per
// precision by kern_gen32.cu and kern_gen64.cu.
#pragma once
#include "chain.cuh"
#include "genpass.cuh"

namespace pfc {
namespace {

// ---------------------------------------------------------------------------------
// complex FFT along a strided axis: element (line o, inner i, position k) at
// base + o*os + i + k*es.  A CTA owns 2^lg elements of w consecutive inner lines each (FP64:
// w = 1, FP32: 1 or 2) of one o.  Forward
// transforms run down from natural order, inverse ones up to it: the inverse is then, bit
// for bit, the one of the stepper's z pass (k_zprop).
// ---------------------------------------------------------------------------------
template <typename T, int DIR, bool ODD>
__global__ void __launch_bounds__(kColThreads<T>, 1)
    k_cols(const cx<T>* in, cx<T>* out, int ni, int64_t es, int64_t os, const __grid_constant__ GPlan p,
           const el<T>* __restrict__ tw, const int* __restrict__ tab, int lg, int w, double scale,
           int64_t ms, int lead) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    el<T>* buf = reinterpret_cast<el<T>*>(smem_raw);
    chain_start(lead);
    chain_wait();
    const ColLines<ODD> lay{lg};
    const ColTile<T> tile{lg, w, ni};
    const int64_t base = (int64_t)blockIdx.y * os + tile.i0 + blockIdx.z * ms;  // grid z: fields of a batch
    in += base;
    out += base;
    const typename Elem<T>::real sc = Elem<T>::bc(scale);
    auto put = [&](cx<T>* g, int i, int64_t step) {
        const bool ok0 = tile.ok(i, 0), ok1 = tile.ok(i, 1);
        cx<T>* h = g + tile.second;
        return [=](int r, el<T> v) {
            v = Elem<T>::make(vmul(Elem<T>::re(v), sc), vmul(Elem<T>::im(v), sc));
            if (ok0) g[r * step] = Elem<T>::template line<0>(v);
            if (Elem<T>::lines > 1 && ok1) h[r * step] = Elem<T>::template line<1>(v);
        };
    };
    if constexpr (DIR < 0) {
        stage_first<T, DIR>(buf, p, lay, tw,
                            [&](int i, int j, int m) { return tile.get(in + i + j * es, i, m * es); });
        __syncthreads();
        stages_mid<T, DIR>(buf, p, lay, tw);
        chain_start();
        stage_last<T, DIR>(buf, p, lay, tw, tab + p.rev,
                           [&](int i, int k0) { return put(out + i + k0 * es, i, p.kstep * es); });
    } else {
        stage_in<T, DIR>(buf, p, lay, tw, tab + p.rev,
                         [&](int i, int k0) { return tile.get(in + i + k0 * es, i, p.kstep * es); });
        __syncthreads();
        stages_back<T, DIR>(buf, p, lay, tw);
        chain_start();
        stage_out<T, DIR>(buf, p, lay, tw,
                          [&](int i, int j, int m) { return put(out + i + j * es, i, m * es); });
    }
}

// ---------------------------------------------------------------------------------
// rows: real <-> half spectrum along x.  Even nx packs x[2m], x[2m+1] into one
// complex and runs an nx/2-point FFT with the split/merge twiddles W_nx^k; odd nx
// runs the full nx-point complex FFT.
// ---------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ el<T> r2c_post(el<T> zk, el<T> zm, el<T> w) {
    // X[k] = 1/2 (Z[k] + conj Z[M-k]) - i/2 W^k (Z[k] - conj Z[M-k])
    using E = Elem<T>;
    const el<T> s = E::make(vadd(E::re(zk), E::re(zm)), vsub(E::im(zk), E::im(zm)));
    const el<T> d = E::make(vsub(E::re(zk), E::re(zm)), vadd(E::im(zk), E::im(zm)));
    return CE<T>::scale(CE<T>::template addi<-1>(s, CE<T>::template cmulw<-1>(d, w)), 0.5);
}
template <typename T>
__device__ __forceinline__ el<T> c2r_pre(el<T> xk, el<T> xm, el<T> w) {
    // Z[k] = (X[k] + conj X[M-k]) + i W^-k (X[k] - conj X[M-k]); IFFT_M(Z) = nx * (x[2m] + i x[2m+1])
    using E = Elem<T>;
    const el<T> e = E::make(vadd(E::re(xk), E::re(xm)), vsub(E::im(xk), E::im(xm)));
    const el<T> d = E::make(vsub(E::re(xk), E::re(xm)), vadd(E::im(xk), E::im(xm)));
    return CE<T>::template addi<1>(e, CE<T>::template cmulw<1>(d, w));
}
// The stepper's cubic term (psi3_split.hpp:8-13 with the stabilisation constant C)
template <typename R>
__device__ __forceinline__ R cubic(R v, R mul, R nC, R nmu) {  // nC = -C, nmu = -mu
    const R t = vmul(v, mul);
    return vfma(vfma(t, t, nC), t, nmu);
}

// kR2C: real rows (in) to half-spectrum rows (out); kC2R: half-spectrum rows to real rows;
// kNonlin: the stepper's x pass, C2R, the cubic nonlinearity, R2C, in place on rows of the
// mixed (kx, y, z) field (in == out).  A CTA owns rpc lines of
// the engine: whole rows (W = 1; FP32: each twice) or pairs of rows (FP32, W = 2).  The transforms leave
// frequencies (or cells) digit-reversed; the R2C merge and the C2R output read them back in
// natural order through the position table, so that global accesses stay contiguous.
template <typename T, int MODE, bool ODD>
__global__ void __launch_bounds__(kGenThreads, kGenCtas<T>)
    k_rows(const void* in, void* out, int nrows, int nx, const __grid_constant__ GPlan p,
           const el<T>* __restrict__ tw, const int* __restrict__ tab, const el<T>* __restrict__ post, int rpc,
           int W, double mul, double C, double mu, int64_t ms, FastDiv by_nxh, int lead) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    el<T>* buf = reinterpret_cast<el<T>*>(smem_raw);
    chain_start(lead);
    chain_wait();
    if (Elem<T>::lines == 1) W = 1;
    const int row0 = blockIdx.x * rpc * W;
    const int nr = min(rpc * W, nrows - row0), nl = W > 1 ? (nr + 1) / 2 : nr;
    const RowLines<ODD> lay{nl, p.np};
    const int L = p.n, nxh = nx / 2 + 1;
    const bool even = (nx & 1) == 0;
    const int* pos = tab + p.pos;
    // the second row of an odd last pair repeats the first (and is not stored)
    auto second = [&](int i, int64_t len) { return W > 1 && 2 * i + 1 < nr ? len : 0; };
    if (MODE == kR2C) {
        const T* rows = static_cast<const T*>(in) + (int64_t)row0 * nx;
        stage_first<T, -1>(buf, p, lay, tw, [&](int i, int j, int m) {
            const T* a = rows + (int64_t)(W * i) * nx;
            const T* b = a + second(i, nx);
            return [=](int r) {
                const int k = j + r * m;
                if (even)
                    return Elem<T>::pack(reinterpret_cast<const cx<T>*>(a)[k], reinterpret_cast<const cx<T>*>(b)[k]);
                return Elem<T>::pack(mkc<T>(a[k], T(0)), mkc<T>(b[k], T(0)));
            };
        });
    } else {
        const cx<T>* rows = static_cast<const cx<T>*>(in) + blockIdx.z * ms + (int64_t)row0 * nxh;  // grid z: batch
        stage_first<T, 1>(buf, p, lay, tw, [&](int i, int j, int m) {
            const cx<T>* a = rows + (int64_t)(W * i) * nxh;
            const cx<T>* b = a + second(i, nxh);
            return [=](int r) {
                const int k = j + r * m;
                if (even)
                    return c2r_pre<T>(Elem<T>::pack(a[k], b[k]), Elem<T>::pack(a[L - k], b[L - k]), post[k]);
                return k < nxh ? Elem<T>::pack(a[k], b[k]) : Elem<T>::pack(cconj(a[nx - k]), cconj(b[nx - k]));
            };
        });
    }
    __syncthreads();
    if (MODE == kR2C) {
        stages_mid<T, -1>(buf, p, lay, tw);
        stage_inplace<T, -1, false, false>(buf, p, p.nst - 1, lay, tw);
        __syncthreads();
    } else {
        stages_mid<T, 1>(buf, p, lay, tw);
    }
    if (MODE == kC2R) {
        stage_inplace<T, 1, false, false>(buf, p, p.nst - 1, lay, tw);
        __syncthreads();
        chain_start();
        T* rows = static_cast<T*>(out) + (int64_t)row0 * nx;
        for (int e = threadIdx.x; e < nl * L; e += blockDim.x) {
            const int i = fdiv(e, p.by_n), m = e - i * L;
            const el<T> v = buf[i * p.np + pos[m]];
            T* a = rows + (int64_t)(W * i) * nx;
            auto put = [&](T* row, cx<T> z) {
                if (even) reinterpret_cast<cx<T>*>(row)[m] = z;
                else row[m] = z.x;
            };
            put(a, Elem<T>::template line<0>(v));
            if (W > 1 && 2 * i + 1 < nr) put(a + nx, Elem<T>::template line<1>(v));
        }
        return;
    }
    if (MODE == kNonlin) {
        // the last inverse stage, the cubic term and the first forward stage on one set of
        // registers: cells rev[b] + r kstep of the row
        const auto bmul = Elem<T>::bc(mul), nC = Elem<T>::bc(-C), nmu = Elem<T>::bc(-mu);
        const GStage& s = p.st[p.nst - 1];
        const int total = lay.count(p.kstep);
        by_radix<ODD>(s.R, [&](auto RC) {
            constexpr int R = decltype(RC)::value;
            if constexpr (R > 0) {
                for (int e = threadIdx.x; e < total; e += blockDim.x) {
                    int i, b;
                    lay.split(e, p.kstep, s.by_nb, i, b);
                    el<T>* a = buf + lay.at(i, b * s.Ms);
                    el<T> v[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) v[r] = a[r];
                    EDft<T, 1, R>::run(v);
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        v[r] = Elem<T>::make(cubic(Elem<T>::re(v[r]), bmul, nC, nmu),
                                             even ? cubic(Elem<T>::im(v[r]), bmul, nC, nmu) : Elem<T>::bc(0.0));
                    EDft<T, -1, R>::run(v);
#pragma unroll
                    for (int r = 0; r < R; ++r) a[r] = v[r];
                }
            }
        });
        __syncthreads();
        stages_back<T, -1>(buf, p, lay, tw);
        stage_inplace<T, -1, true, true>(buf, p, 0, lay, tw);
        __syncthreads();
    }
    chain_start();
    // the merge, in the order of the frequencies: natural after the transform back (kNonlin),
    // through the position table otherwise
    cx<T>* rows = static_cast<cx<T>*>(out) + blockIdx.z * ms + (int64_t)row0 * nxh;
    auto at = [&](int k) { return MODE == kNonlin ? gpad(p, k) : pos[k]; };
    for (int e = threadIdx.x; e < nl * nxh; e += blockDim.x) {
        const int i = fdiv(e, by_nxh), k = e - i * nxh;
        const el<T>* y = buf + i * p.np;
        el<T> v;
        if (even) v = r2c_post<T>(y[at(k == L ? 0 : k)], y[at(k == 0 ? 0 : L - k)], post[k]);
        else v = y[at(k)];
        cx<T>* a = rows + (int64_t)(W * i) * nxh + k;
        a[0] = Elem<T>::template line<0>(v);
        if (W > 1 && 2 * i + 1 < nr) a[nxh] = Elem<T>::template line<1>(v);
    }
}

// f(std::integral_constant<int, R>) for the first radix of a paired plan (2 .. kPairRadix)
template <class F> __device__ __forceinline__ void by_pair_radix(int R, F&& f) {
    switch (R) {
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 3: f(std::integral_constant<int, 3>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
    }
}

// The stepper's x pass for even nx whose plan starts with a small radix (GPlan of the packed
// length L = nx/2): as k_rows<kNonlin>, with the split and the merge of the real transforms in
// the registers of the first stage.  A thread takes the butterflies j and m - j of that stage,
// which hold the mode pairs k, L - k: each mode is loaded once, one twiddle product serves both
// ends of a pair, and the merged modes go straight to global memory, where the general kernel
// wrote the spectrum to shared memory and read every element twice more.
// Z[k] = e + i o, Z[L-k] = conj(e - i o) with e = X[k] + conj X[L-k], o = conj(w)(X[k] - conj X[L-k]);
// X[k] = (s - i t) / 2, X[L-k] = conj(s + i t) / 2 with s, t likewise from Y (w = W_nx^k).
// 80 registers (three CTAs per SM): at 64 the radix-5 pair spills.  A step against the general kernel,
// us: 240x200x180 FP32 149.0 -> 144.2, 1000x900 FP64 39.6 -> 35.1, 90x80x100 FP32
// 37.5 -> 33.7, 2400x2000 FP32 95.8 -> 90.2.
template <typename T, bool ODD>
__global__ void __launch_bounds__(kGenThreads, 3)
    k_xpass(cx<T>* field, int nrows, int nxh, const __grid_constant__ GPlan p, const el<T>* __restrict__ tw,
            const el<T>* __restrict__ post, int rpc, int W, FastDiv by_half, double mul, double C, double mu,
            int64_t ms, int lead) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    el<T>* buf = reinterpret_cast<el<T>*>(smem_raw);
    chain_start(lead);
    chain_wait();
    using E = Elem<T>;
    using CC = CE<T>;
    if (E::lines == 1) W = 1;
    const int row0 = blockIdx.x * rpc * W;
    const int nr = min(rpc * W, nrows - row0), nl = W > 1 ? (nr + 1) / 2 : nr;
    const RowLines<ODD> lay{nl, p.np};
    const int L = p.n;
    const GStage& s0 = p.st[0];
    const int m = s0.m, half = m / 2 + 1, total = nl * half;
    cx<T>* rows = field + blockIdx.z * ms + (int64_t)row0 * nxh;  // grid z: fields of a batch
    by_pair_radix(s0.R, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            const int i = fdiv(e, by_half), j = e - i * half, jm = j ? m - j : 0;
            const cx<T>* a = rows + (int64_t)(W * i) * nxh;
            const cx<T>* b = a + (W > 1 && 2 * i + 1 < nr ? nxh : 0);  // (an odd last row pairs with itself)
            el<T> v[R], u[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int k = j + r * m;
                const el<T> xk = E::pack(a[k], b[k]), xm = E::pack(a[L - k], b[L - k]);
                const el<T> ev = E::make(vadd(E::re(xk), E::re(xm)), vsub(E::im(xk), E::im(xm)));
                const el<T> d = E::make(vsub(E::re(xk), E::re(xm)), vadd(E::im(xk), E::im(xm)));
                const el<T> o = CC::template cmulw<1>(d, post[k]);
                v[r] = CC::template addi<1>(ev, o);
                u[R - 1 - r] = E::make(vadd(E::re(ev), E::im(o)), vsub(E::re(o), E::im(ev)));
            }
            auto store = [&](el<T>* w, int q) {
                EDft<T, 1, R>::run(w);
                el<T>* t = buf + lay.at(i, gpad(p, q));
                const el<T>* tws = tw + s0.tw + q;
                t[0] = w[0];
#pragma unroll
                for (int r = 1; r < R; ++r) t[r * s0.ms] = CC::template cmulw<1>(w[r], tws[(r - 1) * m]);
            };
            store(v, j);
            if (jm != j) store(u, jm);
        }
    });
    __syncthreads();
    stages_mid<T, 1>(buf, p, lay, tw);
    {
        // the last inverse stage, the cubic term and the first forward stage on one set of
        // registers
        const auto bmul = E::bc(mul), nC = E::bc(-C), nmu = E::bc(-mu);
        const GStage& s = p.st[p.nst - 1];
        const int count = lay.count(p.kstep);
        by_radix<ODD>(s.R, [&](auto RC) {
            constexpr int R = decltype(RC)::value;
            if constexpr (R > 0) {
                for (int e = threadIdx.x; e < count; e += blockDim.x) {
                    int i, b;
                    lay.split(e, p.kstep, s.by_nb, i, b);
                    el<T>* a = buf + lay.at(i, b * s.Ms);
                    el<T> v[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) v[r] = a[r];
                    EDft<T, 1, R>::run(v);
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        v[r] = E::make(cubic(E::re(v[r]), bmul, nC, nmu), cubic(E::im(v[r]), bmul, nC, nmu));
                    EDft<T, -1, R>::run(v);
#pragma unroll
                    for (int r = 0; r < R; ++r) a[r] = v[r];
                }
            }
        });
    }
    __syncthreads();
    stages_back<T, -1>(buf, p, lay, tw);
    chain_start();
    by_pair_radix(s0.R, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            const int i = fdiv(e, by_half), j = e - i * half, jm = j ? m - j : 0;
            cx<T>* a = rows + (int64_t)(W * i) * nxh;
            const bool two = W > 1 && 2 * i + 1 < nr;
            auto load = [&](el<T>* w, int q) {
                const el<T>* t = buf + lay.at(i, gpad(p, q));
                const el<T>* tws = tw + s0.tw + q;
                w[0] = t[0];
#pragma unroll
                for (int r = 1; r < R; ++r) w[r] = CC::template cmulw<-1>(t[r * s0.ms], tws[(r - 1) * m]);
                EDft<T, -1, R>::run(w);
            };
            auto put = [&](int k, el<T> z) {
                a[k] = E::template line<0>(z);
                if (two) a[nxh + k] = E::template line<1>(z);
            };
            el<T> v[R], u[R];
            load(v, j);
            if (jm != j) {
                load(u, jm);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int k = j + r * m;
                    const el<T> zk = v[r], zm = u[R - 1 - r];
                    const el<T> s = E::make(vadd(E::re(zk), E::re(zm)), vsub(E::im(zk), E::im(zm)));
                    const el<T> d = E::make(vsub(E::re(zk), E::re(zm)), vadd(E::im(zk), E::im(zm)));
                    const el<T> t = CC::template cmulw<-1>(d, post[k]);
                    put(k, CC::scale(CC::template addi<-1>(s, t), 0.5));
                    const el<T> q = CC::template addi<1>(s, t);
                    put(L - k, E::make(vmul(E::re(q), E::bc(0.5)), vmul(E::im(q), E::bc(-0.5))));
                }
            } else {
                // j = 0 or m/2: the pairs lie within the butterfly (and k = 0 gives k = L too)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int k = j + r * m;
                    const el<T> zm = j ? v[R - 1 - r] : v[(R - r) % R];
                    put(k, r2c_post<T>(v[r], zm, post[k]));
                }
                if (j == 0) put(L, r2c_post<T>(v[0], v[0], post[L]));
            }
        }
    });
}

}  // namespace

template <typename T, bool ODD> cudaError_t gen_attrs_of() {
    const int m = (int)kMaxDynSmem;
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(k_cols<T, -1, ODD>, attr, m);
    if (!e) e = cudaFuncSetAttribute(k_cols<T, 1, ODD>, attr, m);
    if (!e) e = cudaFuncSetAttribute(k_rows<T, kR2C, ODD>, attr, m);
    if (!e) e = cudaFuncSetAttribute(k_rows<T, kC2R, ODD>, attr, m);
    if (!e) e = cudaFuncSetAttribute(k_rows<T, kNonlin, ODD>, attr, m);
    if (!e) e = cudaFuncSetAttribute(k_xpass<T, ODD>, attr, m);
    return e;
}
template <typename T> cudaError_t gen_attrs() {
    const cudaError_t e = gen_attrs_of<T, false>();
    return e ? e : gen_attrs_of<T, true>();
}

template <typename T>
cudaError_t gen_cols(const pfc_ctx* c, int axis, int dir, const void* in, void* out, double scale) {
    const AxisPlan& ap = axis == 1 ? c->py : c->pz;
    const int n = ap.plan.n;
    if (n == 1 && in == out && scale == 1.0) return cudaSuccess;
    int64_t es, os;
    int no;
    if (axis == 1) { es = c->nxh; os = (int64_t)c->ny * c->nxh; no = c->nz; }
    else { es = (int64_t)c->ny * c->nxh; os = c->nxh; no = c->ny; }
    const int tile = ap.w << ap.lg;
    dim3 grid((c->nxh + tile - 1) / tile, no, c->batch);
    auto k = ap.plan.odd ? (dir < 0 ? k_cols<T, -1, true> : k_cols<T, 1, true>)
                         : (dir < 0 ? k_cols<T, -1, false> : k_cols<T, 1, false>);
    return chain_launch(c, k, grid, ap.threads, ap.smem, (const cx<T>*)in, (cx<T>*)out, c->nxh, es, os, ap.plan,
                        (const el<T>*)c->gtw, c->fft_tab, ap.lg, ap.w, scale, c->mstride);
}

template <typename T>
cudaError_t gen_rows(const pfc_ctx* c, int mode, const void* in, void* out, double mul, double C, double mu) {
    const int nrows = c->ny * c->nz;
    if (mode == kNonlin && c->px2.plan.nst) {
        const AxisPlan& ap = c->px2;
        const el<T>* tw = (const el<T>*)c->gtw;
        const int rows = ap.lines * ap.w;
        auto k = ap.plan.odd ? k_xpass<T, true> : k_xpass<T, false>;
        return chain_launch(c, k, dim3((nrows + rows - 1) / rows, 1, c->batch), ap.threads, ap.smem,
                            (cx<T>*)out, nrows, c->nxh, ap.plan, tw, tw + c->post_off, ap.lines, ap.w,
                            make_fastdiv(ap.plan.st[0].m / 2 + 1), mul, C, mu, c->mstride);
    }
    const AxisPlan& ap = c->px;
    const el<T>* tw = (const el<T>*)c->gtw;
    const int rows = ap.lines * ap.w;
    // (the plain transforms run on one field; the x pass on all fields of a batch)
    dim3 grid((nrows + rows - 1) / rows, 1, mode == kNonlin ? c->batch : 1);
    auto k = ap.plan.odd ? (mode == kR2C ? k_rows<T, kR2C, true> : mode == kC2R ? k_rows<T, kC2R, true> : k_rows<T, kNonlin, true>)
                         : (mode == kR2C ? k_rows<T, kR2C, false> : mode == kC2R ? k_rows<T, kC2R, false> : k_rows<T, kNonlin, false>);
    return chain_launch(c, k, grid, ap.threads, ap.smem, in, out, nrows, c->nx, ap.plan, tw, c->fft_tab,
                        tw + c->post_off, ap.lines, ap.w, mul, C, mu, c->mstride, make_fastdiv(c->nxh));
}
}  // namespace pfc
