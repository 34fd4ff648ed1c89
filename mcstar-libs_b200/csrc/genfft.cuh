// The general-length FFT engine: lines of any length with prime factors up to 31, FP32 and
// FP64, in shared memory, for the passes whose length has no register kernel.
//
// A length n is split as R_1 R_2 ... R_S (at least two stages; radices up to 10, chosen on
// the host for the fewest stages: radices 12, 15 and 16 took 128 registers and measured
// slower, 240 x 200 x 180 FP32 z pass 0.088 against 0.060 ms).  The transform is in place, decimation in frequency:
// stage s works on blocks of M_s = n / (R_1 ... R_{s-1}) positions; with m = M_s / R_s,
// butterfly j < m of a block takes the positions j + r m, runs the R_s-point DFT in
// registers, multiplies output r by W_{M_s}^{j r} and writes back to the same positions.
// After the last stage position p holds X[k] with k the digit reversal of p.  The transform
// back (decimation in time) runs the stages in the opposite order, twiddles before the DFT,
// from digit-reversed to natural order.  So
//  - a butterfly reads and writes its own positions: one barrier per stage, one buffer;
//  - the first stage of a column transform reads global memory and the last one writes it
//    (rows k of a column are separate segments anyway: the reversal costs one table read
//    per butterfly): S - 1 trips through shared memory, where a Stockham transform staged
//    in two buffers took S + 1;
//  - a forward and an inverse transform with a pointwise map between them never reorder.
//
// Padding: where R_S is even, one element follows every R_S positions (position p sits at
// p + p / R_S), so that the last stages' strides over the banks are odd.
#pragma once
#include <type_traits>
#include "regfft.cuh"

namespace pfc {

constexpr int kMaxStages = 12;
constexpr int kMaxOddRadix = 31;  // largest prime radix of the general stage

struct GStage {
    int R, m, nb; // radix; butterflies per block; butterflies of a line (n / R)
    int ms, Ms;   // shared-memory distance of a butterfly's elements, of two blocks
    int tw;       // W_M^{j r} at tw + (r - 1) m + j (forward sign; elements, FP32: the factor twice)
    int rt;       // W_R^q of a radix without a hand-written DFT
    FastDiv by_m, by_nb;
};
struct GPlan {
    int n, nst;
    int odd;      // 1: a radix of 7, or of 11 to 31
    int np;       // shared-memory elements of a line (padding included)
    int rl, pad;  // last radix; 1 where it is even (padded)
    int kstep;    // n / rl: distance of the frequencies of a last-stage butterfly
    int rev;      // int table: frequency of output 0 of last-stage butterfly b, b < n / rl
    int pos;      // int table: shared-memory position of frequency k, k < n
    int nbmax;    // the most butterflies of a stage
    int nblong;   // the butterflies of the largest prime radix above 10 (none: nbmax)
    FastDiv by_rl, by_n;
    GStage st[kMaxStages];
};

// ---- elements ---------------------------------------------------------------------------------
// An element of a line is 16 bytes: one complex FP64 value, or in FP32 the complex values of
// two lines (columns or rows) side by side, which every step of a transform treats alike:
// packed FP32 instructions (add, mul, fma .f32x2) do both lines' arithmetic, and one index,
// one twiddle and one shared-memory access serve the two.  The passes are bound by
// instruction issue, not by the FP32 pipe (one line per thread: 111 warp instructions per 32
// elements of a 200-point column, 17% of the FMA pipe).
struct f2 {  // two FP32 values in one 64-bit register pair: the first line's, the second line's
    unsigned long long v;
};
struct __align__(16) c2f {
    f2 re, im;
};
__device__ __forceinline__ f2 mkf2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 f2_of(f2 r) {
    float2 a;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r.v));
    return a;
}
__device__ __forceinline__ f2 vadd(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 vsub(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 vmul(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 vfma(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }
__device__ __forceinline__ double vsub(double a, double b) { return a - b; }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }

template <typename T> struct Elem;
template <> struct Elem<float> {
    using type = c2f;  // the element, and a twiddle factor (the same for both lines)
    using real = f2;
    static constexpr int lines = 2;
    __device__ __forceinline__ static f2 bc(double c) { return mkf2((float)c, (float)c); }
    __device__ __forceinline__ static c2f make(f2 re, f2 im) { return c2f{re, im}; }
    __device__ __forceinline__ static f2 re(const c2f& a) { return a.re; }
    __device__ __forceinline__ static f2 im(const c2f& a) { return a.im; }
    // from and to the values of the two lines
    __device__ __forceinline__ static c2f pack(float2 a, float2 b) { return c2f{mkf2(a.x, b.x), mkf2(a.y, b.y)}; }
    template <int L> __device__ __forceinline__ static float2 line(const c2f& v) {
        const float2 r = f2_of(v.re), i = f2_of(v.im);
        return L == 0 ? make_float2(r.x, i.x) : make_float2(r.y, i.y);
    }
};
template <> struct Elem<double> {
    using type = double2;
    using real = double;
    static constexpr int lines = 1;
    __device__ __forceinline__ static double bc(double c) { return c; }
    __device__ __forceinline__ static double2 make(double re, double im) { return make_double2(re, im); }
    __device__ __forceinline__ static double re(const double2& a) { return a.x; }
    __device__ __forceinline__ static double im(const double2& a) { return a.y; }
    __device__ __forceinline__ static double2 pack(double2 a, double2) { return a; }
    template <int L> __device__ __forceinline__ static double2 line(const double2& v) { return v; }
};
template <typename T> using el = typename Elem<T>::type;

// complex operations on elements
template <typename T> struct CE {
    using E = Elem<T>;
    using e = el<T>;
    using r = typename E::real;
    __device__ __forceinline__ static e add(e a, e b) { return E::make(vadd(E::re(a), E::re(b)), vadd(E::im(a), E::im(b))); }
    __device__ __forceinline__ static e sub(e a, e b) { return E::make(vsub(E::re(a), E::re(b)), vsub(E::im(a), E::im(b))); }
    // a + DIR i b
    template <int DIR> __device__ __forceinline__ static e addi(e a, e b) {
        return DIR > 0 ? E::make(vsub(E::re(a), E::im(b)), vadd(E::im(a), E::re(b)))
                       : E::make(vadd(E::re(a), E::im(b)), vsub(E::im(a), E::re(b)));
    }
    template <int DIR> __device__ __forceinline__ static e rot(e a) {
        const r n = E::bc(-1.0);
        return DIR > 0 ? E::make(vmul(E::im(a), n), E::re(a)) : E::make(E::im(a), vmul(E::re(a), n));
    }
    __device__ __forceinline__ static e neg(e a) {
        const r n = E::bc(-1.0);
        return E::make(vmul(E::re(a), n), vmul(E::im(a), n));
    }
    // a + s b and a + DIR s i b, s a constant
    __device__ __forceinline__ static e fma(e a, e b, double s) {
        const r c = E::bc(s);
        return E::make(vfma(E::re(b), c, E::re(a)), vfma(E::im(b), c, E::im(a)));
    }
    template <int DIR> __device__ __forceinline__ static e fmai(e a, e b, double s) {
        return E::make(vfma(E::im(b), E::bc(-DIR * s), E::re(a)), vfma(E::re(b), E::bc(DIR * s), E::im(a)));
    }
    __device__ __forceinline__ static e scale(e a, double s) {
        const r c = E::bc(s);
        return E::make(vmul(E::re(a), c), vmul(E::im(a), c));
    }
    // a (c + i s), constants
    __device__ __forceinline__ static e cmulc(e a, double c, double s) {
        return E::make(vfma(E::im(a), E::bc(-s), vmul(E::re(a), E::bc(c))),
                       vfma(E::re(a), E::bc(s), vmul(E::im(a), E::bc(c))));
    }
    // a w (DIR < 0) or a conj(w) (DIR > 0): twiddles are stored with the forward sign
    template <int DIR> __device__ __forceinline__ static e cmulw(e a, e w) {
        const r nw = vmul(E::im(w), E::bc(-1.0));
        const r p = DIR < 0 ? nw : E::im(w), q = DIR < 0 ? E::im(w) : nw;
        return E::make(vfma(E::im(a), p, vmul(E::re(a), E::re(w))), vfma(E::re(a), q, vmul(E::im(a), E::re(w))));
    }
};

// ---- DFTs in registers, X[k] = sum_n x[n] exp(DIR 2 pi i n k / R), natural order, in place -----
template <typename T, int DIR, int R> struct EDft;
template <typename T, int DIR> struct EDft<T, DIR, 1> { __device__ __forceinline__ static void run(el<T>*) {} };
template <typename T, int DIR> struct EDft<T, DIR, 2> {
    __device__ __forceinline__ static void run(el<T>* v) {
        const el<T> a = v[0], b = v[1];
        v[0] = CE<T>::add(a, b);
        v[1] = CE<T>::sub(a, b);
    }
};
template <typename T, int DIR> struct EDft<T, DIR, 3> {
    __device__ __forceinline__ static void run(el<T>* v) {
        using C = CE<T>;
        const el<T> t = C::add(v[1], v[2]), d = C::sub(v[1], v[2]);
        const el<T> m = C::fma(v[0], t, -0.5);
        v[0] = C::add(v[0], t);
        v[1] = C::template fmai<DIR>(m, d, 0.86602540378443864676);
        v[2] = C::template fmai<DIR>(m, d, -0.86602540378443864676);
    }
};
template <typename T, int DIR> struct EDft<T, DIR, 4> {
    __device__ __forceinline__ static void run(el<T>* v) {
        using C = CE<T>;
        const el<T> s02 = C::add(v[0], v[2]), d02 = C::sub(v[0], v[2]), s13 = C::add(v[1], v[3]), d13 = C::sub(v[1], v[3]);
        v[0] = C::add(s02, s13);
        v[2] = C::sub(s02, s13);
        v[1] = C::template addi<DIR>(d02, d13);
        v[3] = C::template addi<-DIR>(d02, d13);
    }
};
template <typename T, int DIR> struct EDft<T, DIR, 5> {
    __device__ __forceinline__ static void run(el<T>* v) {
        using C = CE<T>;
        const double c1 = 0.30901699437494742410, c2 = -0.80901699437494742410;
        const double s1 = 0.95105651629515357212, s2 = 0.58778525229247312917;
        const el<T> a14 = C::add(v[1], v[4]), d14 = C::sub(v[1], v[4]), a23 = C::add(v[2], v[3]), d23 = C::sub(v[2], v[3]);
        const el<T> p1 = C::fma(C::fma(v[0], a14, c1), a23, c2), p2 = C::fma(C::fma(v[0], a14, c2), a23, c1);
        const el<T> q1 = C::fma(C::scale(d14, s1), d23, s2), q2 = C::fma(C::scale(d14, s2), d23, -s1);
        v[0] = C::add(v[0], C::add(a14, a23));
        v[1] = C::template addi<DIR>(p1, q1);
        v[4] = C::template addi<-DIR>(p1, q1);
        v[2] = C::template addi<DIR>(p2, q2);
        v[3] = C::template addi<-DIR>(p2, q2);
    }
};
template <typename T, int DIR> struct EDft<T, DIR, 8> {
    __device__ __forceinline__ static void run(el<T>* v) {
        using C = CE<T>;
        const double h = 0.70710678118654752440;
        el<T> e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        EDft<T, DIR, 4>::run(e);
        EDft<T, DIR, 4>::run(o);
        // W8^1 o1 = h (o1 + DIR i o1), W8^2 o2 = DIR i o2, W8^3 o3 = -h (o3 - DIR i o3)
        const el<T> p = C::template addi<DIR>(o[1], o[1]), q = C::template addi<-DIR>(o[3], o[3]);
        v[0] = C::add(e[0], o[0]);
        v[4] = C::sub(e[0], o[0]);
        v[1] = C::fma(e[1], p, h);
        v[5] = C::fma(e[1], p, -h);
        v[2] = C::template addi<DIR>(e[2], o[2]);
        v[6] = C::template addi<-DIR>(e[2], o[2]);
        v[3] = C::fma(e[3], q, -h);
        v[7] = C::fma(e[3], q, h);
    }
};

// a exp(DIR 2 pi i K / N), the trivial angles at compile time
template <int N, int K, int DIR> struct TwD {
    static constexpr double re = ct::cos2pi(K, N);
    static constexpr double im = DIR * ct::sin2pi(K, N);
};
template <typename T, int N, int K, int DIR> __device__ __forceinline__ el<T> twmul_e(el<T> a) {
    constexpr int k = ((K % N) + N) % N;
    if constexpr (k == 0) {
        return a;
    } else if constexpr (4 * k == N) {
        return CE<T>::template rot<DIR>(a);
    } else if constexpr (2 * k == N) {
        return CE<T>::neg(a);
    } else if constexpr (4 * k == 3 * N) {
        return CE<T>::template rot<-DIR>(a);
    } else {
        return CE<T>::cmulc(a, TwD<N, k, DIR>::re, TwD<N, k, DIR>::im);
    }
}

// R = R1 R2 with coprime factors (Good-Thomas: n = R2 n1 + R1 n2, k by the Chinese remainder
// theorem, no twiddles)
constexpr int crt(int k1, int r1, int k2, int r2) {
    for (int k = 0; k < r1 * r2; ++k)
        if (k % r1 == k1 && k % r2 == k2) return k;
    return 0;
}
template <int K1, int R1, int K2, int R2> struct Crt {
    static constexpr int value = crt(K1, R1, K2, R2);
};
template <typename T, int DIR, int R1, int R2> struct DftPfa {
    __device__ __forceinline__ static void run(el<T>* v) {
        el<T> a[R2][R1];
        sfor<0, R2>([&](auto b) {
            sfor<0, R1>([&](auto c) { a[b.value][c.value] = v[(R2 * c.value + R1 * b.value) % (R1 * R2)]; });
            EDft<T, DIR, R1>::run(a[b.value]);
        });
        sfor<0, R1>([&](auto c) {
            el<T> b[R2];
#pragma unroll
            for (int q = 0; q < R2; ++q) b[q] = a[q][c.value];
            EDft<T, DIR, R2>::run(b);
            sfor<0, R2>([&](auto q) { v[Crt<c.value, R1, q.value, R2>::value] = b[q.value]; });
        });
    }
};
// R = Q^2 (Cooley-Tukey: twiddles are compile-time constants)
template <typename T, int DIR, int Q> struct DftSq {
    __device__ __forceinline__ static void run(el<T>* v) {
        el<T> a[Q][Q];
        sfor<0, Q>([&](auto b) {
#pragma unroll
            for (int c = 0; c < Q; ++c) a[b.value][c] = v[Q * c + b.value];
            EDft<T, DIR, Q>::run(a[b.value]);
        });
        sfor<0, Q>([&](auto c) {
            el<T> b[Q];
            sfor<0, Q>([&](auto q) { b[q.value] = twmul_e<T, Q * Q, q.value * c.value, DIR>(a[q.value][c.value]); });
            EDft<T, DIR, Q>::run(b);
#pragma unroll
            for (int q = 0; q < Q; ++q) v[c.value + Q * q] = b[q];
        });
    }
};
// an odd prime R by the sums and differences of the pairs r, R - r
template <typename T, int DIR, int R> struct DftOdd {
    __device__ __forceinline__ static void run(el<T>* v) {
        using C = CE<T>;
        constexpr int h = R / 2;
        el<T> s[h + 1], d[h + 1];
#pragma unroll
        for (int r = 1; r <= h; ++r) {
            s[r] = C::add(v[r], v[R - r]);
            d[r] = C::sub(v[r], v[R - r]);
        }
        const el<T> x0 = v[0];
#pragma unroll
        for (int r = 1; r <= h; ++r) v[0] = C::add(v[0], s[r]);
        sfor<1, h + 1>([&](auto k) {
            el<T> a = x0, b = C::scale(d[1], TwD<R, k.value, 1>::im);
            sfor<1, h + 1>([&](auto r) {
                constexpr int q = k.value * r.value % R;
                a = C::fma(a, s[r.value], TwD<R, q, 1>::re);
                if constexpr (r.value > 1) b = C::fma(b, d[r.value], TwD<R, q, 1>::im);
            });
            v[k.value] = C::template addi<DIR>(a, b);
            v[R - k.value] = C::template addi<-DIR>(a, b);
        });
    }
};
template <typename T, int DIR> struct EDft<T, DIR, 6> : DftPfa<T, DIR, 3, 2> {};
template <typename T, int DIR> struct EDft<T, DIR, 7> : DftOdd<T, DIR, 7> {};
template <typename T, int DIR> struct EDft<T, DIR, 9> : DftSq<T, DIR, 3> {};
template <typename T, int DIR> struct EDft<T, DIR, 10> : DftPfa<T, DIR, 5, 2> {};

// f(std::integral_constant<int, R>) for a stage's radix; 0 stands for a prime radix from 11 up.  ODD:
// the plan may have radices 7 and 11 to 31.  Those are instantiated apart: in one body with the others
// they take registers from all (192^3 FP64 204.6 us per step with all radices in one body, 201.3 so;
// 240 x 200 x 180 FP32 with noise 168.4 and 165.9).
template <bool ODD, class F> __device__ __forceinline__ void by_radix(int R, F&& f) {
    switch (R) {
        case 1: f(std::integral_constant<int, 1>{}); break;
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 3: f(std::integral_constant<int, 3>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 9: f(std::integral_constant<int, 9>{}); break;
        case 10: f(std::integral_constant<int, 10>{}); break;
        default:
            if constexpr (ODD) {
                if (R == 7) f(std::integral_constant<int, 7>{});
                else f(std::integral_constant<int, 0>{});
            }
            break;
    }
}

// One butterfly: values get(r), results put(r, value).  kDit: twiddles before the DFT, else
// after it; kTw false: none (the last stage, m = 1).
template <typename T, int DIR, int R, bool kDit, bool kTw, class Get, class Put>
__device__ __forceinline__ void gbfly(const GStage& s, const el<T>* __restrict__ tw, int j, Get get, Put put) {
    using C = CE<T>;
    const el<T>* tws = tw + s.tw + j;
    if constexpr (R > 0) {
        el<T> v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = get(r);
        if (kTw && kDit) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = C::template cmulw<DIR>(v[r], tws[(r - 1) * s.m]);
        }
        EDft<T, DIR, R>::run(v);
        if (kTw && !kDit) {
#pragma unroll
            for (int r = 1; r < R; ++r) v[r] = C::template cmulw<DIR>(v[r], tws[(r - 1) * s.m]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) put(r, v[r]);
    } else {
        // A prime radix from 11 up, the roots of unity W_R^q from the plan's table: with the sums and
        // differences s_r, d_r of the pairs r, R - r,
        //   X[k], X[R-k] = x_0 + sum_r s_r cos(2 pi k r / R) +- DIR i sum_r d_r sin(2 pi k r / R),
        // two k at a time, and the loads of four pairs in flight.  (Loaded one by one, and multiplied
        // out as R^2 complex products, with the row plan of one row per CTA: a 247 x 105 x 182 FP64
        // step 3860 us, now 367.)
        using RR = typename Elem<T>::real;
        el<T> v[kMaxOddRadix];
        const el<T>* wr = tw + s.rt;
        const int n = s.R, h = n / 2;
        v[0] = get(0);
        el<T> sum = v[0];
#pragma unroll 4
        for (int r = 1; r <= h; ++r) {
            el<T> a = get(r), b = get(n - r);
            if (kTw && kDit) {
                a = C::template cmulw<DIR>(a, tws[(r - 1) * s.m]);
                b = C::template cmulw<DIR>(b, tws[(n - r - 1) * s.m]);
            }
            v[r] = C::add(a, b);
            v[n - r] = C::sub(a, b);
            sum = C::add(sum, v[r]);
        }
        put(0, sum);
        for (int k = 1; k <= h; k += 2) {
            el<T> a0 = v[0], a1 = v[0], b0 = Elem<T>::make(Elem<T>::bc(0.0), Elem<T>::bc(0.0)), b1 = b0;
            int q0 = 0, q1 = 0;
#pragma unroll 4
            for (int r = 1; r <= h; ++r) {
                q0 += k;
                if (q0 >= n) q0 -= n;
                q1 += k + 1;
                if (q1 >= n) q1 -= n;
                const el<T> x = v[r], y = v[n - r];
                auto acc = [&](el<T>& a, el<T>& b, const el<T>& w) {  // w = (cos, -sin)
                    const RR c = Elem<T>::re(w), t = Elem<T>::im(w);
                    a = Elem<T>::make(vfma(Elem<T>::re(x), c, Elem<T>::re(a)), vfma(Elem<T>::im(x), c, Elem<T>::im(a)));
                    b = Elem<T>::make(vfma(Elem<T>::re(y), t, Elem<T>::re(b)), vfma(Elem<T>::im(y), t, Elem<T>::im(b)));
                };
                acc(a0, b0, wr[q0]);
                acc(a1, b1, wr[q1]);
            }
            auto out = [&](int j, el<T> x) {
                put(j, kTw && !kDit ? C::template cmulw<DIR>(x, tws[(j - 1) * s.m]) : x);
            };
            out(k, C::template addi<-DIR>(a0, b0));
            out(n - k, C::template addi<DIR>(a0, b0));
            if (k < h) {
                out(k + 1, C::template addi<-DIR>(a1, b1));
                out(n - k - 1, C::template addi<DIR>(a1, b1));
            }
        }
    }
}

// Shared-memory position of position p of a line.
__device__ __forceinline__ int gpad(const GPlan& p, int i) { return p.pad ? i + fdiv(i, p.by_rl) : i; }

// How a pass lays its lines out: element position a of line i at at(i, a), and butterfly
// e of a stage with nb butterflies per line -> (line, index).
template <bool ODD> struct ColLines {  // lines interleaved: consecutive threads move one element of each of 2^lg lines (FP32: pairs)
    static constexpr bool odd = ODD;
    int lg;
    __device__ __forceinline__ int count(int nb) const { return nb << lg; }
    __device__ __forceinline__ void split(int e, int, FastDiv, int& i, int& q) const {
        i = e & ((1 << lg) - 1);
        q = e >> lg;
    }
    __device__ __forceinline__ int at(int i, int a) const { return (a << lg) + i; }
    __device__ __forceinline__ int step(int a) const { return a << lg; }
};
template <bool ODD> struct RowLines {  // whole lines one after the other: consecutive threads move consecutive elements
    static constexpr bool odd = ODD;
    int lines, np;
    __device__ __forceinline__ int count(int nb) const { return lines * nb; }
    __device__ __forceinline__ void split(int e, int nb, FastDiv by_nb, int& i, int& q) const {
        i = fdiv(e, by_nb);
        q = e - i * nb;
    }
    __device__ __forceinline__ int at(int i, int a) const { return i * np + a; }
    __device__ __forceinline__ int step(int a) const { return a; }
};

// A stage from and to shared memory, in place.  kTw false: the last stage (m = 1).
template <typename T, int DIR, bool kDit, bool kTw, class L>
__device__ __forceinline__ void stage_inplace(el<T>* buf, const GPlan& p, int si, const L& lay,
                                              const el<T>* __restrict__ tw) {
    const GStage& s = p.st[si];
    const int total = lay.count(s.nb), step = lay.step(s.ms);
    by_radix<L::odd>(s.R, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            int i, q;
            lay.split(e, s.nb, s.by_nb, i, q);
            const int b = kTw ? fdiv(q, s.by_m) : q, j = kTw ? q - b * s.m : 0;
            el<T>* a = buf + lay.at(i, b * s.Ms + (kTw ? gpad(p, j) : 0));
            gbfly<T, DIR, R, kDit, kTw>(
                s, tw, j, [&](int r) { return a[r * step]; }, [&](int r, el<T> v) { a[r * step] = v; });
        }
    });
}

// The first stage of a transform from natural order: values in(i, k) of line i at k, into
// shared memory.
template <typename T, int DIR, class L, class In>
__device__ __forceinline__ void stage_first(el<T>* buf, const GPlan& p, const L& lay, const el<T>* __restrict__ tw,
                                            In in) {
    const GStage& s = p.st[0];
    const int total = lay.count(s.m), step = lay.step(s.ms);
    by_radix<L::odd>(s.R, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            int i, j;
            lay.split(e, s.m, s.by_nb, i, j);
            el<T>* a = buf + lay.at(i, gpad(p, j));
            gbfly<T, DIR, R, false, true>(
                s, tw, j, in(i, j, s.m), [&](int r, el<T> v) { a[r * step] = v; });
        }
    });
}

// The last stage (no twiddles) from shared memory: butterfly b of line i holds the
// frequencies k0 + r p.kstep, handed to out(i, k0)(r, value).
template <typename T, int DIR, class L, class Out>
__device__ __forceinline__ void stage_last(el<T>* buf, const GPlan& p, const L& lay, const el<T>* __restrict__ tw,
                                           const int* __restrict__ rev, Out out) {
    const GStage& s = p.st[p.nst - 1];
    const int total = lay.count(p.kstep), step = lay.step(1);
    by_radix<L::odd>(s.R, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        if constexpr (R > 0) {  // (the host appends a stage of radix 1 to a prime radix)
            for (int e = threadIdx.x; e < total; e += blockDim.x) {
                int i, b;
                lay.split(e, p.kstep, s.by_nb, i, b);
                const el<T>* a = buf + lay.at(i, b * s.Ms);
                gbfly<T, DIR, R, false, false>(
                    s, tw, 0, [&](int r) { return a[r * step]; }, out(i, rev[b]));
            }
        }
    });
}

// The last stage (no twiddles) at the start of a transform back to natural order: butterfly b
// of line i takes the frequencies k0 + r p.kstep, in(i, k0)(r), into shared memory.
template <typename T, int DIR, class L, class In>
__device__ __forceinline__ void stage_in(el<T>* buf, const GPlan& p, const L& lay, const el<T>* __restrict__ tw,
                                         const int* __restrict__ rev, In in) {
    const GStage& s = p.st[p.nst - 1];
    const int total = lay.count(p.kstep), step = lay.step(1);
    by_radix<L::odd>(s.R, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        if constexpr (R > 0) {
            for (int e = threadIdx.x; e < total; e += blockDim.x) {
                int i, b;
                lay.split(e, p.kstep, s.by_nb, i, b);
                el<T>* a = buf + lay.at(i, b * s.Ms);
                gbfly<T, DIR, R, true, false>(
                    s, tw, 0, in(i, rev[b]), [&](int r, el<T> v) { a[r * step] = v; });
            }
        }
    });
}

// The first stage's counterpart at the end of a transform back to natural order: butterfly
// j of line i holds the values at j + r m, handed to out(i, j, m)(r, value).
template <typename T, int DIR, class L, class Out>
__device__ __forceinline__ void stage_out(el<T>* buf, const GPlan& p, const L& lay, const el<T>* __restrict__ tw,
                                          Out out) {
    const GStage& s = p.st[0];
    const int total = lay.count(s.m), step = lay.step(s.ms);
    by_radix<L::odd>(s.R, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        for (int e = threadIdx.x; e < total; e += blockDim.x) {
            int i, j;
            lay.split(e, s.m, s.by_nb, i, j);
            const el<T>* a = buf + lay.at(i, gpad(p, j));
            gbfly<T, DIR, R, true, true>(s, tw, j, [&](int r) { return a[r * step]; }, out(i, j, s.m));
        }
    });
}

// Stages 1 .. S-2 (between the first and the last), a barrier after each: downwards from
// natural order, or upwards back to it.
template <typename T, int DIR, class L>
__device__ __forceinline__ void stages_mid(el<T>* buf, const GPlan& p, const L& lay, const el<T>* __restrict__ tw) {
    for (int s = 1; s + 1 < p.nst; ++s) {
        stage_inplace<T, DIR, false, true>(buf, p, s, lay, tw);
        __syncthreads();
    }
}
template <typename T, int DIR, class L>
__device__ __forceinline__ void stages_back(el<T>* buf, const GPlan& p, const L& lay, const el<T>* __restrict__ tw) {
    for (int s = p.nst - 2; s >= 1; --s) {
        stage_inplace<T, DIR, true, true>(buf, p, s, lay, tw);
        __syncthreads();
    }
}

}  // namespace pfc
