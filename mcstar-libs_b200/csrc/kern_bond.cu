// Steinhardt bond-order analysis of peak lists on the GPU, restating
// bond_order_analysis (bond-order-analysis/bond-order.cpp:289-349) in FP64:
//   keep atoms with field > ths; neighbours within rlim under the reference's
//   get_diff minimum image (bond-order.cpp:53-64); q_lm = <Y_lm> over neighbours for
//   l = 4, 6, 8; q_l, w_4 (and w_6, which the reference lacks), the neighbour-averaged
//   q-bar_l (self included), the reference's w4b (which averages only the last
//   neighbour, bond-order.cpp:205-219) and the solid-bond count xi (q6 dot > 0.7).
// The neighbour search bins atoms into cells of side >= rlim; each atom's list is
// sorted by index so the sums run in the reference's order.  Y_lm come from the
// normalised associated-Legendre upward recurrences with e^{i m phi} built by complex
// powers of (dx + i dy)/rho; the reference's pole band (prefF, bond-order.cpp:123-133:
// Y_lm = 0 for m > 0 when |1 - cos theta| < 1e-3 and for m < 0 when |1 + cos theta| <
// 1e-3) is kept.  Wigner 3j symbols come from the Racah formula, evaluated on the host.
#include <algorithm>
#include <cmath>
#include <vector>
#include "pfc_ctx.h"

namespace pfc {
namespace {

constexpr int kNQ = 9 + 13 + 17;         // q_lm, l = 4, 6, 8, m = -l..l
constexpr int kW4 = 61, kW6 = 127;       // (l l l; m1 m2 m3) with m1 + m2 + m3 = 0
__constant__ double c_nlm[3][9];         // normalisation of (l - m)! P_l^m, l = 4, 6, 8, m = 0..l
__constant__ double c_w4[kW4];
__constant__ int c_w4m[kW4][2];
__constant__ double c_w6[kW6];
__constant__ int c_w6m[kW6][2];
__constant__ int c_tables_ready;

struct BondScratch {
    double* pos;      // 3 * P
    int* keep_cnt;    // blocks
    int* keep_off;    // blocks + 1
    int* nb;          // P: neighbours of each atom
    int* nb_off;      // P + 1: exclusive scan of nb, the start of each atom's list in the pair buffer
    int* maxj;        // P
    double2* q;       // P * kNQ
    int* row_cnt;     // blocks
    int* row_off;     // blocks + 1
    int* cell_cnt;    // cells
    int* cell_off;    // cells + 1
    int* cell_fill;   // cells
    int* cell_atoms;  // P
    int* flags;       // [1] position outside the box, [2] kept count
};
constexpr int kMaxCellsDim = 64;
constexpr int kBlk = 256;

size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

// The per-atom scratch of P atoms (the neighbour lists live in a separate pair buffer,
// sized by the neighbour count the search finds).
size_t scratch_layout(int P, BondScratch* s, char* base) {
    const size_t blocks = (size_t)(P + kBlk - 1) / kBlk + 1;
    const size_t cells = (size_t)kMaxCellsDim * kMaxCellsDim * kMaxCellsDim;
    size_t off = 0;
    auto take = [&](size_t bytes) { char* p = base ? base + off : nullptr; off += align_up(bytes); return p; };
    BondScratch t;
    t.pos = (double*)take(sizeof(double) * 3 * P);
    t.keep_cnt = (int*)take(sizeof(int) * blocks);
    t.keep_off = (int*)take(sizeof(int) * (blocks + 1));
    t.nb = (int*)take(sizeof(int) * P);
    t.nb_off = (int*)take(sizeof(int) * ((size_t)P + 1));
    t.maxj = (int*)take(sizeof(int) * P);
    t.q = (double2*)take(sizeof(double2) * (size_t)P * kNQ);
    t.row_cnt = (int*)take(sizeof(int) * blocks);
    t.row_off = (int*)take(sizeof(int) * (blocks + 1));
    t.cell_cnt = (int*)take(sizeof(int) * cells);
    t.cell_off = (int*)take(sizeof(int) * (cells + 1));
    t.cell_fill = (int*)take(sizeof(int) * cells);
    t.cell_atoms = (int*)take(sizeof(int) * P);
    t.flags = (int*)take(sizeof(int) * 8);
    if (s) *s = t;
    return off;
}

template <typename T> struct MaxRecB;
template <> struct MaxRecB<float> { float i0, i1, i2; float field; };
template <> struct MaxRecB<double> { double i0, i1, i2; float field; };

// ---- compaction helpers -------------------------------------------------------------
// Exclusive scan of nb counts (and their total) by one CTA: tiles of 8 counts per thread, warp
// scans, a running total (a strided serial scan per thread took 8.3 us for 24 k counts, 7.2 now).
__global__ void __launch_bounds__(1024) k_scan_b(const int* __restrict__ counts, int nb, int* __restrict__ offsets) {
    constexpr int E = 8;
    __shared__ int wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int run = 0;
    for (int base = 0; base < nb; base += 1024 * E) {
        const int b = base + threadIdx.x * E;
        int v[E], s = 0;
#pragma unroll
        for (int i = 0; i < E; ++i) {
            v[i] = b + i < nb ? counts[b + i] : 0;
            s += v[i];
        }
        int inc = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        __syncthreads();  // (the last tile's reads of wsum)
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            int w = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += t;
            }
            wsum[lane] = w;
        }
        __syncthreads();
        int pos = run + inc - s + (warp ? wsum[warp - 1] : 0);
#pragma unroll
        for (int i = 0; i < E; ++i) {
            if (b + i < nb) offsets[b + i] = pos;
            pos += v[i];
        }
        run += wsum[31];
    }
    if (threadIdx.x == 0) offsets[nb] = run;
}

__device__ __forceinline__ int block_rank(bool f, int* wsum) {
    const unsigned m = __ballot_sync(0xffffffffu, f);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) wsum[warp] = __popc(m);
    __syncthreads();
    int pos = __popc(m & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w) pos += wsum[w];
    return pos;
}

template <typename T>
__global__ void __launch_bounds__(kBlk) k_keep_count(const MaxRecB<T>* __restrict__ in, int n, double ths,
                                                     int* __restrict__ cnt) {
    const int i = blockIdx.x * kBlk + threadIdx.x;
    const bool f = i < n && (double)in[i].field > ths;
    const int c = __syncthreads_count(f);
    if (threadIdx.x == 0) cnt[blockIdx.x] = c;
}

template <typename T>
__global__ void __launch_bounds__(kBlk) k_keep_write(const MaxRecB<T>* __restrict__ in, int n, double ths, double h0,
                                                     double h1, double h2, double box, const int* __restrict__ off,
                                                     double* __restrict__ pos, int* __restrict__ flags) {
    __shared__ int wsum[kBlk / 32];
    const int i = blockIdx.x * kBlk + threadIdx.x;
    const bool f = i < n && (double)in[i].field > ths;
    const int r = block_rank(f, wsum);
    if (!f) return;
    const int p = off[blockIdx.x] + r;
    const double x = (double)in[i].i0 * h0, y = (double)in[i].i1 * h1, z = (double)in[i].i2 * h2;
    pos[3 * p] = x; pos[3 * p + 1] = y; pos[3 * p + 2] = z;
    if (!(x >= 0.0 && x < box && y >= 0.0 && y < box && z >= 0.0 && z < box)) atomicOr(&flags[1], 1);
}

// ---- cells -----------------------------------------------------------------------------
__device__ __forceinline__ int cell_of(double v, double box, int nc) {
    int c = (int)floor(v / box * nc);
    return c < 0 ? 0 : (c >= nc ? nc - 1 : c);
}

__global__ void k_cell_count(const double* __restrict__ pos, const int* __restrict__ np, double box, int nc,
                             int* __restrict__ cnt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *np) return;
    const int c = (cell_of(pos[3 * i + 2], box, nc) * nc + cell_of(pos[3 * i + 1], box, nc)) * nc +
                  cell_of(pos[3 * i], box, nc);
    atomicAdd(&cnt[c], 1);
}

__global__ void k_cell_fill(const double* __restrict__ pos, const int* __restrict__ np, double box, int nc,
                            const int* __restrict__ off, int* __restrict__ fill, int* __restrict__ atoms) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *np) return;
    const int c = (cell_of(pos[3 * i + 2], box, nc) * nc + cell_of(pos[3 * i + 1], box, nc)) * nc +
                  cell_of(pos[3 * i], box, nc);
    atomicExch(&atoms[off[c] + atomicAdd(&fill[c], 1)], i);
}

// get_diff (bond-order.cpp:53-64) with its tie order
__device__ __forceinline__ double get_diff(double x1, double x2, double w) {
    const double d1 = x1 - x2, d2 = d1 - w, d3 = d1 + w;
    if (fabs(d1) < fabs(d2)) return fabs(d1) < fabs(d3) ? d1 : d3;
    return fabs(d2) < fabs(d3) ? d2 : d3;
}

// Whether r = sqrt(d2) <= rlim, the root taken only within 1e-12 of the limit
struct Within {
    double rlim, lo, hi;
    explicit Within(double r) : rlim(r), lo(r * r * (1.0 - 1e-12)), hi(r * r * (1.0 + 1e-12)) {
        if (!(r > 1e-100 && r < 1e150)) {  // (no square to compare with: always the root)
            lo = -1.0;
            hi = INFINITY;
        }
    }
    __device__ __forceinline__ bool operator()(double d2) const {
        return d2 <= lo || (d2 <= hi && sqrt(d2) <= rlim);
    }
};

// One warp per atom, its lanes over the atoms of the 27 cells around it (about 80 candidates in
// a crystal; a thread per atom left most of the GPU waiting for one dependent load after the
// other: 24 k atoms 63 and 70 us; now 20 and 25).  nc == 0 selects all pairs (positions outside the box or a
// box too small for three cells per side).  Counting pass (kFill false): nbc, maxjs.
// Filling pass: the list of atom i at nbr + nb_off[i], sorted by index (the reference sums
// over neighbours in index order, bond-order.cpp:289-349): each neighbour goes to its rank
// among the atom's neighbours; lists longer than kNbList are sorted in place by one lane.
constexpr int kNbWarps = 8, kNbList = 96;
template <bool kFill>
__global__ void __launch_bounds__(32 * kNbWarps)
    k_neighbours(const double* __restrict__ pos, const int* __restrict__ np, double box, Within within, int nc,
                 const int* __restrict__ cell_off, const int* __restrict__ cell_atoms,
                 const int* __restrict__ nb_off, int* __restrict__ nbr, int* __restrict__ nbc,
                 int* __restrict__ maxjs) {
    __shared__ int cell_end[kNbWarps][32], cell_at[kNbWarps][32], found[kNbWarps][kNbList];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blockIdx.x * kNbWarps + w;
    const int P = *np;
    if (i >= P) return;
    const double xi = pos[3 * i], yi = pos[3 * i + 1], zi = pos[3 * i + 2];
    const bool fits = !kFill || nbc[i] <= kNbList;
    int* list = kFill ? (fits ? found[w] : nbr + nb_off[i]) : nullptr;
    int cnt = 0, maxj = -1;
    auto visit = [&](int j, bool valid) {
        bool in = false;
        if (valid && j != i) {
            const double dx = get_diff(pos[3 * j], xi, box);
            const double dy = get_diff(pos[3 * j + 1], yi, box);
            const double dz = get_diff(pos[3 * j + 2], zi, box);
            in = within(dx * dx + dy * dy + dz * dz);
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (in) {
            if (kFill) list[cnt + __popc(m & ((1u << lane) - 1u))] = j;
            maxj = max(maxj, j);
        }
        cnt += __popc(m);
    };
    if (nc == 0) {
        for (int j = lane; j - lane < P; j += 32) visit(j, j < P);
    } else {
        // lane c < 27: cell c of the neighbourhood, its first atom and the running count
        int len = 0, at = 0;
        if (lane < 27) {
            const int cx = cell_of(xi, box, nc) + lane % 3 - 1, cy = cell_of(yi, box, nc) + lane / 3 % 3 - 1,
                      cz = cell_of(zi, box, nc) + lane / 9 - 1;
            const int c = ((cz + nc) % nc * nc + (cy + nc) % nc) * nc + (cx + nc) % nc;
            at = cell_off[c];
            len = cell_off[c + 1] - at;
        }
        int end = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += t;
        }
        cell_end[w][lane] = end;
        cell_at[w][lane] = at - (end - len);  // + candidate number = index into cell_atoms
        const int total = __shfl_sync(0xffffffffu, end, 31);
        __syncwarp();
        for (int f = lane; f - lane < total; f += 32) {
            int c = 0;  // the first cell whose end is beyond f
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                if (cell_end[w][c + o - 1] <= f) c += o;
            const bool valid = f < total;
            visit(valid ? cell_atoms[cell_at[w][c] + f] : 0, valid);
        }
    }
    if (!kFill) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) maxj = max(maxj, __shfl_xor_sync(0xffffffffu, maxj, o));
        if (lane == 0) {
            nbc[i] = cnt;
            maxjs[i] = maxj;
        }
        return;
    }
    __syncwarp();
    if (fits) {
        int* out = nbr + nb_off[i];
        for (int a = lane; a < cnt; a += 32) {
            const int v = list[a];
            int rank = 0;
            for (int b = 0; b < cnt; ++b) rank += list[b] < v;
            out[rank] = v;
        }
    } else if (lane == 0) {
        for (int a = 1; a < cnt; ++a) {
            const int v = list[a];
            int b = a - 1;
            while (b >= 0 && list[b] > v) { list[b + 1] = list[b]; --b; }
            list[b + 1] = v;
        }
    }
}

// q_lm of every atom, l = 4, 6, 8: nine lanes per atom (three atoms per warp), lane m = 0 .. 8 for
// +m and -m of all three l, whose P_l^m come from one upward recurrence in l.  The geometry of a
// neighbour is computed once, by one of the nine lanes, and passed round by shuffles; the
// sums over neighbours keep the list's order.  (A thread per atom and l: 132 us for 24 k atoms,
// the recurrences and the geometry three times over with FP64 divisions; now 46 us, half of the
// FP64 pipe.)
__global__ void __launch_bounds__(128) k_qlm(const double* __restrict__ pos, const int* __restrict__ np,
                                             const int* __restrict__ nbr, const int* __restrict__ nb_off,
                                             const int* __restrict__ nbc, double box, double2* __restrict__ q) {
    const int lane = threadIdx.x & 31, g = min(lane / 9, 2), m = lane < 27 ? lane - 9 * g : 0;
    const int P = *np;
    const int i = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 3 + g;
    const bool mine = i < P && lane < 27;
    const int cnt = i < P ? nbc[i] : 0;
    const int most = max(__shfl_sync(0xffffffffu, cnt, 0),
                         max(__shfl_sync(0xffffffffu, cnt, 9), __shfl_sync(0xffffffffu, cnt, 18)));
    if (most == 0) return;
    const int* list = nbr + (i < P ? nb_off[i] : 0);
    double xi = 0.0, yi = 0.0, zi = 0.0;
    if (i < P) { xi = pos[3 * i]; yi = pos[3 * i + 1]; zi = pos[3 * i + 2]; }
    // Q_l = (l - m)! P_l^m: Q_l = (2 l - 1) x Q_{l-1} - (l + m - 1)(l - m - 1) Q_{l-2}, whole
    // numbers where the recurrence of P_l^m divides by l - m (multiplying by its rounded reciprocal
    // instead costs digits)
    double rb[9];
#pragma unroll
    for (int l = 1; l <= 8; ++l) rb[l] = l > m ? (double)((l + m - 1) * (l - m - 1)) : 0.0;
    const double n4 = c_nlm[0][m], n6 = c_nlm[1][m], n8 = c_nlm[2][m];
    double2 p4 = make_double2(0.0, 0.0), p6 = p4, p8 = p4, s4 = p4, s6 = p4, s8 = p4;  // sums for +m, -m
    for (int a0 = 0; a0 < most; a0 += 9) {
        double x = 0.0, sn = 0.0, ex = 1.0, ey = 0.0;
        if (mine && a0 + m < cnt) {
            const int j = list[a0 + m];
            const double dx = get_diff(pos[3 * j], xi, box);
            const double dy = get_diff(pos[3 * j + 1], yi, box);
            const double dz = get_diff(pos[3 * j + 2], zi, box);
            x = dz / sqrt(dx * dx + dy * dy + dz * dz);
            const double rho = sqrt(dx * dx + dy * dy);
            if (rho > 0.0) { ex = dx / rho; ey = dy / rho; }
            sn = sqrt(fmax(0.0, 1.0 - x * x));
        }
        for (int b = 0; b < 9 && a0 + b < most; ++b) {
            const int src = 9 * g + b;
            const double xb = __shfl_sync(0xffffffffu, x, src), sb = __shfl_sync(0xffffffffu, sn, src);
            const double cb = __shfl_sync(0xffffffffu, ex, src), db = __shfl_sync(0xffffffffu, ey, src);
            if (a0 + b >= cnt) continue;
            double pmm = 1.0, fct = 1.0;
            double2 em = make_double2(1.0, 0.0);
#pragma unroll
            for (int k = 1; k <= 8; ++k) {
                if (k <= m) {
                    pmm = -pmm * fct * sb;
                    em = make_double2(em.x * cb - em.y * db, em.x * db + em.y * cb);
                }
                fct += 2.0;
            }
            double p0 = 0.0, p1 = m == 0 ? 1.0 : 0.0, v4 = 0.0, v6 = 0.0, v8 = 0.0;
#pragma unroll
            for (int l = 1; l <= 8; ++l) {
                const double p2 = l == m ? pmm : (double)(2 * l - 1) * xb * p1 - rb[l] * p0;  // (0 while l < m)
                p0 = p1;
                p1 = p2;
                if (l == 4) v4 = n4 * p2;
                if (l == 6) v6 = n6 * p2;
                if (l == 8) v8 = n8 * p2;
            }
            const bool north = fabs(1.0 - xb) < 1e-3, south = fabs(1.0 + xb) < 1e-3;
            if (m == 0 || !north) {
                p4.x += v4 * em.x; p4.y += v4 * em.y;
                p6.x += v6 * em.x; p6.y += v6 * em.y;
                p8.x += v8 * em.x; p8.y += v8 * em.y;
            }
            if (!south) {  // Y_l^-m = (-1)^m conj(Y_l^m)
                s4.x += v4 * em.x; s4.y += v4 * em.y;
                s6.x += v6 * em.x; s6.y += v6 * em.y;
                s8.x += v8 * em.x; s8.y += v8 * em.y;
            }
        }
    }
    if (!mine || cnt == 0) return;
    const double inv = 1.0 / (double)cnt, sg = (m & 1) ? -inv : inv;
    double2* qi = q + (size_t)i * kNQ;
    if (m <= 4) qi[4 + m] = make_double2(p4.x * inv, p4.y * inv);
    if (m <= 6) qi[9 + 6 + m] = make_double2(p6.x * inv, p6.y * inv);
    qi[22 + 8 + m] = make_double2(p8.x * inv, p8.y * inv);
    if (m > 0) {
        if (m <= 4) qi[4 - m] = make_double2(s4.x * sg, -s4.y * sg);
        if (m <= 6) qi[9 + 6 - m] = make_double2(s6.x * sg, -s6.y * sg);
        qi[22 + 8 - m] = make_double2(s8.x * sg, -s8.y * sg);
    }
}

__device__ __forceinline__ double sumsq(const double2* a, int n) {
    double s = 0.0;
    for (int m = 0; m < n; ++m) s += a[m].x * a[m].x + a[m].y * a[m].y;
    return s;
}
constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// sum over the terms k of w3j_k Re(q_m1 q_m2 q_m3), a warp's lanes over the terms
__device__ __forceinline__ double wigner_sum(const double2* q, int l, const double* w3j, const int2* ms, int terms,
                                             int lane) {
    double re = 0.0;
    for (int k = lane; k < terms; k += 32) {
        const int2 m = ms[k];
        const double2 a = q[m.x + l], b = q[m.y + l], c = q[l - m.x - m.y];
        const double2 ab = make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
        re += w3j[k] * (ab.x * c.x - ab.y * c.y);
    }
    return warp_sum(re);
}

// rows: atoms with neighbours, counted per block of kBlk atoms
__global__ void __launch_bounds__(kBlk) k_row_count(const int* __restrict__ np, const int* __restrict__ nbc,
                                                    int* __restrict__ row_cnt) {
    const int i = blockIdx.x * kBlk + threadIdx.x;
    const int c = __syncthreads_count(i < *np && nbc[i] > 0);
    if (threadIdx.x == 0) row_cnt[blockIdx.x] = c;
}

// Per-atom invariants; rows of PFC_BOND_NCOL doubles for atoms with neighbours.  A warp per atom:
// its lanes hold the 39 components of q_lm (so that a neighbour's are read as one block), the
// terms of the Wigner sums, and for xi half a warp each takes every other neighbour.  (A
// thread per atom, 24 k atoms with 14 neighbours: 112 us, every load its own sector; now 79 us, bound
// by the instructions of the sums: reducing all of them together, or the list by 32 entries,
// changed nothing.)
constexpr int kRowWarps = 8;
__global__ void __launch_bounds__(32 * kRowWarps)
    k_bond_rows(const double* __restrict__ pos, const int* __restrict__ np, const int* __restrict__ nbr,
                const int* __restrict__ nb_off, const int* __restrict__ nbc, const int* __restrict__ maxjs,
                const double2* __restrict__ q, const int* __restrict__ row_off, double* __restrict__ rows,
                int row_capacity) {
    __shared__ double w4[kW4], w6[kW6];
    __shared__ int2 m4[kW4], m6[kW6];
    __shared__ double2 own[kRowWarps][kNQ], last[kRowWarps][9];
    __shared__ double sq[kRowWarps][kNQ], sqb[kRowWarps][kNQ], out[kRowWarps][PFC_BOND_NCOL];
    for (int k = threadIdx.x; k < kW6; k += blockDim.x) {
        w6[k] = c_w6[k];
        m6[k] = make_int2(c_w6m[k][0], c_w6m[k][1]);
        if (k < kW4) {
            w4[k] = c_w4[k];
            m4[k] = make_int2(c_w4m[k][0], c_w4m[k][1]);
        }
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int P = *np;
    for (int i = blockIdx.x * kRowWarps + w; i < P; i += gridDim.x * kRowWarps) {
        const int cnt = nbc[i];
        if (cnt == 0) continue;
        // the row: the rows of the blocks before, and of the atoms before in this one
        const int blk = i / kBlk;
        int row = row_off[blk];
        for (int t = blk * kBlk; t < i; t += 32) {
            const int j = t + lane;
            row += __popc(__ballot_sync(0xffffffffu, j < i && nbc[j] > 0));
        }
        if (row >= row_capacity) continue;
        const int* list = nbr + nb_off[i];
        const double2* qi = q + (size_t)i * kNQ;
        const double invn = 1.0 / (1.0 + (double)cnt);
        for (int c = lane; c < kNQ; c += 32) {
            const double2 v = qi[c];
            own[w][c] = v;
            sq[w][c] = v.x * v.x + v.y * v.y;
            double2 s = v;  // q-bar_l, self included (bond-order.cpp:221-250)
            for (int a = 0; a < cnt; ++a) {
                const double2 o = q[(size_t)list[a] * kNQ + c];
                s.x += o.x;
                s.y += o.y;
            }
            s.x *= invn;
            s.y *= invn;
            sqb[w][c] = s.x * s.x + s.y * s.y;
        }
        if (lane < 9) {  // w4b as the reference computes it: the last neighbour's q4m divided by Nb
            const double2 v = q[(size_t)maxjs[i] * kNQ + lane];
            last[w][lane] = make_double2(v.x / (double)cnt, v.y / (double)cnt);
        }
        __syncwarp();
        const double r4 = wigner_sum(own[w], 4, w4, m4, kW4, lane), r6 = wigner_sum(own[w] + 9, 6, w6, m6, kW6, lane),
                     rb = wigner_sum(last[w], 4, w4, m4, kW4, lane);
        // xi: neighbours with normalised q6 . conj(q6) > 0.7 (bond-order.cpp:267-287)
        double n6 = 0.0;
        for (int m = 0; m < 13; ++m) n6 += sq[w][9 + m];
        const double ni = sqrt(n6);
        const int hl = lane & 15, half = lane >> 4;
        const double2 mine = hl < 13 ? own[w][9 + hl] : make_double2(0.0, 0.0);
        int solid = 0;
        for (int a = half; a - half < cnt; a += 2) {
            double d = 0.0, s = 0.0;
            if (a < cnt && hl < 13) {
                const double2 o = q[(size_t)list[a] * kNQ + 9 + hl];
                d = mine.x * o.x + mine.y * o.y;
                s = o.x * o.x + o.y * o.y;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) {
                d += __shfl_xor_sync(0xffffffffu, d, o);
                s += __shfl_xor_sync(0xffffffffu, s, o);
            }
            // d / (sqrt(n6) sqrt(s)) > 0.7, the roots taken only within 1e-12 of it
            const double d2 = d * d, lim = 0.49 * (n6 * s);
            if (a < cnt && d > 0.0 && (d2 > lim * (1.0 + 1e-12) || (!(d2 < lim * (1.0 - 1e-12)) && d / (ni * sqrt(s)) > 0.7)))
                ++solid;
        }
        solid += __shfl_xor_sync(0xffffffffu, solid, 16);
        if (lane < 3) {
            out[w][lane] = pos[3 * i + lane];
            const int o = lane == 0 ? 0 : lane == 1 ? 9 : 22, n = lane == 0 ? 9 : lane == 1 ? 13 : 17;
            double s = 0.0, sb = 0.0;
            for (int m = 0; m < n; ++m) {
                s += sq[w][o + m];
                sb += sqb[w][o + m];
            }
            out[w][5 + lane] = sqrt(4.0 * kPi / (double)n * s);
            out[w][9 + lane] = sqrt(4.0 * kPi / (double)n * sb);
            if (lane == 0) {
                out[w][3] = (double)cnt;
                out[w][4] = (double)solid;
                out[w][8] = r4 / sqrt(s * s * s);
                const double l2 = sumsq(last[w], 9);
                out[w][12] = rb / sqrt(l2 * l2 * l2);
            }
            if (lane == 1) out[w][13] = r6 / sqrt(s * s * s);
        }
        __syncwarp();
        if (lane < PFC_BOND_NCOL) rows[(size_t)row * PFC_BOND_NCOL + lane] = out[w][lane];
        __syncwarp();  // before the next atom's values
    }
}

double fact(int n) { double r = 1.0; for (int k = 2; k <= n; ++k) r *= k; return r; }

// Wigner 3j (l l l; m1 m2 m3) by the Racah formula, evaluated in long double.
double wigner3j_lll(int l, int m1, int m2, int m3) {
    if (m1 + m2 + m3 != 0) return 0.0;
    const int j1 = l, j2 = l, j3 = l;
    auto lf = [](int n) { long double r = 1.0L; for (int k = 2; k <= n; ++k) r *= k; return r; };
    const long double tri = lf(j1 + j2 - j3) * lf(j1 - j2 + j3) * lf(-j1 + j2 + j3) / lf(j1 + j2 + j3 + 1);
    const long double pref = sqrtl(tri * lf(j1 + m1) * lf(j1 - m1) * lf(j2 + m2) * lf(j2 - m2) * lf(j3 + m3) * lf(j3 - m3));
    const int kmin = std::max(0, std::max(j2 - j3 - m1, j1 - j3 + m2));
    const int kmax = std::min(j1 + j2 - j3, std::min(j1 - m1, j2 + m2));
    long double s = 0.0L;
    for (int k = kmin; k <= kmax; ++k) {
        const long double den = lf(k) * lf(j1 + j2 - j3 - k) * lf(j1 - m1 - k) * lf(j2 + m2 - k) *
                                lf(j3 - j2 + m1 + k) * lf(j3 - j1 - m2 + k);
        s += ((k & 1) ? -1.0L : 1.0L) / den;
    }
    const int sg = ((j1 - j2 - m3) % 2 == 0) ? 1 : -1;
    return (double)(sg * pref * s);
}

cudaError_t upload_tables() {
    int ready = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&ready, c_tables_ready, sizeof(int));
    if (e) return e;
    if (ready) return cudaSuccess;
    double nlm[3][9] = {};
    const int ls[3] = {4, 6, 8};
    for (int li = 0; li < 3; ++li)
        for (int m = 0; m <= ls[li]; ++m)
            nlm[li][m] = std::sqrt((2 * ls[li] + 1) / (4.0 * kPi) / (fact(ls[li] - m) * fact(ls[li] + m)));
    std::vector<double> w4, w6;
    std::vector<int> m4, m6;
    for (int a = -4; a <= 4; ++a)
        for (int b = -4; b <= 4; ++b)
            if (std::abs(a + b) <= 4) { w4.push_back(wigner3j_lll(4, a, b, -a - b)); m4.push_back(a); m4.push_back(b); }
    for (int a = -6; a <= 6; ++a)
        for (int b = -6; b <= 6; ++b)
            if (std::abs(a + b) <= 6) { w6.push_back(wigner3j_lll(6, a, b, -a - b)); m6.push_back(a); m6.push_back(b); }
    if ((int)w4.size() != kW4 || (int)w6.size() != kW6) return cudaErrorInvalidValue;
    if ((e = cudaMemcpyToSymbol(c_nlm, nlm, sizeof(nlm)))) return e;
    if ((e = cudaMemcpyToSymbol(c_w4, w4.data(), sizeof(double) * kW4))) return e;
    if ((e = cudaMemcpyToSymbol(c_w4m, m4.data(), sizeof(int) * 2 * kW4))) return e;
    if ((e = cudaMemcpyToSymbol(c_w6, w6.data(), sizeof(double) * kW6))) return e;
    if ((e = cudaMemcpyToSymbol(c_w6m, m6.data(), sizeof(int) * 2 * kW6))) return e;
    ready = 1;
    return cudaMemcpyToSymbol(c_tables_ready, &ready, sizeof(int));
}

}  // namespace

size_t bond_scratch_bytes(int max_atoms) { return scratch_layout(max_atoms, nullptr, nullptr); }

// Grows the context's bond-order scratch to hold `atoms` atoms and `pairs` neighbour
// entries (allocation sizes only grow; nothing is kept across calls, so no copy).
cudaError_t bond_reserve(pfc_ctx* c, int atoms, int64_t pairs) {
    cudaError_t e = cudaSuccess;
    if (atoms > c->max_atoms) {
        const int want = std::max(atoms, c->max_atoms + c->max_atoms / 2);
        void* p = nullptr;
        if ((e = cudaMalloc(&p, bond_scratch_bytes(want)))) return e;
        if (c->bond_scratch) cudaFree(c->bond_scratch);
        c->bond_scratch = p;
        c->max_atoms = want;
        c->bond_scratch_bytes = bond_scratch_bytes(want);
    }
    if (pairs > c->max_pairs) {
        const int64_t want = std::max<int64_t>(pairs, c->max_pairs + c->max_pairs / 2);
        void* p = nullptr;
        if ((e = cudaMalloc(&p, sizeof(int) * (size_t)want))) return e;
        if (c->bond_pairs) cudaFree(c->bond_pairs);
        c->bond_pairs = (int*)p;
        c->max_pairs = want;
    }
    return cudaSuccess;
}

cudaError_t launch_bond_order(pfc_ctx* c, const void* maxima, int n, double h0, double h1, double h2, double ths,
                              double boxsize, double rlim, double* out_rows, int row_capacity, int* n_rows_host) {
    cudaError_t e = cudaSuccess;
    if (!c->bond_tables) {
        if ((e = upload_tables())) return e;
        c->bond_tables = true;
    }
    if ((e = bond_reserve(c, n, 0))) return e;
    BondScratch s;
    scratch_layout(c->max_atoms, &s, (char*)c->bond_scratch);
    cudaStream_t st = c->stream;
    const int nblk = (n + kBlk - 1) / kBlk;
    if ((e = cudaMemsetAsync(s.flags, 0, sizeof(int) * 8, st))) return e;
    // 1. keep field > ths (order preserved)
    if (nblk > 0) {
        if (c->dtype == PFC_F64) k_keep_count<double><<<nblk, kBlk, 0, st>>>((const MaxRecB<double>*)maxima, n, ths, s.keep_cnt);
        else k_keep_count<float><<<nblk, kBlk, 0, st>>>((const MaxRecB<float>*)maxima, n, ths, s.keep_cnt);
        k_scan_b<<<1, 1024, 0, st>>>(s.keep_cnt, nblk, s.keep_off);
        if (c->dtype == PFC_F64)
            k_keep_write<double><<<nblk, kBlk, 0, st>>>((const MaxRecB<double>*)maxima, n, ths, h0, h1, h2, boxsize,
                                                         s.keep_off, s.pos, s.flags);
        else
            k_keep_write<float><<<nblk, kBlk, 0, st>>>((const MaxRecB<float>*)maxima, n, ths, h0, h1, h2, boxsize,
                                                        s.keep_off, s.pos, s.flags);
        if ((e = cudaMemcpyAsync(s.flags + 2, s.keep_off + nblk, sizeof(int), cudaMemcpyDeviceToDevice, st))) return e;
    }
    int hflags[3] = {0, 0, 0};
    if ((e = cudaMemcpyAsync(hflags, s.flags, sizeof(int) * 3, cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaStreamSynchronize(st))) return e;
    const int P = hflags[2];
    const int* np = s.flags + 2;
    if (P == 0) { *n_rows_host = 0; return cudaSuccess; }
    // 2. cells of side >= rlim (all pairs when fewer than 3 per side or atoms outside the box)
    int nc = (int)std::floor(boxsize / rlim);
    if (nc > kMaxCellsDim) nc = kMaxCellsDim;
    if (nc < 3 || hflags[1] || !(rlim > 0.0)) nc = 0;
    const int pb = (P + 255) / 256;
    if (nc > 0) {
        const int cells = nc * nc * nc;
        if ((e = cudaMemsetAsync(s.cell_cnt, 0, sizeof(int) * cells, st))) return e;
        if ((e = cudaMemsetAsync(s.cell_fill, 0, sizeof(int) * cells, st))) return e;
        k_cell_count<<<pb, 256, 0, st>>>(s.pos, np, boxsize, nc, s.cell_cnt);
        k_scan_b<<<1, 1024, 0, st>>>(s.cell_cnt, cells, s.cell_off);
        k_cell_fill<<<pb, 256, 0, st>>>(s.pos, np, boxsize, nc, s.cell_off, s.cell_fill, s.cell_atoms);
    }
    // 3. neighbour lists: count, scan into list offsets, grow the pair buffer, fill
    const int nwb = (P + kNbWarps - 1) / kNbWarps;
    const Within within(rlim);
    k_neighbours<false><<<nwb, 32 * kNbWarps, 0, st>>>(s.pos, np, boxsize, within, nc, s.cell_off, s.cell_atoms,
                                                       nullptr, nullptr, s.nb, s.maxj);
    k_scan_b<<<1, 1024, 0, st>>>(s.nb, P, s.nb_off);
    if ((e = cudaGetLastError())) return e;
    int pairs = 0;
    if ((e = cudaMemcpyAsync(&pairs, s.nb_off + P, sizeof(int), cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaStreamSynchronize(st))) return e;
    if ((e = bond_reserve(c, 0, pairs))) return e;
    k_neighbours<true><<<nwb, 32 * kNbWarps, 0, st>>>(s.pos, np, boxsize, within, nc, s.cell_off, s.cell_atoms,
                                                      s.nb_off, c->bond_pairs, s.nb, nullptr);
    k_qlm<<<(P + 11) / 12, 128, 0, st>>>(s.pos, np, c->bond_pairs, s.nb_off, s.nb, boxsize, s.q);
    const int rb = (P + kBlk - 1) / kBlk;
    k_row_count<<<rb, kBlk, 0, st>>>(np, s.nb, s.row_cnt);
    k_scan_b<<<1, 1024, 0, st>>>(s.row_cnt, rb, s.row_off);
    // (the Wigner tables are copied into shared memory once per CTA: a grid that fills the GPU)
    k_bond_rows<<<std::min((P + kRowWarps - 1) / kRowWarps, 4 * c->num_sms), 32 * kRowWarps, 0, st>>>(
        s.pos, np, c->bond_pairs, s.nb_off, s.nb, s.maxj, s.q, s.row_off, out_rows, row_capacity);
    if ((e = cudaGetLastError())) return e;
    int rows = 0;
    if ((e = cudaMemcpyAsync(&rows, s.row_off + rb, sizeof(int), cudaMemcpyDeviceToHost, st))) return e;
    if ((e = cudaStreamSynchronize(st))) return e;
    *n_rows_host = rows;
    return cudaSuccess;
}

}  // namespace pfc
