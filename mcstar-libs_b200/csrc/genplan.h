// Host side of the general-length passes (genfft.cuh, genpass.cuh): the plans of a context's
// three axes and the launch shapes of its passes.
#pragma once
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>
#include "genpass.cuh"
#include "pfc_ctx.h"

namespace pfc {

// The stages of an n-point plan of the general engine (genfft.cuh), in order.  order 0: the
// fewest stages with radices up to `cap`, as equal as possible (the least sum), larger
// radices first; 1: radices up to 5 (4 before 2), and 7; 2: as 0 with the odd radices first.  7 is
// taken at any cap; primes from 11 to kMaxOddRadix are stages of their own.  At least two stages, the last with a
// hand-written DFT: a stage of radix 1 is appended where needed.  first > 0: only plans without
// primes whose smallest radix is at most that, in ascending order.
inline bool factor_radices(int n, std::vector<int>& rs, int order, int cap, int first) {
    rs.clear();
    if (n < 1) return false;
    std::vector<int> primes;
    for (int p = 11; p <= kMaxOddRadix; p += 2) {
        bool prime = true;
        for (int d = 3; d * d <= p; d += 2) prime = prime && (p % d != 0);
        if (!prime) continue;
        while (n % p == 0) { primes.push_back(p); n /= p; }
    }
    std::vector<int> best;
    if (first > 0 && !primes.empty()) return false;
    if (order == 1) {
        for (int r : {4, 2, 3, 5, 7})
            while (n % r == 0) { best.push_back(r); n /= r; }
        if (n != 1) return false;
    } else {
        static const int kRadix[] = {10, 9, 8, 7, 6, 5, 4, 3, 2};
        std::vector<int> cur;
        int best_len = kMaxStages + 1, best_sum = 0;
        // descending factorisations of n; the number of stages bounded by the best so far
        auto search = [&](auto&& self, int rest, int from) -> void {
            if (rest == 1) {
                if (first > 0 && (cur.empty() || cur.back() > first)) return;
                const int len = (int)cur.size();
                int sum = 0;
                for (int r : cur) sum += r;
                if (len < best_len || (len == best_len && sum < best_sum)) {
                    best = cur;
                    best_len = len;
                    best_sum = sum;
                }
                return;
            }
            if ((int)cur.size() >= best_len) return;
            for (int i = from; i < (int)(sizeof(kRadix) / sizeof(kRadix[0])); ++i)
                if (rest % kRadix[i] == 0 && (kRadix[i] <= cap || kRadix[i] == 7)) {
                    cur.push_back(kRadix[i]);
                    self(self, rest / kRadix[i], i);
                    cur.pop_back();
                }
        };
        search(search, n, 0);
        if (best_len > kMaxStages) return false;
        if (order == 2) std::stable_partition(best.begin(), best.end(), [](int r) { return r % 2 != 0; });
    }
    if (first > 0) {
        std::sort(best.begin(), best.end());
        if (best.empty() || best[0] > first) return false;
    }
    rs = primes;
    rs.insert(rs.end(), best.begin(), best.end());
    if (best.empty() || rs.size() < 2) rs.push_back(1);
    if (rs.size() < 2) rs.push_back(1);
    return (int)rs.size() <= kMaxStages;
}

// Makes an n-point plan: appends its twiddles to tab (forward sign, FP64) and its index
// tables to itab.  A line whose padding would take it above max_np elements goes without.
inline bool make_plan(int n, GPlan& p, std::vector<std::complex<double>>& tab, std::vector<int>& itab, int order,
                      int cap, int max_np, int first = 0) {
    std::vector<int> rs;
    if (!factor_radices(n, rs, order, cap, first)) return false;
    std::memset(&p, 0, sizeof(p));
    p.n = n;
    p.nst = (int)rs.size();
    p.rl = rs.back();
    p.kstep = n / p.rl;
    p.pad = p.rl % 2 == 0 && n + p.kstep <= max_np;
    p.np = n + p.pad * p.kstep;
    p.by_rl = make_fastdiv(p.rl);
    p.by_n = make_fastdiv(n);
    auto padded = [&](int i) { return i + p.pad * (i / p.rl); };
    int M = n;
    for (int s = 0; s < p.nst; ++s) {
        GStage& g = p.st[s];
        g.R = rs[s];
        if (g.R == 7 || g.R > 10) p.odd = 1;
        g.m = M / g.R;
        g.nb = n / g.R;
        p.nbmax = std::max(p.nbmax, g.nb);
        if (g.R > 10) p.nblong = p.nblong ? std::min(p.nblong, g.nb) : g.nb;
        g.ms = s == p.nst - 1 ? 1 : padded(g.m);
        g.Ms = padded(M);
        g.by_m = make_fastdiv(g.m);
        g.by_nb = make_fastdiv(g.nb);
        g.tw = (int)tab.size();
        for (int r = 1; r < g.R; ++r)
            for (int j = 0; j < g.m; ++j) {
                const double ang = -2.0 * M_PI * (double)(((long long)r * j) % M) / (double)M;
                tab.emplace_back(std::cos(ang), std::sin(ang));
            }
        g.rt = (int)tab.size();
        if (g.R > 10)
            for (int q = 0; q < g.R; ++q) {
                const double ang = -2.0 * M_PI * (double)q / (double)g.R;
                tab.emplace_back(std::cos(ang), std::sin(ang));
            }
        M = g.m;
    }
    if (!p.nblong) p.nblong = p.nbmax;
    // frequency of position q: digits of q by the stages, reversed
    std::vector<int> freq(n);
    for (int q = 0; q < n; ++q) {
        int rest = q, k = 0, w = 1;
        for (int s = 0; s < p.nst; ++s) {
            const int d = rest / p.st[s].m;
            rest -= d * p.st[s].m;
            k += d * w;
            w *= p.st[s].R;
        }
        freq[q] = k;
    }
    p.rev = (int)itab.size();
    for (int b = 0; b < p.kstep; ++b) itab.push_back(freq[b * p.rl]);
    p.pos = (int)itab.size();
    itab.resize(itab.size() + n);
    for (int q = 0; q < n; ++q) itab[p.pos + freq[q]] = padded(q);
    return true;
}

// Lines per CTA and threads of the general passes for `batch` fields on `sms` multiprocessors (a
// class of an ensemble shares the GPU with the other classes).
inline void plan_launches(pfc_ctx* c, const pfc_options& o, int batch, int sms) {
    // Columns: 128-byte segments (8 elements of 16 bytes:
    // 16 FP32 or 8 FP64 columns), halved down to the 32-byte sectors of L2 while the tile's
    // shared memory would leave fewer than three CTAs per SM, or the pass fewer than two CTAs
    // per SM; on down to one column while that gives no more than a CTA per SM and an eighth: a
    // pass with so few CTAs takes as long as one of them, whatever it wastes.  y columns and update
    // of FP32 fields, us at 4, 2 and 1 columns: 64 x 2048 (33 columns) 15.8, 11.6, 9.7 and 37.6,
    // 25.4, 20.9; 256 x 1500 (129) 10.3, 8.1, 7.2 and 26.4, 19.6, 16.6; 300 x 300 (151) 4.9, 4.8, 4.8
    // and 11.5, 10.7, 10.0; 1000 x 1000 (501) 8.0, 8.9, 10.8 and 20.1, 21.4, 29.9.  Then tile_shift
    // times.  Threads: one butterfly each in the stage with the most, up to 256 (FP64: 128, for
    // more CTAs per SM); a pass with at most four CTAs per SM takes 256, with at most two the SM's
    // whole register file, and an update pass with few CTAs one mode per thread: the update is its
    // longest part (1000^2 FP32 step, 126 CTAs: 46.3 us at 256 threads, 28.3 at 1000; with noise 59.6
    // and 31.7; two-column tiles at 256 threads 33.4 and 34.0).
    // Rows: as many as fill those threads, by the butterflies of the largest prime radix where there is
    // one (a 209-point row in FP64 has 11 of radix 19, and by the stage with the most, the appended one of
    // radix 1, one row per CTA: 209x57x260 x pass 679 us, now 133).  With at most four CTAs per SM
    // k_rows takes at least a thread for two points, for its loops over the row's modes (1024 x 240 FP32, two
    // rows: C2R rows 10.6 us at 64 threads, 9.0 at 256; 128 x 45 x 30, eight rows: R2C 5.1 at 64,
    // 4.4 at 256).
    const int W = c->dtype == PFC_F64 ? 1 : 2;  // lines of an element
    const int many = c->dtype == PFC_F64 ? 128 : 256;
    auto columns = [&](AxisPlan& ap, int64_t planes, int fields, bool update, int shift) {
        const size_t line = (size_t)ap.plan.np * 16 * fields;
        int cols = 8 * W;  // columns of a CTA
        auto shape = [&](int n) {
            cols = n;
            ap.w = std::min(W, n);
            ap.lg = 0;
            while ((ap.w << ap.lg) < n) ++ap.lg;
        };
        auto ctas = [&] { return (c->nxh + cols - 1) / cols * planes * batch; };
        auto bytes = [&] { return line * (size_t)std::max(1, cols / W); };
        while (cols > 2 && cols / 2 >= c->nxh) cols /= 2;
        while (cols > 2 * W && (bytes() > 72 * 1024 || ctas() < 2 * (int64_t)sms)) cols /= 2;
        while (cols > 1 && (c->nxh + cols / 2 - 1) / (cols / 2) * planes * batch <= sms + sms / 8) cols /= 2;
        while (cols > W && bytes() > kMaxDynSmem) cols /= 2;
        shape(std::max(1, cols >> shift));
        const int64_t per_sm = (ctas() + sms - 1) / sms;
        const bool few = per_sm <= 4;
        const int work = ((few && update ? ap.plan.n : ap.plan.nbmax * fields) << ap.lg) + 31;
        const int full = c->dtype == PFC_F64 ? kColThreads<double> : kColThreads<float>;
        const int most = !few ? many : per_sm <= 2 ? (int)(full / per_sm) & ~31 : kGenThreads;
        ap.threads = std::min(most, std::max(32, work & ~31));
        ap.smem = ((size_t)ap.plan.np * 16) << ap.lg;
    };
    columns(c->py, c->nz, 1, false, o.tile_shift[1]);
    columns(c->pz, c->ny, 1, false, o.tile_shift[2]);
    columns(c->pzprop, c->ny, 1, true, o.tile_shift[3]);
    columns(c->pz2, c->ny, 2, true, o.tile_shift[3]);
    columns(c->py2, 1, 1, true, o.tile_shift[3]);
    // work: the most items of a line in a stage; longest: in the stage that takes longest; merge: a pass
    // with loops over the row's modes
    auto rows = [&](AxisPlan& ap, int work, int longest, bool merge) {
        const int64_t nrows = (int64_t)c->ny * c->nz;
        int rpc = std::max(1, many / longest) * W;  // rows of a CTA
        auto bytes = [&] { return (size_t)(rpc / W) * ap.plan.np * 16; };
        while (rpc > W && bytes() > 72 * 1024) rpc = rpc / (2 * W) * W;
        while (rpc > W && (nrows + rpc - 1) / rpc * batch < 2 * (int64_t)sms) rpc = rpc / (2 * W) * W;
        for (int i = 0; i < o.tile_shift[0] && rpc > 1; ++i) rpc = rpc > W ? rpc / (2 * W) * W : 1;
        ap.w = std::min(W, rpc);
        ap.lines = rpc / ap.w;
        int items = ap.lines * work;
        if (merge && (nrows + rpc - 1) / rpc * batch <= 4 * (int64_t)sms) items = std::max(items, ap.lines * ap.plan.n / 2);
        ap.threads = std::min(kGenThreads, std::max(32, (items + 31) & ~31));
        ap.smem = (size_t)ap.lines * ap.plan.np * 16;
    };
    rows(c->px, c->px.plan.nbmax, c->px.plan.nblong, true);
    if (c->px2.plan.nst) {
        const GPlan& q = c->px2.plan;
        int work = q.st[0].m / 2 + 1;
        for (int i = 1; i < q.nst; ++i) work = std::max(work, q.st[i].nb);
        rows(c->px2, work, work, false);
    }
}

// The lengths a context accepts: per axis two lines (z: four) padded by one element in 32 within
// a CTA's shared memory, and prime factors up to kMaxOddRadix.  The passes hold one line (z carrying
// A: two) of np elements of 16 bytes and fit every such length, the longest ones unpadded.
inline bool length_accepted(int n, int lines, size_t csz) {
    return (size_t)lines * ((n + (n >> 5) + 1) | 1) * csz <= kMaxDynSmem;
}

// The plans of c's axes (shape and precision set); false: a length is not supported.
inline bool plan_general(pfc_ctx* c, const pfc_options& o, std::vector<std::complex<double>>& gtab,
                         std::vector<int>& itab) {
    const bool even = (c->nx % 2) == 0;
    const int lx = even ? c->nx / 2 : c->nx;
    const size_t csz = 2 * c->fsize;
    if (!length_accepted(lx, 2, csz) || !length_accepted(c->ny, 2, csz) || !length_accepted(c->nz, 4, csz)) return false;
    // Radices of the general passes by field size.  Small fields leave most of the GPU idle and
    // pay for every instruction fetched, so small radices (more threads, less code) win: 256^2
    // FP64 x pass 5.7 us at radices up to 6, 7.0 at 8 and 10; 600 x 500 FP32 8.0 at 8, 10.0 at
    // 10; from about a million modes fewer stages win (160 x 150 x 160 FP32 x pass 14.7 at 10,
    // 17.4 at 8).
    const int cap = c->n_cmpl < 100000 ? 6 : c->n_cmpl < 1000000 ? 8 : 10;
    const int one = (int)(kMaxDynSmem / 16), two = one / 2;
    if (!make_plan(lx, c->px.plan, gtab, itab, o.radix_order, cap, one) ||
        !make_plan(c->ny, c->py.plan, gtab, itab, o.radix_order, cap, one) ||
        !make_plan(c->nz, c->pz.plan, gtab, itab, o.radix_order, cap, one))
        return false;
    // the paired x pass, where it takes no stage more than the general one (160 x 150 x 160 FP32:
    // 10 x 8 unpaired 69.5 us per step, 5 x 4 x 4 paired 72)
    if (!even || !make_plan(lx, c->px2.plan, gtab, itab, o.radix_order, cap, one, kPairRadix) ||
        c->px2.plan.nst > c->px.plan.nst)
        c->px2.plan = GPlan{};
    c->pzprop.plan = c->pz2.plan = c->pz.plan;
    if (c->pz.plan.np > two && !make_plan(c->nz, c->pz2.plan, gtab, itab, o.radix_order, cap, two)) return false;
    c->py2.plan = c->py.plan;
    c->post_off = (int)gtab.size();
    for (int k = 0; k <= c->nx / 2; ++k) {
        const double ang = -2.0 * M_PI * (double)k / (double)c->nx;
        gtab.emplace_back(std::cos(ang), std::sin(ang));
    }
    return true;
}

}  // namespace pfc
