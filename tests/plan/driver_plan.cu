// Host check of csrc/genplan.h: prints every length whose plans a context refuses although the
// rule accepts it, or whose launches do not fit a CTA's shared memory, and the number of lengths seen.
#include <cstdio>
#include <mutex>
#include <thread>
#include "../../mcstar-libs_b200/csrc/genplan.h"

namespace {

std::mutex mu;
long long seen = 0;

bool smooth(int n) {
    for (int p = 2; p <= 31; ++p)
        while (n % p == 0) n /= p;
    return n == 1;
}
// the rule of creation: `lines` lines of n complex values, one of padding in 32, in 200 KB
bool rule(int n, int lines, int bytes) { return (long long)lines * ((n + n / 32 + 1) | 1) * bytes <= 204800; }

void check(int nx, int ny, int nz, int dtype, int order) {
    const int bytes = dtype == PFC_F64 ? 16 : 8, lx = nx % 2 ? nx : nx / 2;
    const bool want = smooth(lx) && smooth(ny) && smooth(nz) && rule(lx, 2, bytes) && rule(ny, 2, bytes) && rule(nz, 4, bytes);
    pfc_ctx c;
    c.nx = nx; c.ny = ny; c.nz = nz; c.nxh = nx / 2 + 1;
    c.dtype = dtype;
    c.fsize = bytes / 2;
    c.n_real = (size_t)nx * ny * nz;
    c.n_cmpl = (size_t)c.nxh * ny * nz;
    pfc_options o{-1, -1, -1, order, {0, 0, 0, 0}, -1};
    std::vector<std::complex<double>> tw;
    std::vector<int> tab;
    const bool got = pfc::plan_general(&c, o, tw, tab);
    size_t worst = 0;
    int threads = 32;
    if (got) {
        pfc::plan_launches(&c, o, 1, 148);
        const pfc::AxisPlan* all[] = {&c.px, &c.px2, &c.py, &c.pz, &c.pzprop, &c.pz2, &c.py2};
        for (const pfc::AxisPlan* p : all)
            if (p->plan.nst) {
                worst = std::max(worst, p->smem * (p == &c.pz2 ? 2 : 1));
                if (p->threads < 32 || p->threads > 1024 || p->threads % 32) threads = p->threads;
            }
    }
    std::lock_guard<std::mutex> lock(mu);
    ++seen;
    if (got != want || worst > pfc::kMaxDynSmem || threads != 32)
        std::printf("bad %dx%dx%d dtype %d order %d: accepted %d (rule %d), shared memory %zu, threads %d\n", nx, ny, nz,
                    dtype, order, (int)got, (int)want, worst, threads);
}

}  // namespace

int main() {
    const int workers = 8;
    std::vector<std::thread> pool;
    for (int w = 0; w < workers; ++w)
        pool.emplace_back([w] {
            for (int n = 4000 + w; n <= 12600; n += workers) {
                if (!smooth(n)) continue;
                for (int order = 0; order < 3; ++order) {
                    check(16, n, 1, PFC_F32, order);
                    check(2 * n, 3, 1, PFC_F32, order);
                    if (n < 6600) {
                        check(6, 4, n, PFC_F32, order);
                        check(16, n, 1, PFC_F64, order);
                    }
                }
                check(5, n, 1, PFC_F32, 0);     // (the radices depend on the field's size)
                check(300, n, 1, PFC_F32, 0);
                check(2 * n, 300, 1, PFC_F32, 0);
                if (n % 2) check(n, 8, 1, PFC_F32, 0);
                if (n < 6600) check(64, 20, n, PFC_F32, 0);
            }
            for (int n = 1 + w; n <= 4000; n += workers)
                if (n < 300 || n % 7 == 0) {
                    check(n, 10, 1, PFC_F32, n % 3);
                    check(10, n, 3, PFC_F64, n % 3);
                    check(8, 5, n, n % 2 ? PFC_F32 : PFC_F64, n % 3);
                }
        });
    for (auto& t : pool) t.join();
    std::printf("seen %lld\n", seen);
    return 0;
}
