// Host check of csrc/genplan.h: prints every field whose column passes would leave multiprocessors
// idle although its columns could be spread further.
#include <cstdio>
#include "../../mcstar-libs_b200/csrc/genplan.h"

int main() {
    const int sides[] = {2, 30, 64, 75, 96, 100, 128, 150, 200, 256, 300, 384, 512, 640, 1000, 1024, 1500, 2048, 2700, 3072, 4000};
    const int sms = 148;
    long long seen = 0;
    for (int dtype : {PFC_F32, PFC_F64})
        for (int nx : sides)
            for (int ny : sides)
                for (int nz : {1, 4, 30}) {
                    if ((long long)nx * ny * nz > 20000000) continue;
                    pfc_ctx c;
                    c.nx = nx; c.ny = ny; c.nz = nz; c.nxh = nx / 2 + 1;
                    c.dtype = dtype;
                    c.fsize = dtype == PFC_F64 ? 8 : 4;
                    c.n_real = (size_t)nx * ny * nz;
                    c.n_cmpl = (size_t)c.nxh * ny * nz;
                    pfc_options o{-1, -1, -1, 0, {0, 0, 0, 0}, -1};
                    std::vector<std::complex<double>> tw;
                    std::vector<int> tab;
                    if (!pfc::plan_general(&c, o, tw, tab)) continue;
                    pfc::plan_launches(&c, o, 1, sms);
                    auto check = [&](const char* name, const pfc::AxisPlan& p, long long planes) {
                        const int cols = p.w << p.lg;
                        const long long ctas = (c.nxh + cols - 1) / cols * planes, most = c.nxh * planes;
                        ++seen;
                        if (ctas < std::min<long long>(most, sms / 2))
                            std::printf("bad %s of %dx%dx%d dtype %d: %lld CTAs of %d columns\n", name, nx, ny, nz, dtype, ctas, cols);
                    };
                    check("y columns", c.py, nz);
                    if (nz == 1) check("2D update", c.py2, 1);
                    else check("z update", c.pzprop, ny);
                }
    std::printf("seen %lld\n", seen);
    return 0;
}
