// Host build of the drift medium's point update on tables turned into the frame
// of a plane's two axes (csrc/fold3d_tables.cpp: orient_table), which every
// dataflow pass uses, swept over a field plane by plane as the passes walk it.
// Test code only.
#include <cmath>
#include <cstdint>

#include "fold3d_fast.cuh"
#include "fold3d_internal.h"

using namespace fold3d;

namespace {

struct HostDir {
    int nrm, sg, xa, xs, ya, ys;
};
const HostDir kHostDirs[6] = {
    {0, +1, 2, +1, 1, +1}, {0, -1, 2, -1, 1, -1}, {2, +1, 1, +1, 0, +1},
    {2, -1, 1, -1, 0, -1}, {1, -1, 0, -1, 2, -1}, {1, +1, 0, +1, 2, +1},
};

}  // namespace

// `sweeps` sweeps on T.  plain: the tables in the local frame and the sources in
// its order; otherwise both in the order of the plane's axes u and v.
extern "C" void orient_sweeps(double *T, int nx, int ny, int nz, double dx, double dy, double dz, double F, double a0,
                              double a1, double a2, int sweeps, int plain)
{
    const int n[3] = {nx, ny, nz};
    const int64_t stride[3] = {1, (int64_t)nx + 2, ((int64_t)nx + 2) * (ny + 2)};
    const double h[3] = {dx, dy, dz}, a[3] = {a0, a1, a2};
    static const int I[8] = {1, 1, 0, -1, -1, -1, 0, 1}, J[8] = {0, 1, 1, 1, 0, -1, -1, -1};
    DirTable tabs[6];
    for (int dir = 0; dir < 6; ++dir) {
        const HostDir &d = kHostDirs[dir];
        LocalFrameH L;
        L.F = F;
        L.ax = d.xs * a[d.xa];
        L.ay = d.ys * a[d.ya];
        L.az = d.sg * a[d.nrm];
        L.hz = h[d.nrm];
        L.hx = h[d.xa];
        L.hy = h[d.ya];
        L.hxy = std::sqrt(L.hx * L.hx + L.hy * L.hy);
        L.hxz = std::sqrt(L.hx * L.hx + L.hz * L.hz);
        L.hyz = std::sqrt(L.hy * L.hy + L.hz * L.hz);
        build_dir_table(L, tabs[dir], true);
        if (!plain) orient_table(tabs[dir], d.xa == ((d.nrm == 0) ? 1 : 0), d.xs, d.ys);
    }
    for (int s = 0; s < sweeps; ++s)
        for (int dir = 0; dir < 6; ++dir) {
            const HostDir &d = kHostDirs[dir];
            const int u = (d.nrm == 0) ? 1 : 0, v = (d.nrm == 2) ? 1 : 2;
            const int64_t sx = plain ? d.xs * stride[d.xa] : stride[u], sy = plain ? d.ys * stride[d.ya] : stride[v];
            for (int q = 0; q < n[d.nrm] - 1; ++q) {
                const int src = d.sg > 0 ? 1 + q : n[d.nrm] - q;
                for (int b = 1; b <= n[v]; ++b)
                    for (int c = 1; c <= n[u]; ++c) {
                        const int64_t si = src * stride[d.nrm] + c * stride[u] + b * stride[v];
                        double fan[9], sh[9];
                        float ch[9];
                        for (int r = 0; r < 8; ++r) fan[r] = std::fabs(T[si + I[r] * sx + J[r] * sy]);
                        fan[8] = std::fabs(T[si]);
                        double &t = T[si + d.sg * stride[d.nrm]];
                        t = point_update_fan(true, t, fan, tabs[dir], sh, ch, 1);
                    }
            }
        }
}
