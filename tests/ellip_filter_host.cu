// Host build of the elliptical medium's FP64 update with its float filter
// (csrc/fold3d_ellip.cuh: ell_update_fan), swept over a field like the point
// update in ellip_solver_host.cu.  Test code only.
#include <cmath>
#include <cstdint>
#include <cstring>

#include "fold3d_ellip.cuh"

using namespace fold3d;

namespace {

struct HostDir {
    int nrm, sg, xa, xs, ya, ys;
};
const HostDir kHostDirs[6] = {
    {0, +1, 2, +1, 1, +1}, {0, -1, 2, -1, 1, -1}, {2, +1, 1, +1, 0, +1},
    {2, -1, 1, -1, 0, -1}, {1, -1, 0, -1, 2, -1}, {1, +1, 0, +1, 2, +1},
};
constexpr int kCands = 33;

// The direction's metric gather and signs, as the library forms them.
EllipDir host_dir(int dir, const double h[3])
{
    static const int pair[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
    const HostDir &d = kHostDirs[dir];
    EllipDir e;
    e.hx = h[d.xa];
    e.hy = h[d.ya];
    e.hz = h[d.nrm];
    e.sxy = d.xs * d.ys;
    e.sxz = d.xs * d.sg;
    e.syz = d.ys * d.sg;
    e.ixx = pair[d.xa][d.xa];
    e.iyy = pair[d.ya][d.ya];
    e.izz = pair[d.nrm][d.nrm];
    e.ixy = pair[d.xa][d.ya];
    e.ixz = pair[d.xa][d.nrm];
    e.iyz = pair[d.ya][d.nrm];
    return e;
}

}  // namespace

// `count` sweeps on T with its winner record W.  param: M holds the four
// parameter arrays (double), else the six float metric arrays.
extern "C" int ellip_filter_sweeps(double *T, unsigned char *W, const void *const *M, int param, int nx, int ny, int nz,
                                   double dx, double dy, double dz, int count)
{
    const double h[3] = {dx, dy, dz};
    const int n[3] = {nx, ny, nz};
    const int64_t stride[3] = {1, (int64_t)nx + 2, ((int64_t)nx + 2) * (ny + 2)};
    EllipMedium med;
    for (int k = 0; k < 6; ++k) med.m[k] = (param && k > 3) ? nullptr : M[k];
    med.kind = param ? kParamF64 : kMetricF32;
    for (int s = 0; s < count; ++s)
        for (int dir = 0; dir < 6; ++dir) {
            const HostDir &d = kHostDirs[dir];
            const EllipDir D = host_dir(dir, h);
            const int u = (d.nrm == 0) ? 1 : 0, v = (d.nrm == 2) ? 1 : 2;
            const int64_t sx = d.xs * stride[d.xa], sy = d.ys * stride[d.ya], sn = stride[d.nrm];
            const int nn = n[d.nrm];
            for (int q = 0; q < nn - 1; ++q) {
                const int src = d.sg > 0 ? 1 + q : nn - q;
                for (int b = 1; b <= n[v]; ++b)
                    for (int c = 1; c <= n[u]; ++c) {
                        const int64_t si = (int64_t)src * sn + c * stride[u] + b * stride[v];
                        const int64_t ti = si + d.sg * sn;
                        const double *p = T + si;
                        double fan[9], val[6], sh[9];
                        for (int r = 0; r < 8; ++r) fan[r] = std::fabs(p[ell_ri(r) * sx + ell_rj(r) * sy]);
                        fan[8] = std::fabs(p[0]);
                        ell_values(med, D, ti, val);
                        int win;
                        const double told = T[ti];
                        const double tnew = ell_update_fan(true, told, fan, val, med.kind, D, sh, 1, win);
                        if (std::memcmp(&tnew, &told, sizeof tnew) != 0) {
                            W[ti] = (win < 0) ? 0xffu : (unsigned char)(dir * kCands + win);
                            T[ti] = tnew;
                        }
                    }
            }
        }
    return 0;
}
