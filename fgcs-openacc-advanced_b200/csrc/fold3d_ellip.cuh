// fold3d_ellip.cuh -- local solver for a per-cell elliptical (tilted
// transversely isotropic) medium.  No counterpart in the reference, whose
// solver only knows the drift medium.
//
// The medium is a per-cell symmetric positive definite metric M: the travel
// time along a short straight segment d is sqrt(d^T M d).  For a tilted
// elliptical medium with vertical speed Vz, Thomsen epsilon and symmetry
// axis n, M = a I + b n n^T with a = 1/(Vz^2 (1 + 2 eps)), b = 1/Vz^2 - a.
//
// In a sweep direction's local frame (x, y in the source plane, z towards
// the target) the target X is at (0, 0, hz) above the source point st and
// the eight neighbours are at (i hx, j hy, 0).  With the time linear on each
// vertex, edge and triangle of that 3 x 3 fan, the new time is the minimum
// of t(p) + ||X - p||_M over the fan, made of: the 9 vertex values, the
// interior stationary points of the 16 edges (8 spokes st-P, 8 rim edges
// between adjacent neighbours) and of the 8 triangles (st, P, next P), all in
// closed form.  Every candidate exceeds the smallest time it is built from,
// and each is only computed while the running time is above that smallest
// time, so, like the drift solver, the update is min(T_old, candidates): the
// WAVEFRONT engine's tile skipping holds unchanged.
//
// Each candidate is t(p) + ||X - p||_M at a point p of its vertex, edge or
// triangle (the closed forms are the exact stationary values), and t(p) is
// at least the smallest time it is built from.  ||X - p||_M is at least
// B = min over the whole source plane of ||X - p||_M, which in the scaled
// local frame (X = (0, 0, 1)) is the square root of the Schur complement
// Azz - [Axz Ayz] [[Axx Axy] [Axy Ayy]]^-1 [Axz Ayz]^T.  So a candidate is
// only computed while the running time is above its smallest input plus
// B (1 - 1e-3): a candidate skipped that way could not have lowered it.  The
// margin 1e-3 is far above the rounding of the closed forms near that bound
// (their square roots are well conditioned there), in float as in double;
// with B = 0 (a rounded Schur complement <= 0) the gates are the plain ones.
//
// Those gates serve float fields; double fields are updated behind a float
// filter instead (ell_update_fan, below).
//
// oracle/fold3d_oracle.c (orc_ell_*) states the same computation on the
// CPU; this file follows it operation by operation (no FMA contraction), so
// the two agree bit for bit.
#pragma once

namespace fold3d {

// Constants of one sweep direction for the elliptical solver.
struct EllipDir {
    double hx, hy, hz;  // spacings along local x, y and the normal
    int sxy, sxz, syz;  // signs of the local off-diagonal metric entries
    int ixx, iyy, izz, ixy, ixz, iyz;  // which global metric array feeds each local entry
};

// How the per-cell medium is stored (field layout, axes i, j, k):
//  kMetricF32: six float32 arrays of the metric, ordered xx xy xz yy yz zz;
//  kParamF64:  four float64 arrays of the tilted elliptical medium's
//              parameters -- slowness s = 1/Vz, Thomsen epsilon, and the x
//              and y components of the unit symmetry axis n (its z
//              component sqrt(1 - nx^2 - ny^2) >= 0; n and -n are the same
//              axis) -- from which the metric is formed per cell in FP64
//              (ell_metric_from_param).
enum { kMetricF32 = 0, kParamF64 = 1 };
struct EllipMedium {
    const void *m[6];
    int kind;
};

struct EllipParam {
    EllipDir dir;
    EllipMedium med;
};

#ifdef __CUDACC__
// The solver is written once for the field's type R: double (the default
// build) or float (the float32 build).  All arithmetic stays in R (literals
// included), so the float build is float arithmetic throughout.  It also
// compiles for the host, where a test runs it against the CPU statement.

// Local metric scaled by the spacings (Axx = M'xx hx hx, Axy = M'xy hx hy, ...).
template <class R> struct EllipAT {
    R xx, yy, zz, xy, xz, yz;
};
using EllipA = EllipAT<double>;

template <class R> __host__ __device__ __forceinline__ R ell_sqrt(R x);
template <> __host__ __device__ __forceinline__ double ell_sqrt<double>(double x) { return sqrt(x); }
template <> __host__ __device__ __forceinline__ float ell_sqrt<float>(float x) { return sqrtf(x); }

// A read-only metric word (through the read-only data cache on the device).
__host__ __device__ __forceinline__ float ell_ld(const float *p)
{
#ifdef __CUDA_ARCH__
    return __ldg(p);
#else
    return *p;
#endif
}

// u^T M' v with u = (ui hx, uj hy, uk hz) and v likewise.
template <class R>
__host__ __device__ __forceinline__ R ell_bf(const EllipAT<R> &A, int ui, int uj, int uk, int vi, int vj, int vk)
{
    return (R)(ui * vi) * A.xx + (R)(uj * vj) * A.yy + (R)(uk * vk) * A.zz + (R)(ui * vj + uj * vi) * A.xy +
           (R)(ui * vk + uk * vi) * A.xz + (R)(uj * vk + uk * vj) * A.yz;
}

template <class R> __host__ __device__ __forceinline__ R ell_min(R a, R b) { return (a < b) ? a : b; }

// B (1 - 1e-3), B the smallest ||X - p||_M over the source plane (header
// comment), or 0 when the rounded Schur complement is not positive.
template <class R> __host__ __device__ __forceinline__ R ell_skip_bound(const EllipAT<R> &A)
{
    const R cof = A.xx * A.yy - A.xy * A.xy;
    if (!(cof > R(0))) return R(0);
    const R sch = A.zz - (A.xz * (A.xz * A.yy - A.yz * A.xy) + A.yz * (A.yz * A.xx - A.xz * A.xy)) / cof;
    return (sch > R(0)) ? ell_sqrt(sch) * R(0.999) : R(0);
}

// Candidate ids (the adjoint's winner record): 0 vertex st, 1+r rim vertex r,
// 9+r spoke st-rim[r], 17+r rim edge rim[r]-rim[r+1], 25+r triangle
// (st, rim[r], rim[r+1]).  Each routine sets win when it lowers tn, and runs
// only while tn is above its smallest input time plus gate (ell_skip_bound).
template <class R>
__host__ __device__ __forceinline__ void ell_vertex(R &tn, int &win, int id, const EllipAT<R> &A, R gate, R tp, int i,
                                                    int j)
{
    if (!(tn > tp + gate)) return;
    const R c = ell_bf(A, -i, -j, 1, -i, -j, 1);
    if (c > R(0)) {
        const R cand = tp + ell_sqrt(c);
        if (cand < tn) {
            tn = cand;
            win = id;
        }
    }
}

template <bool kOwnBound, class R>
__host__ __device__ __forceinline__ void ell_edge(R &tn, int &win, int id, const EllipAT<R> &A, R gate, R tp, R tq,
                                                  int pi, int pj, int qi, int qj)
{
    const R mn = ell_min(tp, tq);
    if (!(tn > mn + gate)) return;
    const int ei = qi - pi, ej = qj - pj;
    const R a = ell_bf(A, ei, ej, 0, ei, ej, 0);
    const R b = ell_bf(A, ei, ej, 0, -pi, -pj, 1);
    const R c = ell_bf(A, -pi, -pj, 1, -pi, -pj, 1);
    // kOwnBound (the rim edges, away from the foot of X): the edge's own
    // distance bound.  The candidate is at least mn plus the smallest
    // ||X - p|| over the segment, whose square is c (b <= 0), c - 2b + a
    // (b >= a) or (ac - b^2)/a; skip while tn - mn is at most 0.999 of it,
    // compared in squares (ac - b^2 = ac sin^2 of the angle between the edge
    // and X - P, far from 0 for an edge of the source plane).
    if (kOwnBound && a > R(0)) {
        const R e2 = (tn - mn) * (tn - mn);
        const bool skip = !(b > R(0))  ? e2 <= R(0.998) * c
                          : !(b < a)   ? e2 <= R(0.998) * (c - R(2) * b + a)
                                       : e2 * a <= R(0.998) * (a * c - b * b);
        if (skip) return;
    }
    const R d = tq - tp;
    const R den = a - d * d;
    const R disc = a * c - b * b;
    if (den > R(0) && disc > R(0)) {
        const R n = ell_sqrt(disc / den);
        const R lam = (b - d * n) / a;
        if (lam > R(0) && lam < R(1)) {
            const R cand = tp + lam * d + n;
            if (cand < tn) {
                tn = cand;
                win = id;
            }
        }
    }
}

template <class R>
__host__ __device__ __forceinline__ void ell_tri(R &tn, int &win, int id, const EllipAT<R> &A, R gate, R t0, R ta,
                                                 R tb, int ai, int aj, int bi, int bj)
{
    if (!(tn > ell_min(t0, ell_min(ta, tb)) + gate)) return;
    const R p11 = ell_bf(A, ai, aj, 0, ai, aj, 0);
    const R p12 = ell_bf(A, ai, aj, 0, bi, bj, 0);
    const R p22 = ell_bf(A, bi, bj, 0, bi, bj, 0);
    const R q1 = ell_bf(A, ai, aj, 0, 0, 0, 1);
    const R q2 = ell_bf(A, bi, bj, 0, 0, 0, 1);
    const R c = A.zz;
    const R d1 = ta - t0, d2 = tb - t0;
    const R det = p11 * p22 - p12 * p12;
    if (!(det > R(0))) return;
    const R u1 = p22 * d1 - p12 * d2, u2 = p11 * d2 - p12 * d1;
    const R w1 = p22 * q1 - p12 * q2, w2 = p11 * q2 - p12 * q1;
    const R s = (d1 * u1 + d2 * u2) / det;
    const R r = c - (q1 * w1 + q2 * w2) / det;
    if (s < R(1) && r > R(0)) {
        const R n = ell_sqrt(r / (R(1) - s));
        const R l1 = (w1 - n * u1) / det, l2 = (w2 - n * u2) / det;
        if (l1 > R(0) && l2 > R(0) && l1 + l2 < R(1)) {
            const R cand = t0 + (l1 * d1 + l2 * d2) + n;
            if (cand < tn) {
                tn = cand;
                win = id;
            }
        }
    }
}

// Rim of the fan in order: (1,0) xt, (1,1) txy, (0,1) yt, (-1,1) tym,
// (-1,0) xnt, (-1,-1) txnyn, (0,-1) ynt, (1,-1) txm.
__host__ __device__ __forceinline__ int ell_ri(int r)
{
    return (r == 0 || r == 1 || r == 7) ? 1 : (r >= 3 && r <= 5) ? -1 : 0;
}
__host__ __device__ __forceinline__ int ell_rj(int r) { return (r >= 1 && r <= 3) ? 1 : (r >= 5) ? -1 : 0; }

__host__ __device__ __forceinline__ double ell_ld(const double *p)
{
#ifdef __CUDA_ARCH__
    return __ldg(p);
#else
    return *p;
#endif
}

// The metric M = a I + b n n^T of the tilted elliptical medium from its
// parameters: a = s^2 / (1 + 2 eps), b = s^2 - a, n = (nx, ny, nz) with
// nz = sqrt(max(0, (1 - nx nx) - ny ny)).  Entries xx xy xz yy yz zz, in this
// operation order on every side (the oracle's orc_tti_metric states the
// same), so host and device agree bit for bit.
__host__ __device__ __forceinline__ void ell_metric_from_param(double s, double eps, double nx, double ny,
                                                               double out[6])
{
    const double s2 = s * s;
    const double a = s2 / (1.0 + 2.0 * eps);
    const double b = s2 - a;
    const double q = (1.0 - nx * nx) - ny * ny;
    const double nz = sqrt(q > 0.0 ? q : 0.0);
    const double bx = b * nx, by = b * ny, bz = b * nz;
    out[0] = a + bx * nx;
    out[1] = bx * ny;
    out[2] = bx * nz;
    out[3] = a + by * ny;
    out[4] = by * nz;
    out[5] = a + bz * nz;
}

// Metric entry k (xx xy xz yy yz zz) of cell t, stored as float32.
__host__ __device__ __forceinline__ double ell_entry(const EllipMedium &M, int k, long long t)
{
    return (double)ell_ld(static_cast<const float *>(M.m[k]) + t);
}

// Scaled local metric of the target at field index t.
template <class R>
__host__ __device__ __forceinline__ EllipAT<R> ell_local(const EllipMedium &M, const EllipDir &D, long long t)
{
    const R hx = (R)D.hx, hy = (R)D.hy, hz = (R)D.hz;
    EllipAT<R> A;
    if (M.kind == kParamF64) {
        double m[6];
        ell_metric_from_param(ell_ld(static_cast<const double *>(M.m[0]) + t),
                              ell_ld(static_cast<const double *>(M.m[1]) + t),
                              ell_ld(static_cast<const double *>(M.m[2]) + t),
                              ell_ld(static_cast<const double *>(M.m[3]) + t), m);
        A.xx = (R)m[D.ixx] * hx * hx;
        A.yy = (R)m[D.iyy] * hy * hy;
        A.zz = (R)m[D.izz] * hz * hz;
        A.xy = (R)D.sxy * (R)m[D.ixy] * hx * hy;
        A.xz = (R)D.sxz * (R)m[D.ixz] * hx * hz;
        A.yz = (R)D.syz * (R)m[D.iyz] * hy * hz;
        return A;
    }
    const float *const *f = reinterpret_cast<const float *const *>(M.m);
    A.xx = (R)ell_ld(f[D.ixx] + t) * hx * hx;
    A.yy = (R)ell_ld(f[D.iyy] + t) * hy * hy;
    A.zz = (R)ell_ld(f[D.izz] + t) * hz * hz;
    A.xy = (R)D.sxy * (R)ell_ld(f[D.ixy] + t) * hx * hy;
    A.xz = (R)D.sxz * (R)ell_ld(f[D.ixz] + t) * hx * hz;
    A.yz = (R)D.syz * (R)ell_ld(f[D.iyz] + t) * hy * hz;
    return A;
}

// New signed value of a target from st and its rim values (rim order above);
// win: id of the candidate that set it, -1 if none did.
template <class R>
__host__ __device__ __forceinline__ R point_update_ellip(R told, R st, const R nb[8], const EllipAT<R> &A, int &win)
{
    R tn = fabs(told);
    win = -1;
    const R gate = ell_skip_bound(A);
    ell_vertex(tn, win, 0, A, gate, st, 0, 0);
    R m = st;
#pragma unroll
    for (int r = 0; r < 8; ++r) m = ell_min(m, nb[r]);
    if (tn > m + gate) {  // otherwise every routine below would return at its gate
#pragma unroll
        for (int r = 0; r < 8; ++r) ell_vertex(tn, win, 1 + r, A, gate, nb[r], ell_ri(r), ell_rj(r));
#pragma unroll
        for (int r = 0; r < 8; ++r) ell_edge<false>(tn, win, 9 + r, A, gate, st, nb[r], 0, 0, ell_ri(r), ell_rj(r));
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = (r + 1) & 7;
            ell_edge<true>(tn, win, 17 + r, A, gate, nb[r], nb[s], ell_ri(r), ell_rj(r), ell_ri(s), ell_rj(s));
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int s = (r + 1) & 7;
            ell_tri(tn, win, 25 + r, A, gate, st, nb[r], nb[s], ell_ri(r), ell_rj(r), ell_ri(s), ell_rj(s));
        }
    }
    return ((told > R(0)) ? R(1) : R(-1)) * tn;
}
// ---------------------------------------------------------------------------
// The FP64 update with a float filter.
//
// Over one triangle of the fan, f(p) = t(p) + ||X - p||_M is convex, and its
// smallest value there is at its stationary point u over the whole plane when
// u lies inside, and otherwise on an edge that u lies beyond (walking from the
// smallest point towards u lowers f, so the walk leaves the triangle at once).
// In the scaled local frame, with P the in-plane part of A, p0 = P^-1 (xz, yz)
// the foot of X, r = ||X - p0||^2 and g the gradient of t on the triangle,
// h = P^-1 g and s = g.h, u = p0 - n h with n = sqrt(r / (1 - s)) and
// f(u) = t(p0) + sqrt(r (1 - s)).  For s >= 1 there is no such u, but any point
// far enough along -h has a lower f than the triangle and serves as well.  P,
// p0 and r are the same for all eight triangles.
//
// The filter works this out in float for the triangles that could hold a time
// below the current one, from differences rounded once, and keeps a candidate
// only where the smallest value over the fan can lie at it: a triangle's
// interior when u may be inside; a spoke when u may lie beyond it seen from
// both its triangles, a rim edge from its one; a vertex when each of its
// triangles may have its smallest point on an edge that ends there.  A triangle
// whose f(u) is above the time holds nothing, nor does a rim edge or vertex on a
// side of the fan that is too far from X for its times.  Every smallest point of the fan
// passes all of these tests, equal ones too, so what is dropped can neither
// lower the time nor have been the winner on a tie.
//
// Errors: the filter is used where |corr| of every pair of axes is small
// enough that P's determinant and r keep a quarter of their leading product
// (A's entries are off by 1e-6 relative, P^-1 by 1e-5, s by 2e-4 s), where r is
// at least 1e-3 of A.xx and A.yy, and where the triangle's source times are
// within 1e4 of sqrt(A.xx), sqrt(A.yy) of each other (their differences are off
// by 1e-3 of those); it takes s off by up to 1e-3 (1 + s) and u by 0.01 plus
// 1e-4 n |h|, in units of the spacings.  Elsewhere every candidate is kept.
// Where a source is NaN the tests of point_update_ellip decide, for their order
// does.
//
// The tests tell the candidates' exact values apart, the update the rounded
// ones.  What the margin of u (0.01 of a weight, so 0.007 of a spacing) keeps
// out is above the smallest value by at least 2.5e-5 times f's curvature, which
// for a u inside is at least 0.007 min(A.xx, A.yy, r) / sqrt(r) within the
// limits above; a candidate is rounded to 4 ulp of T, the smaller of st and the
// time.  So the tests are used up to T sqrt(r) = 2^26 min(A.xx, A.yy, r): 2^26
// cell times where the spacings are alike, and less than half of where they
// could disagree (with point sources the first differing records came at 1e11).
// Beyond it, which takes a source on an absolute clock, the gates of
// point_update_ellip choose: a candidate's rounded value is at least its
// smallest source plus sqrt(r), rounded.  (256^3, FP64 parameters, 6 sweeps: 101
// ms from a source at 1e10 s, 63 at 1e5 s, where the filter still judges; 86 and
// 94 with the gates alone, as before the filter.)
//
// What is kept runs through the FP64 candidates in the order of their ids, each
// lane its own list, so the time and the winner are the same bits.
//
// float32 fields do not take this path: their times are rounded to 1e-7 of
// their own size, so candidates that the filter tells apart often tie.
//
// ms before (gated FP64 candidates) and now, with the passes' other changes of
// the time (waits, barriers, batch chunks), one source each (a 512^3 solve takes
// 190 to 310 by where its source lies): TTI 512^3 to 1e-10 374, 248; 24
// instances of 96 to 200 points per axis 476, 264; 8 sources at 192^3 with their gradients 471,
// 249; 128^3 14.3, 12.5.  A point now costs 0.3 to 0.4 FP64 candidates of the
// 33; what bounds a pass is in fold3d_wavefront.cu.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ float ell_rsqrt(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / sqrtf(x);
#endif
}
__host__ __device__ __forceinline__ float ell_rcp(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / x;
#endif
}
__host__ __device__ __forceinline__ bool ell_any(bool p)
{
#ifdef __CUDA_ARCH__
    return __any_sync(0xffffffffu, p);
#else
    return p;
#endif
}
__host__ __device__ __forceinline__ int ell_low(unsigned m)
{
#ifdef __CUDA_ARCH__
    return __ffs((int)m) - 1;
#else
    return __builtin_ctz(m);
#endif
}

// The biased exponent of x.
__host__ __device__ __forceinline__ unsigned ell_exp(double x)
{
#ifdef __CUDA_ARCH__
    return ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
#else
    unsigned long long b;
    __builtin_memcpy(&b, &x, sizeof b);
    return (unsigned)(b >> 52) & 0x7ffu;
#endif
}
// log2(a / b) of positive floats, off by less than one.
__host__ __device__ __forceinline__ int ell_log2(float a, float b)
{
#ifdef __CUDA_ARCH__
    return (__float_as_int(a) - __float_as_int(b)) >> 23;
#else
    int x, y;
    __builtin_memcpy(&x, &a, sizeof x);
    __builtin_memcpy(&y, &b, sizeof y);
    return (x - y) >> 23;
#endif
}

// m[k] for a k that is the same in the whole launch (selects, not memory).
__host__ __device__ __forceinline__ double ell_pick(const double m[6], int k)
{
    const double a = k == 0 ? m[0] : m[1], b = k == 2 ? m[2] : m[3], c = k == 4 ? m[4] : m[5];
    return k < 2 ? a : k < 4 ? b : c;
}

// ell_local in float to a few ulp, from the medium's values v (the six metric
// words in local order, or s, eps, nx, ny).
__host__ __device__ __forceinline__ EllipAT<float> ell_local_f(int kind, const EllipDir &D, const double v[6])
{
    const float hx = (float)D.hx, hy = (float)D.hy, hz = (float)D.hz;
    EllipAT<float> A;
    if (kind == kParamF64) {
        const float s = (float)v[0], e = (float)v[1], n0 = (float)v[2], n1 = (float)v[3];
        const float s2 = s * s, a = s2 * ell_rcp(1.0f + 2.0f * e), b = s2 - a;
        const float n2 = sqrtf(fmaxf((float)((1.0 - v[2] * v[2]) - v[3] * v[3]), 0.0f));
        const float x = hx * (D.ixx == 0 ? n0 : D.ixx == 3 ? n1 : n2), y = hy * (D.iyy == 0 ? n0 : D.iyy == 3 ? n1 : n2),
                    z = hz * (D.izz == 0 ? n0 : D.izz == 3 ? n1 : n2);
        A.xx = fmaf(b * x, x, a * hx * hx);
        A.yy = fmaf(b * y, y, a * hy * hy);
        A.zz = fmaf(b * z, z, a * hz * hz);
        A.xy = (float)D.sxy * b * x * y;
        A.xz = (float)D.sxz * b * x * z;
        A.yz = (float)D.syz * b * y * z;
    } else {
        A.xx = (float)v[0] * hx * hx;
        A.yy = (float)v[1] * hy * hy;
        A.zz = (float)v[2] * hz * hz;
        A.xy = (float)D.sxy * (float)v[3] * hx * hy;
        A.xz = (float)D.sxz * (float)v[4] * hx * hz;
        A.yz = (float)D.syz * (float)v[5] * hy * hz;
    }
    return A;
}

// The medium's values at cell t, as ell_local_f and ell_local_v take them.
__host__ __device__ __forceinline__ void ell_values(const EllipMedium &M, const EllipDir &D, long long t, double v[6])
{
    if (M.kind == kParamF64) {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = ell_ld(static_cast<const double *>(M.m[k]) + t);
        v[4] = v[5] = 0.0;
    } else {
        const float *const *f = reinterpret_cast<const float *const *>(M.m);
        v[0] = ell_ld(f[D.ixx] + t);
        v[1] = ell_ld(f[D.iyy] + t);
        v[2] = ell_ld(f[D.izz] + t);
        v[3] = ell_ld(f[D.ixy] + t);
        v[4] = ell_ld(f[D.ixz] + t);
        v[5] = ell_ld(f[D.iyz] + t);
    }
}

// ell_local<double> from the medium's values: the same operations.
__host__ __device__ __forceinline__ EllipA ell_local_v(int kind, const EllipDir &D, const double v[6])
{
    double l[6] = {v[0], v[1], v[2], v[3], v[4], v[5]};  // xx yy zz xy xz yz
    if (kind == kParamF64) {
        double m[6];
        ell_metric_from_param(v[0], v[1], v[2], v[3], m);
        l[0] = ell_pick(m, D.ixx);
        l[1] = ell_pick(m, D.iyy);
        l[2] = ell_pick(m, D.izz);
        l[3] = ell_pick(m, D.ixy);
        l[4] = ell_pick(m, D.ixz);
        l[5] = ell_pick(m, D.iyz);
    }
    EllipA A;
    A.xx = l[0] * D.hx * D.hx;
    A.yy = l[1] * D.hy * D.hy;
    A.zz = l[2] * D.hz * D.hz;
    A.xy = (double)D.sxy * l[3] * D.hx * D.hy;
    A.xz = (double)D.sxz * l[4] * D.hx * D.hz;
    A.yz = (double)D.syz * l[5] * D.hy * D.hz;
    return A;
}

// Candidates kept by the filter: bit r of each, the rim's r-th vertex, spoke,
// rim edge and triangle; bit 8 of vert, st.
struct EllKeep {
    unsigned vert, spoke, rim, tri;
    // above the new time's distance from st; where all are kept, +inf, or -inf
    // for times too large to judge, or NaN for a NaN among the sources
    float Eb;
};

// The largest; NaN if one of them is.
__host__ __device__ __forceinline__ float ell_max_nan(float a, float b, float c)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
    return y;
#else
    return a != a ? a : b != b ? b : c != c ? c : fmaxf(fmaxf(a, b), c);
#endif
}

// c: float(st - s_r) of the rim, E: float(tn - st), eT: the exponent (ell_exp)
// of the smaller of st and tn.
__host__ __device__ __forceinline__ EllKeep ell_filter(bool active, const float c[8], float E, unsigned eT,
                                                       const EllipAT<float> &A)
{
    EllKeep K = {0u, 0u, 0u, 0u, HUGE_VALF};
    const float cof = A.xx * A.yy - A.xy * A.xy, icof = ell_rcp(cof);
    const float px = (A.yy * A.xz - A.xy * A.yz) * icof, py = (A.xx * A.yz - A.xy * A.xz) * icof;
    const float r = A.zz - (A.xz * px + A.yz * py);
    const float big = fmaxf(A.xx, A.yy), small = fminf(A.xx, A.yy);
    float mx = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; k += 2) mx = ell_max_nan(mx, c[k], c[k + 1]);
    // every comparison is false for a NaN
    const bool sane = small > 1e-30f && big < 1e30f && A.zz < 1e30f && cof > 0.25f * (A.xx * A.yy) &&
                      r > 0.25f * A.zz && r > 1e-3f * big && E > -1e30f && mx < 1e30f;
    float Eb = fmaf(fabsf(E), 1e-6f, E);  // above the new time's distance from st
    const float sr = r * ell_rsqrt(fmaxf(r, 1e-36f));
    const float far2 = 1e8f * small;
    const bool near = active && (!sane || Eb + mx > 0.99f * sr);
    if (!ell_any(near)) return K;
    // T above 2^26 min(small, r) / sr, to a factor of two
    const bool coarse = sane && (int)eT - 1023 > 25 + ell_log2(fminf(small, r), sr);
    const bool go = near && sane && !coarse;
    unsigned VA = 0, VB = 0, VC = 0, TR = 0;
    // ||X - p|| is at least this on the fan's sides x = 1, y = 1, x = -1, y = -1
    const float kx = cof * ell_rcp(A.yy), ky = cof * ell_rcp(A.xx);
    float side[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float off = (q < 2 ? 1.0f : -1.0f) - ((q & 1) ? py : px), d2 = fmaf(off * off, (q & 1) ? ky : kx, r);
        side[q] = 0.995f * (d2 * ell_rsqrt(fmaxf(d2, 1e-36f)));
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int ka = (k & 1) ? (k + 1) & 7 : k, kc = (k & 1) ? k : k + 1;  // axis neighbour and corner
        const float ca = c[ka], cc = c[kc];
        const bool in = go && Eb + fmaxf(fmaxf(ca, cc), 0.0f) > 0.99f * sr;
        if (ell_any(in)) {
            const bool along_x = (ka & 3) == 0;
            const float sa = (ka < 4) ? 1.0f : -1.0f;                       // sign of the axis neighbour
            const float sc = (float)(along_x ? ell_rj(kc) : ell_ri(kc));    // and of the corner, across
            const float ga = -sa * ca, gc = sc * (ca - cc);
            const float gx = along_x ? ga : gc, gy = along_x ? gc : ga;
            const float hx = fmaf(A.yy, gx, -(A.xy * gy)) * icof, hy = fmaf(A.xx, gy, -(A.xy * gx)) * icof;
            const float s = fmaf(gx, hx, gy * hy), ds = fmaf(1e-3f, s, 1e-3f), e = 1.0f - s;
            const float elo = e - ds, ehi = e + ds;
            const float bx = gx * px, by = gy * py, base = bx + by;
            const float tol = 1e-3f * (sr + fabsf(bx) + fabsf(by));
            const float qlo = fmaxf(elo, 1e-6f), qhi = fmaxf(ehi, 1e-6f);
            const float rlo = ell_rsqrt(qlo), rhi = ell_rsqrt(qhi);
            const float n_hi = sr * rlo, n_lo = sr * rhi;
            const float ux0 = fmaf(-n_lo, hx, px), uy0 = fmaf(-n_lo, hy, py);
            const float ux1 = fmaf(-n_hi, hx, px), uy1 = fmaf(-n_hi, hy, py);
            const float m0 = sa * (along_x ? ux0 : uy0), w0 = sc * (along_x ? uy0 : ux0);
            const float m1 = sa * (along_x ? ux1 : uy1), w1 = sc * (along_x ? uy1 : ux1);
            // weights of the corner, of the axis neighbour and of st at u, over the range of n
            const float lc = fminf(w0, w1), la = fminf(m0 - w0, m1 - w1), l0 = 1.0f - fmaxf(m0, m1);
            const float hc = fmaxf(w0, w1), ha = fmaxf(m0 - w0, m1 - w1), h0 = 1.0f - fminf(m0, m1);
            const float mg = fmaf(1e-4f * n_hi, fabsf(hx) + fabsf(hy), 0.01f);
            const bool odd = !(fmaxf(ca * ca, cc * cc) < far2);  // differences too coarse, or not finite
            const bool late = !odd && elo > 0.0f && base + sr * (qlo * rlo) - tol > Eb;
            if (in && !late) {
                const bool vc_ = odd || lc < mg, va_ = odd || la < mg, v0_ = odd || l0 < mg;
                // u's weight of a vertex may be negative: the opposite edge may hold the smallest point
                VA |= (unsigned)((k & 1) ? va_ : vc_) << k;
                VB |= (unsigned)((k & 1) ? vc_ : va_) << k;
                VC |= (unsigned)(v0_ && (odd || Eb + fmaxf(ca, cc) > side[ka >> 1])) << k;
                TR |= (unsigned)(odd || (ehi > 0.0f && hc > -mg && ha > -mg && h0 > -mg)) << k;
                if (!(va_ | vc_ | v0_) && elo > 0.0f) Eb = fminf(Eb, base + sr * (qhi * rhi) + tol);
            }
        }
    }
    auto prev = [](unsigned m) { return ((m << 1) | (m >> 7)) & 0xffu; };  // of the triangle before
    K.tri = TR;
    K.rim = VC;
    K.spoke = VA & prev(VB);
    unsigned early = 0;  // rim vertices that are not too far for their times
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float d = (k & 1) ? fmaxf(side[k >> 1], side[((k + 1) >> 1) & 3]) : side[k >> 1];
        early |= (unsigned)!(Eb + c[k] < d) << k;
    }
    K.vert = ((VA | VC) & prev(VB | VC) & early) | (((VA | VB) == 0xffu) ? 0x100u : 0u);
    K.Eb = Eb;
    if (near && !go) K = {0x1ffu, 0xffu, 0xffu, 0xffu, coarse ? -HUGE_VALF : mx == mx ? HUGE_VALF : mx};
    return K;
}

// Whether an edge kept by ell_filter still may: its own stationary point in
// float.  cp, cq: c of its ends (0 for st).  Judged only where the ends' times
// are within 30 sqrt(a) of st's (a the edge's length squared), which leaves
// their difference within 4e-6 sqrt(a), and away from den = 0.
__host__ __device__ __forceinline__ bool ell_edge_may(const EllipAT<float> &A, float Eb, float cp, float cq, int pi,
                                                      int pj, int qi, int qj)
{
    const float x = (float)pi, y = (float)pj, ex = (float)(qi - pi), ey = (float)(qj - pj);
    const float gx = fmaf(A.xx, ex, A.xy * ey), gy = fmaf(A.xy, ex, A.yy * ey);  // P e
    const float a = fmaf(ex, gx, ey * gy);
    const float b = fmaf(ex, A.xz, ey * A.yz) - fmaf(x, gx, y * gy);
    const float c = A.zz + x * fmaf(A.xx, x, 2.0f * (A.xy * y - A.xz)) + y * fmaf(A.yy, y, -2.0f * A.yz);
    const float d = cp - cq, dd = d * d, den = a - dd, w = 0.01f * (a + dd);
    if (!(fmaxf(cp * cp, cq * cq) < 1e3f * a) || fabsf(den) < w) return true;
    if (den < 0.0f) return false;
    const float q = fmaxf(fmaf(a, c, -(b * b)), 0.0f) * ell_rcp(den), n = q * ell_rsqrt(fmaxf(q, 1e-36f));
    const float ia = ell_rcp(a), lam = fmaf(-d, n, b) * ia, mg = fmaf(1e-3f * fabsf(d * n), ia, 0.01f);
    if (lam < -mg || lam > 1.0f + mg) return false;
    return !(fmaf(lam, d, n) - cp > Eb + 2e-3f * (n + fabsf(d)));
}

// And a rim vertex (i, j); cv: its c.
__host__ __device__ __forceinline__ bool ell_vertex_may(const EllipAT<float> &A, float Eb, float cv, int i, int j)
{
    const float x = (float)i, y = (float)j;
    const float c = A.zz + x * fmaf(A.xx, x, 2.0f * (A.xy * y - A.xz)) + y * fmaf(A.yy, y, -2.0f * A.yz);
    const float n = c * ell_rsqrt(fmaxf(c, 1e-36f));
    return !(0.999f * n > Eb + cv);
}

// x / c from r = RN(1/c) where that is exact (Markstein's two remainder
// corrections, as div_by_const in fold3d_fast.cuh), else x / c.
__host__ __device__ __forceinline__ double ell_div(double x, double c, double r, bool ok)
{
    if (!ok || ell_exp(x) - (1023u - 400u) > 800u) return x / c;
    double q = x * r;
    double e = fma(-q, c, x);
    q = fma(e, r, q);
    e = fma(-q, c, x);
    return fma(e, r, q);
}

// ell_tri and ell_edge for a run-time r without their skips.  The terms that
// ell_bf multiplies by zero are left out (A is finite here, so they add
// nothing), and the divisions by one denominator share its reciprocal.
__host__ __device__ __forceinline__ void ell_try_tri(double &tn, int &win, int r, const EllipA &A, double t0, double ta,
                                                     double tb)
{
    const int q = (r + 1) & 7;
    const double ai = ell_ri(r), aj = ell_rj(r), bi = ell_ri(q), bj = ell_rj(q);
    const bool odd = r & 1;                    // a is the corner, b the axis neighbour
    const bool x = ((odd ? q : r) & 3) == 0;   // that neighbour lies along x
    const double ci = odd ? ai : bi, cj = odd ? aj : bj;
    const double pax = x ? A.xx : A.yy;                                   // axis . axis
    const double pc = (A.xx + A.yy) + 2.0 * (ci * cj) * A.xy;             // corner . corner
    const double p12 = pax + (ci * cj) * A.xy;                            // axis . corner
    const double p11 = odd ? pc : pax, p22 = odd ? pax : pc;
    const double qax = x ? ci * A.xz : cj * A.yz, qc = ci * A.xz + cj * A.yz;
    const double q1 = odd ? qc : qax, q2 = odd ? qax : qc;
    const double d1 = ta - t0, d2 = tb - t0;
    const double det = p11 * p22 - p12 * p12;
    if (!(det > 0.0)) return;
    const double u1 = p22 * d1 - p12 * d2, u2 = p11 * d2 - p12 * d1;
    const double w1 = p22 * q1 - p12 * q2, w2 = p11 * q2 - p12 * q1;
    const double rd = 1.0 / det;
    const bool ok = ell_exp(det) - (1023u - 400u) <= 800u && ell_exp(rd) - (1023u - 400u) <= 800u;
    const double s = ell_div(d1 * u1 + d2 * u2, det, rd, ok);
    const double rr = A.zz - ell_div(q1 * w1 + q2 * w2, det, rd, ok);
    if (!(s < 1.0 && rr > 0.0)) return;
    const double n = sqrt(rr / (1.0 - s));
    const double l1 = ell_div(w1 - n * u1, det, rd, ok), l2 = ell_div(w2 - n * u2, det, rd, ok);
    if (l1 > 0.0 && l2 > 0.0 && l1 + l2 < 1.0) {
        const double cand = t0 + (l1 * d1 + l2 * d2) + n;
        if (cand < tn) {
            tn = cand;
            win = 25 + r;
        }
    }
}
__host__ __device__ __forceinline__ void ell_try_edge(double &tn, int &win, int id, const EllipA &A, double tp,
                                                      double tq, int pi, int pj, int qi, int qj)
{
    const int ei = qi - pi, ej = qj - pj;
    const double a = ell_bf(A, ei, ej, 0, ei, ej, 0);
    const double b = ell_bf(A, ei, ej, 0, -pi, -pj, 1);
    const double c = ell_bf(A, -pi, -pj, 1, -pi, -pj, 1);
    const double d = tq - tp;
    const double den = a - d * d;
    const double disc = a * c - b * b;
    if (den > 0.0 && disc > 0.0) {
        const double n = sqrt(disc / den);
        const double lam = (b - d * n) / a;
        if (lam > 0.0 && lam < 1.0) {
            const double cand = tp + lam * d + n;
            if (cand < tn) {
                tn = cand;
                win = id;
            }
        }
    }
}

// New signed value of the target at field index t whose stored value is `told`
// from the nine previous-plane magnitudes (rim order, st last), and the winning
// candidate (-1: none).  Every lane of the warp calls it; a lane that is not
// `active` changes nothing.  sh: scratch of nine doubles, `stride` elements
// apart (shared memory on the device).
__host__ __device__ __forceinline__ double ell_update_fan(bool active, double told, const double (&s)[9],
                                                          const double (&v)[6], int kind, const EllipDir &D, double *sh,
                                                          int stride, int &win)
{
    const double st = s[8];
    double tn = fabs(told);
    win = -1;
    float c[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        c[r] = (float)(st - s[r]);
        sh[r * stride] = s[r];
    }
    sh[8 * stride] = st;
    const EllipAT<float> Af = ell_local_f(kind, D, v);
    EllKeep K = ell_filter(active, c, (float)(tn - st), ell_exp(tn < st ? tn : st), Af);
    if (ell_any((K.vert | K.spoke | K.rim | K.tri) != 0)) {
        const bool known = fabsf(K.Eb) < HUGE_VALF;
        const bool gates = K.Eb != K.Eb || K.Eb == -HUGE_VALF;
        if (ell_any(gates)) {  // point_update_ellip's tests in place of the filter's
            if (gates) {
                const EllipA A = ell_local_v(kind, D, v);
                if (K.vert >> 8) ell_vertex(tn, win, 0, A, 0.0, st, 0, 0);
                K.vert &= 0xffu;
                double m = st;
#pragma unroll 1
                for (int r = 0; r < 8; ++r) m = ell_min(m, sh[r * stride]);
                if (!(tn > m)) K.vert = K.spoke = K.rim = K.tri = 0;  // a NaN among the sources decides it, too
                const double g = K.Eb == K.Eb ? ell_skip_bound(A) : 0.0;
#pragma unroll 1
                for (int r = 0; r < 8; ++r) {
                    const double a = sh[r * stride], b = ell_min(a, sh[((r + 1) & 7) * stride]);
                    if (tn <= a + g) K.vert &= ~(1u << r);
                    if (tn <= ell_min(st, a) + g) K.spoke &= ~(1u << r);
                    if (tn <= b + g) K.rim &= ~(1u << r);
                    if (tn <= ell_min(st, b) + g) K.tri &= ~(1u << r);
                }
            }
        }
        unsigned vert = K.vert & 0xffu, edge = known ? 0u : K.spoke | (K.rim << 8);
        for (unsigned m = known ? vert : 0u; ell_any(m != 0);) {
            if (m) {
                const int r = ell_low(m);
                m &= m - 1;
                if (!ell_vertex_may(Af, K.Eb, (float)(st - sh[r * stride]), ell_ri(r), ell_rj(r))) vert &= ~(1u << r);
            }
        }
        for (unsigned m = known ? K.spoke | (K.rim << 8) : 0u; ell_any(m != 0);) {
            if (m) {
                const int k = ell_low(m), r = k & 7, q = (k < 8) ? r : (r + 1) & 7;
                m &= m - 1;
                const bool spoke = k < 8;
                if (ell_edge_may(Af, K.Eb, spoke ? 0.0f : (float)(st - sh[r * stride]), (float)(st - sh[q * stride]),
                                 spoke ? 0 : ell_ri(r), spoke ? 0 : ell_rj(r), ell_ri(q), ell_rj(q)))
                    edge |= 1u << k;
            }
        }
        if (ell_any((vert | edge | K.tri | (K.vert >> 8)) != 0)) {
            const EllipA A = ell_local_v(kind, D, v);
            const bool finite = fabs(A.xx) + fabs(A.yy) + fabs(A.zz) + fabs(A.xy) + fabs(A.xz) + fabs(A.yz) < 1e300;
            if (K.vert >> 8) ell_vertex(tn, win, 0, A, 0.0, st, 0, 0);
            while (ell_any(vert != 0)) {
                if (vert) {
                    const int r = ell_low(vert);
                    vert &= vert - 1;
                    ell_vertex(tn, win, 1 + r, A, 0.0, sh[r * stride], ell_ri(r), ell_rj(r));
                }
            }
            while (ell_any(edge != 0)) {
                if (edge) {
                    const int k = ell_low(edge), r = k & 7, q = (k < 8) ? r : (r + 1) & 7;
                    edge &= edge - 1;
                    const bool spoke = k < 8;
                    ell_try_edge(tn, win, 9 + k, A, spoke ? st : sh[r * stride], sh[q * stride], spoke ? 0 : ell_ri(r),
                                 spoke ? 0 : ell_rj(r), ell_ri(q), ell_rj(q));
                }
            }
            unsigned tri = K.tri;
            while (ell_any(tri != 0)) {
                if (tri) {
                    const int r = ell_low(tri), q = (r + 1) & 7;
                    tri &= tri - 1;
                    if (finite) ell_try_tri(tn, win, r, A, st, sh[r * stride], sh[q * stride]);
                    else ell_tri(tn, win, 25 + r, A, 0.0, st, sh[r * stride], sh[q * stride], ell_ri(r), ell_rj(r),
                                 ell_ri(q), ell_rj(q));
                }
            }
        }
    }
    return ((told > 0.0) ? 1.0 : -1.0) * tn;
}
#endif  // __CUDACC__

}  // namespace fold3d
