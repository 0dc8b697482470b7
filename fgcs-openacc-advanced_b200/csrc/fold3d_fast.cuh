// fold3d_fast.cuh -- the Fold3dPMM point update with its per-direction
// constants folded on the host.
//
// Same results as fold3d_solver.cuh, bit for bit.  Two facts make that
// possible:
//
// 1. Every argument of the reference's 24 local-solver calls that does not
//    depend on the previous-plane values -- the rotated drifts
//    ((ax*dxx + ay*dyy)/dxy and the like, AN_ISO_1_OpenACC.c:243-253,
//    :172-173), F*F - ay*ay, F*F - az*az, the whole fall-back candidate of
//    FoldEdge2Points except the final addition (:99-113), and the 1-D normal
//    candidate except the final addition (:214-228) -- is a constant of the
//    sweep direction and of the side of the target (the drift is negated on
//    the negative side).  The host evaluates those constants with the same
//    expressions and the same IEEE double rounding (no FMA contraction), and
//    the kernel reads them from a table.
//
// 2. Three of the four divisions in each solver body divide by such a
//    constant c.  They are computed as correctly rounded quotients without a
//    division instruction, from r = RN(1/c) (Markstein's method, P. Markstein,
//    "Computation of elementary functions on the IBM RISC System/6000
//    processor", IBM J. Res. Dev. 34(1), 1990): q0 = RN(x*r); one
//    remainder-correction step with the exact FMA remainder x - c*q gives a
//    quotient within one ulp, and a second step then yields RN(x/c).  This
//    holds for normal, finite operands and quotients, which is the case for
//    every such division in the sweep (travel-time differences over grid
//    spacings and bounded slowness terms).
//
// Data-dependent square roots and the two divisions by data-dependent
// values keep CUDA's IEEE operations.  Each solver call only accepts
// candidates strictly below the current time, and the calls' own gates on the
// current time only skip calls that could not lower it, so the calls may be
// visited in any order.  One gate of the reference is different: its early
// exit (:231) leaves all sixteen calls out when the time after the 1-D
// candidate is below seven of the nine sources, xnt and ynt not among them.
// It is kept as it is.  (Evaluating a point again with the same sources still
// changes nothing: its time has only fallen, so the exit is taken again
// wherever it was, and elsewhere the same candidates are not below it.)
//
// 3. One more such gate skips a FoldSurf3Points body (its nested edge still
//    runs) when the current time is at most min(s0, s1, s2) + B.  The body
//    solves the drift medium's eikonal F|p| + a.p = 1 for the plane wave
//    through the three base values and takes the root whose ray, of
//    direction F p/|p| + a, points from the base plane to the target (:152);
//    it accepts the candidate only if that ray leaves the base triangle at a
//    point inside it (:158-163).  The time there, interpolated linearly, is
//    at least the smallest base value, and the ray then crosses the slab of
//    width dzz between base and target, which takes at least dzz / (F + az):
//    one time unit after leaving a point, the front is the sphere
//    |x - a| = F.  B is the larger of that bound and one proved per call
//    site by a search over the body's two gradients (fold3d_tables.cpp),
//    less a relative 1e-3, far above the body's rounding (below 1e-6
//    relative where F^2 >= 1.1 |a|^2, through the square root of a cancelled
//    difference); 0 for stronger drifts.
//
// 4. FoldEdge2Points bodies get a gate of the same kind, B in EdgeK.
//    Its footpoint test (:88,92) does not follow the ray of its own root: it
//    uses the direction w = (F'/F) p/|p| + a2 (F' = sqrt(F^2 - ay^2),
//    a2 = (ax, az), p = (d, c) the plane wave's slowness, which satisfies
//    F'|p| + a2.p = 1), where the ray is F' p/|p| + a2.  So the candidate
//    exceeds the linear time at the test's footpoint (at least min(s0, s1))
//    by dzz (p.w) / w_z, with p.w = 1 - F'|p| (1 - 1/F).  When
//      - ga > 0 and |ax| < sqrt(ga) (then c0 = 1 - d ax > 0 wherever the
//        root exists, and the root is the upper one of F'|p| + a2.p = 1,
//        whose ray points towards the target),
//      - F' > |a2| (so |p| <= 1 / (F' - |a2|)), and
//      - F >= 1 with az >= 0, or F <= 1 with az <= 0 (then w_z > 0 too),
//    p.w >= 1 - F'(1 - 1/F) / (F' - |a2|) for F >= 1 (>= 1 for F <= 1) and
//    w_z <= F'/F + az, which gives one bound; elsewhere it is 0.  B is the
//    larger of that and one proved per call site by an interval search over
//    the body's single gradient d (fold3d_tables.cpp), less the same
//    relative 1e-3 margin.  The fall-back candidate from s1 alone is not
//    gated.
//
// 5. Gates and bodies in float first.  A body that passes its gate costs 100
//    to 150 FP64 instructions of which most depend on one another, and in a
//    settled field it nearly always ends in a rejection: over 192^3 sweeps of
//    the reference's workload a warp row enters 4.5 bodies and 0.17 of its
//    points improve; with the filter it enters 0.4.  So every gate and every
//    body is first judged in float, from differences rounded once:
//    c_r = float(st - s_r), E = float(tn - st).
//
//    Gates.  tn - min(sources) = E + max(c), so a call can only matter when
//    E + max(c) > B (its skip bound; an edge's fall-back when E + c > K,
//    covered by taking min(B, K)).  E is raised by 4e-7 |E|, more than the
//    roundings of E, c and the sum where the two are about equal, and the
//    thresholds are rounded down, so no call that could matter is dropped.
//    The calls' fixed early returns (:71, :132, :170) are signs of c and of
//    c_r - c_s, which rounding never turns into a false return.
//
//    Bodies.  Scaled by F (u = F dx, v = F dy, a/F) the triangle's body is
//    al = 1 - a.(u,v), q = al^2 - g(u^2 + v^2), S = sqrt q,
//    z = (S - az al)/g, w = al - az z (= F|p| while F > |a|), and the ray is
//    (u + ax w, v + ay w, S): its time and its four footpoint tests need one
//    square root and no division.  An edge is the same in two dimensions, with
//    the reference's own footpoint direction (4. above).  A rejection counts
//    only if it is clear by m = eps (1 + u^2 + v^2 + al^2)/S, eps = 1e-3.
//    Bound on the errors, M^2 = 1 + u^2 + v^2 + al^2 and spacings within a
//    factor of 8 of each other: u and v are off by 2e-6 M (their c by 2^-24
//    relative, |c| F/h <= 20 M; for a nested edge M^2 also holds
//    (c F/(4h))^2), al by 8e-6 M, q by 4e-5 M^2, so S by 2e-5 M^2/S; with
//    F^2 >= 1.1 |a|^2 (az^2/g <= 10) z, w and the ray are then off by at most
//    3.2e-4 M^2/S, a third of m.  Other media and spacings set eps = +inf,
//    which rejects nothing, and a non-finite value makes m infinite or NaN,
//    which rejects nothing either.  What is left goes through the FP64 bodies
//    with all their gates, so the result is the same bits; a footpoint that
//    the filter finds inside by m on all sides is not tested again, and a
//    certain acceptance (its time above all sources' by m too) lowers the
//    bound that later bodies are judged against.
#pragma once
#include <cstdint>
#include <cstring>

namespace fold3d {

// Constants of one FoldEdge2Points call site (AN_ISO_1_OpenACC.c:59-114).
struct EdgeK {
    double ax, ay, az;  // drift arguments as passed
    double hx, hz;      // spacing arguments (dxx, dzz)
    double rhx;         // RN(1/hx)
    double g, rg;       // F*F - ay*ay and RN(1/g)
    double ga, rga;     // g - az*az and RN(1/ga)
    double K;           // fall-back increment g'/c' of :99-113 (when fb_ok)
    double B;           // body skipped when the time is <= min(s0, s1) + B (4. above)
    int early;          // ax > 0: return when s1 > s0 (:71)
    int fb_ok;          // fall-back defined: its q > 0 and c > 0
};

// Constants of one FoldSurf3Points call site (:119-175).
struct SurfK {
    double ax, ay;      // drift arguments (az, F, hz are common)
    double hx, hy;      // dxx, dyy as passed
    double rhx, rhy;
    int e1, e2;         // ax > 0, ay > 0 (early returns of :132)
    int nblock;         // ax*dzz + az*dxx > 0: nested edge skipped when s1 > s2 (:170)
    int pad_;
    double B;           // body skipped when the time is <= min(s0, s1, s2) + B (3. above)
    EdgeK nest;         // the nested FoldEdge2Points call (:172-173)
};

// Float constants of the filter (5. above) of one FoldSurf3Points body and of
// one FoldEdge2Points call, in the order the kernels read them (16-byte
// loads).  Drifts are divided by the body's speed (F, or F' = sqrt(F^2 -
// ay^2) for an edge), slownesses multiplied by it.
struct alignas(16) TriF {
    float kx, ky;      // F/dxx, F/dyy
    float ax, ay;      // drift / F
    float r1, r2;      // dyy/(dxx+dyy), dxx/(dxx+dyy)
    float s1, s2;      // dzz/(dxx+dzz), dxx/(dxx+dzz)
};
struct alignas(16) EdgeF {
    float k, kz;       // F'/dxx, F'/dzz
    float ax, az;      // drift / F'
    float ga, iga;     // 1 - az^2, 1/(1 - az^2)
    float fx, fz;      // F ax, F az: the drift in the footpoint's direction (4. above)
    float s1, s2;      // dzz/(dxx+dzz), dxx/(dxx+dzz)
    float ka;          // 1 + |fx| + |fz|
    float K;           // fall-back increment, rounded down; +inf where it is undefined
};

// Sources of a target point: the rim of the fan in order xt, txy, yt, tym,
// xnt, txnyn, ynt, txm (0..7) and st (8).  The sources of call k of the
// eight FoldSurf3Points (:233-240), four bits each, k = 0 lowest.
constexpr unsigned kTriS1 = 0x22664400u;  // xt xt xnt xnt ynt ynt yt yt
constexpr unsigned kTriS2 = 0x31753571u;  // txy txm txnyn tym txnyn txm txy tym

// The filter's constants of one side (5. above).  Call k of the bit masks and
// thresholds is triangle k, nested edge 8 + k, outer edge 16 + k.  Built in
// the direction's local frame; orient_table() turns it into the frame of the
// plane's two axes for the kernels that walk a plane's rows.
struct alignas(16) SideFilter {
    float gB[24];             // thresholds of the gates, rounded down
    float outer;              // the smallest of gB
    float eps;                // margin, +inf where the bodies are not filtered
    float faz, fg, fig, fkz;  // az/F, 1 - faz^2, 1/fg, F/dzz
    float fhz;                // dzz/F, rounded up
    unsigned every;           // calls that are never gated (all of them, or none)
    // the calls' fixed early returns as bit masks, bit k for call k
    unsigned m_e1, m_e2;      // surf[k].e1, .e2
    unsigned m_nest_early;    // surf[k].nest.early
    unsigned m_edge_early;    // edge[k].early
    int d1_ok;                // 1-D candidate
    int named[2];             // rim points that the early exit (:231) names: 0 or 4, and 2 or 6
    double K1;
    // the FP64 constants' entries of triangle k and outer edge k (orient_table)
    unsigned char surf_at[8], edge_at[8];
    TriF tri[8];
    EdgeF ef[16];             // nested edges, then outer edges
};

// All constants of one direction on one side of the source surface.
struct alignas(16) SideTable {
    double F, az, hz;
    double g, rg;       // F*F - az*az, RN(1/g)          (:147)
    double K1;          // 1-D candidate increment dzz*dzz/q (:225)
    int d1_ok;          // 1-D candidate defined (:219, :223)
    // the per-call flags below as bit masks, bit k for call k
    unsigned m_e1, m_e2, m_nblock;  // surf[k].e1, .e2, .nblock
    unsigned m_nest_early;          // surf[k].nest.early
    unsigned m_edge_early;          // edge[k].early
    SurfK surf[8];      // the eight FoldSurf3Points calls (:233-240), in order
    EdgeK edge[8];      // the eight FoldEdge2Points calls (:242-253), in order
    SideFilter flt;     // the float filter (5. above)
};

struct DirTable {
    SideTable side[2];  // [0]: target >= 0 (or 0), [1]: target < 0 (drift negated)
};

// The filter's parts of a table turned from the local frame into the frame of
// the plane's axes u and v (rim point 0 at u + 1, 2 at v + 1): x_is_u, the
// local x axis is u; xs, ys, the signs of the local axes.
void orient_table(DirTable &tab, bool x_is_u, int xs, int ys);

// Safe operand range of div_by_const: |x| and |c| in [2^-400, 2^401), which
// keeps the quotient, the products and the remainders normal.  The host
// stores r = 0 for a constant outside that range.
constexpr unsigned kDivExpLo = 1023 - 400;
constexpr unsigned kDivExpSpan = 800;

#ifdef __CUDACC__
// The functions below also compile for the host (IEEE double, fma, sqrt and
// division correctly rounded on both sides, no contraction), where a test
// runs them against the CPU statement of the reference.
__host__ __device__ __forceinline__ unsigned hi_word(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(x);
#else
    uint64_t b;
    std::memcpy(&b, &x, sizeof b);
    return (unsigned)(b >> 32);
#endif
}

// Correctly rounded x / c for a constant c given r = RN(1/c) (r == 0: use
// the IEEE division); see above.  Operands outside the safe range, zero
// included, also take the IEEE division.
__host__ __device__ __forceinline__ double div_by_const(double x, double c, double r)
{
    const unsigned ex = (hi_word(x) >> 20) & 0x7ffu;
    if (ex - kDivExpLo > kDivExpSpan || r == 0.0) return x / c;
    double q = x * r;
    double e = fma(-q, c, x);
    q = fma(e, r, q);
    e = fma(-q, c, x);
    return fma(e, r, q);
}

__host__ __device__ __forceinline__ double kmin(double a, double b) { return (a < b) ? a : b; }

// Fixed early returns: of a FoldSurf3Points call (:132), of its nested
// FoldEdge2Points call (:170, :71, behind the former), of an outer one (:71).
__host__ __device__ __forceinline__ bool surf_closed(double s0, double s1, double s2, const SurfK &k)
{
    return ((k.e1 != 0) & (s1 > s0)) | ((k.e2 != 0) & (s2 > s1));
}
__host__ __device__ __forceinline__ bool nest_closed(double s0, double s1, double s2, const SurfK &k)
{
    return surf_closed(s0, s1, s2, k) | ((k.nblock != 0) & (s1 > s2)) | ((k.nest.early != 0) & (s2 > s1));
}

// FoldEdge2Points' own body (:75-97).  inside: the footpoint is known to lie
// on the edge (5. below), so its test is left out.
__host__ __device__ __forceinline__ void edge_body(double &tn, double s0, double s1, const EdgeK &k, double F,
                                                   bool inside)
{
    const double mn = kmin(s1, s0);
    if (tn <= mn + k.B) return;  // 4. above
    const double d = div_by_const(s1 - s0, k.hx, k.rhx);
    double c = (1.0 - d * k.ax);
    double q = k.g * (c * c - d * d * k.ga);
    if (!(0.0 < q)) return;
    c = div_by_const(-k.az * c + sqrt(q), k.ga, k.rga);
    q = s0 + k.hz * c;
    if (!(q < tn && q > mn)) return;
    if (!inside) {
        const double g = sqrt(div_by_const((d * d + c * c) * F * F, k.g, k.rg));
        const double xe = -k.hz * (d + k.ax * g) / (c + k.az * g);
        if (!(0.0 < xe && xe < k.hx)) return;
    }
    tn = q;
}

// FoldSurf3Points' own body (:131-165); inside as above.
__host__ __device__ __forceinline__ void surf_body(double &tn, double s0, double s1, double s2, const SurfK &k,
                                                   const SideTable &t, bool inside)
{
    const double mn = kmin(s0, kmin(s1, s2));
    if (tn <= mn + k.B) return;  // 3. above
    const double dx = div_by_const(s1 - s0, k.hx, k.rhx);
    const double dy = div_by_const(s2 - s1, k.hy, k.rhy);
    double dd = dx * dx + dy * dy;
    double al = 1.0 - k.ax * dx - k.ay * dy;
    double q = al * al - dd * t.g;
    if (!(q > 0.0)) return;
    al = div_by_const(-t.az * al + t.F * sqrt(q), t.g, t.rg);
    const double g = s0 + t.hz * al;
    if (!(g < tn && g > mn)) return;
    if (!inside) {
        q = sqrt(dd + al * al);
        dd = -t.hz / (t.F * al + t.az * q);
        const double xe = dd * (t.F * dx + k.ax * q);
        const double ye = dd * (t.F * dy + k.ay * q);
        if (!(0.0 <= kmin(xe, ye) && ye * k.hx <= xe * k.hy && xe <= k.hx)) return;
    }
    tn = g;
}

// ---------------------------------------------------------------------------
// The float filter (5. above) and the point update built on it.  On the
// device a warp's lanes hold 32 points and the calls are visited for all of
// them together: the warp walks the union of its lanes' calls, so call
// numbers and table addresses are uniform, and an FP64 body runs only when
// some lane needs it.  On the host a "warp" is one point.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ bool lanes_any(bool p)
{
#ifdef __CUDA_ARCH__
    return __any_sync(0xffffffffu, p);
#else
    return p;
#endif
}

__host__ __device__ __forceinline__ unsigned lanes_or(unsigned m)
{
#ifdef __CUDA_ARCH__
    return __reduce_or_sync(0xffffffffu, m);
#else
    return m;
#endif
}

// 1/sqrt(x) to a few ulp, x normal and > 0.
__host__ __device__ __forceinline__ float filter_rsqrt(float x)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / sqrtf(x);
#endif
}

// The larger one; NaN if either is.
__host__ __device__ __forceinline__ float max_nan(float a, float b)
{
#ifdef __CUDA_ARCH__
    float y;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
    return y;
#else
    return a != a ? a : b != b ? b : fmaxf(a, b);
#endif
}

// m with the sign bit of x appended.
__host__ __device__ __forceinline__ unsigned push_sign(unsigned m, float x)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(__float_as_uint(x), m, 1);
#else
    uint32_t b;
    std::memcpy(&b, &x, sizeof b);
    return (m << 1) | (x != x ? 0u : b >> 31);  // the device's NaN has a clear sign
#endif
}

// 16-byte loads of a call's constants.
template <class K> __host__ __device__ __forceinline__ K load_consts(const K &k)
{
    static_assert(sizeof(K) % 16 == 0, "whole 16-byte words");
    K r;
#pragma unroll
    for (int i = 0; i < (int)(sizeof(K) / 16); ++i) reinterpret_cast<float4 *>(&r)[i] = reinterpret_cast<const float4 *>(&k)[i];
    return r;
}

// What the filter says of a body: it certainly cannot lower the time, its
// footpoint is certainly inside, or neither.
enum Verdict { kNever = 0, kPerhaps = 1, kInside = 3 };

// A triangle's body.  E: a bound of the new time above st; lowered when the
// body is certain to accept a smaller one.
__host__ __device__ __forceinline__ unsigned tri_may(float &E, float c1, float c2, const TriF &k, const SideFilter &t)
{
    const float u = -c1 * k.kx, v = (c1 - c2) * k.ky;
    const float al = fmaf(-k.ay, v, fmaf(-k.ax, u, 1.0f));
    const float dd = fmaf(u, u, v * v);
    const float sc = t.eps * fmaf(al, al, dd + 1.0f);
    const float q = fmaf(al, al, -(t.fg * dd));
    const float qp = fmaxf(q, 1e-20f);
    const float rs = filter_rsqrt(qp), S = qp * rs;
    const float z = fmaf(-t.faz, al, S) * t.fig;
    const float w = fmaf(-t.faz, z, al);
    const float nx = fmaf(k.ax, w, u), ny = fmaf(k.ay, w, v);
    const float late = fmaf(-E, t.fkz, z);                                      // later than the time
    const float diag = fmaf(nx, k.r1, -(ny * k.r2)), far = -fmaf(nx, k.s1, S * k.s2);  // beyond the far sides
    const float out = fmaxf(fmaxf(nx, ny), fmaxf(diag, far)), m = sc * rs;
    const bool never = fmaxf(out, late) > m || q < -0.04f * sc;
    const bool inside = out < -m && q > 0.04f * sc && z > m && v != 0.0f;  // v = 0: :132 is undecided
    if (inside) E = fminf(E, (z + m) * t.fhz);
    return never ? kNever : inside ? kInside : kPerhaps;
}

// An edge's body; ca, cb: c of its two sources.
__host__ __device__ __forceinline__ unsigned edge_may(float &E, float ca, float cb, const EdgeF &k, const SideFilter &t)
{
    const float u = (ca - cb) * k.k, b = 0.25f * ca * k.k;
    const float c0 = fmaf(-k.ax, u, 1.0f);
    const float uu = u * u;
    const float sc = t.eps * fmaf(b, b, fmaf(c0, c0, uu + 1.0f));
    const float q = fmaf(c0, c0, -(k.ga * uu));
    const float qp = fmaxf(q, 1e-20f);
    const float rs = filter_rsqrt(qp), S = qp * rs;
    const float z = fmaf(-k.az, c0, S) * k.iga;
    const float m = sc * rs, mk = m * k.ka;
    const float late = fmaf(-(E + ca), k.kz, z);
    const float w = fmaf(-k.az, z, c0);
    const float nx = fmaf(k.fx, w, u), nz = fmaf(k.fz, w, z);
    const float far = fmaf(fabsf(nx), k.s1, -(fabsf(nz) * k.s2));     // |xe| > dxx
    const float same = fmaxf(fminf(nx, nz), -fmaxf(nx, nz));          // > 0: one sign, xe < 0
    const float out = fmaxf(far, same);
    const bool never = late > m || out > mk || q < -0.04f * sc;
    const bool inside = out < -mk && q > 0.04f * sc && z > m;
    return never ? kNever : inside ? kInside : kPerhaps;
}

// The calls that could lower a point's time after its 1-D candidate, as a bit
// mask; c: float(st - s_r) of the rim, E: float(tn - st).
__host__ __device__ __forceinline__ unsigned gate_mask(const float c[8], float E, const SideFilter &t)
{
    float gB[24];
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        const float4 b = reinterpret_cast<const float4 *>(t.gB)[i];
        gB[4 * i] = b.x;
        gB[4 * i + 1] = b.y;
        gB[4 * i + 2] = b.z;
        gB[4 * i + 3] = b.w;
    }
    const float Eu = fmaf(fabsf(E), 4e-7f, E);
    const float m01 = fmaxf(c[0], c[1]), m12 = fmaxf(c[1], c[2]), m23 = fmaxf(c[2], c[3]), m34 = fmaxf(c[3], c[4]),
                m45 = fmaxf(c[4], c[5]), m56 = fmaxf(c[5], c[6]), m67 = fmaxf(c[6], c[7]), m70 = fmaxf(c[7], c[0]);
    const float X[8] = {m01, m70, m45, m34, m56, m67, m12, m23};  // per triangle, the larger of its rim points
    // the sign bits of threshold - (time - smallest source); four independent
    // chains of shifts
    unsigned spokes = 0, nests = 0, tris = 0, up2 = 0, spoke = 0;
    constexpr int S1[8] = {0, 0, 4, 4, 6, 6, 2, 2}, S2[8] = {1, 7, 5, 3, 5, 7, 1, 3};
#pragma unroll
    for (int k = 7; k >= 0; --k) {
        tris = push_sign(tris, gB[k] - (Eu + fmaxf(X[k], 0.0f)));
        nests = push_sign(nests, gB[8 + k] - (Eu + X[k]));
        spokes = push_sign(spokes, gB[16 + k] - (Eu + fmaxf(c[k], 0.0f)));
        // fixed early returns: bit k of up2: s2 > s1 (per triangle), of spoke: s_r > st
        spoke = push_sign(spoke, c[k]);
        up2 = push_sign(up2, c[S2[k]] - c[S1[k]]);
    }
    // bit k of up1: s1 > st
    const unsigned up1 = (spoke & 1u) * 0x03u | ((spoke >> 4) & 1u) * 0x0cu | ((spoke >> 6) & 1u) * 0x30u |
                         ((spoke >> 2) & 1u) * 0xc0u;
    const unsigned gone = (t.m_e1 & up1) | (t.m_e2 & up2);
    return (tris & ~gone) | ((nests & ~(gone | (t.m_nest_early & up2))) << 8) | ((spokes & ~(t.m_edge_early & spoke)) << 16);
}

__host__ __device__ __forceinline__ int low_bit(unsigned m)
{
#ifdef __CUDA_ARCH__
    return __ffs((int)m) - 1;
#else
    return __builtin_ctz(m);
#endif
}

// New signed value of a target whose stored value is `told` from the nine
// previous-plane magnitudes `s` (rim order, st last).  Every lane of the warp
// calls it; a lane that is not `active` changes nothing.  sh, ch: scratch of
// nine doubles and nine floats of this point, `stride` elements apart (shared
// memory on the device: the walks index the sources by call); tab in shared
// memory too, since lanes read different calls' constants.
//
// The warp walks the union of its lanes' gated calls with the float filter,
// and each lane notes the bodies that it needs; then every lane runs its own
// list, so a warp runs as many FP64 bodies as its longest lane's list, not as
// the lanes' union.
__host__ __device__ __forceinline__ double point_update_fan(bool active, double told, const double (&s)[9],
                                                            const DirTable &tab, double *sh, float *ch, int stride)
{
    const double st = s[8];
    double tn = fabs(told);
    const SideTable &t = tab.side[told < 0 ? 1 : 0];
    const SideFilter &f = t.flt;
    float c[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        c[r] = (float)(st - s[r]);
        sh[r * stride] = s[r];
        ch[r * stride] = c[r];
    }
    sh[8 * stride] = st;
    ch[8 * stride] = 0.0f;
    if (st < tn && f.d1_ok) tn = kmin(tn, st + f.K1);
    float E = (float)(tn - st);
    const bool odd = !(fabsf(E) < 3e38f) || f.every;  // a time infinite or beyond float, or a NaN: gate nothing
    const float mx = fmaxf(fmaxf(fmaxf(fmaxf(c[0], c[1]), fmaxf(c[2], c[3])), fmaxf(fmaxf(c[4], c[5]), fmaxf(c[6], c[7]))),
                           0.0f);
    if (lanes_any(active && (odd || fmaf(fabsf(E), 4e-7f, E) + mx > f.outer))) {
        unsigned mask = gate_mask(c, E, f);
        if (odd) mask = 0xffffffu;
        // the reference's early exit (:231), on the sources it names (not xnt
        // and ynt): a gate of its own, so judged in FP64 where float is unsure
        // (NaN where one of them is NaN)
        const float lead = E + max_nan(max_nan(max_nan(f.named[0] ? c[4] : c[0], f.named[1] == 2 ? c[2] : c[6]),
                                               max_nan(c[1], c[7])),
                                       max_nan(c[5], c[3]));
        const float unsure = 4e-7f * fabsf(E);
        if (tn < st && mask && !(lead > unsure)) {
            if (lead < -unsure || (tn < kmin(sh[f.named[0] * stride], sh[f.named[1] * stride]) &&
                                   tn < kmin(sh[1 * stride], sh[7 * stride]) &&
                                   tn < kmin(sh[5 * stride], sh[3 * stride])))
                mask = 0;
        }
        if (!active) mask = 0;
        // The filter, a triangle and an edge at a time (two chains to overlap).
        unsigned need = 0, in = 0;  // bodies to run, and those with their footpoint known inside
        float Eb = odd ? E : fmaf(fabsf(E), 1e-6f, E);  // bound of the new time above st
        const unsigned all = lanes_or(mask);
        for (unsigned wt = all & 0xffu, we = all >> 8; wt | we; wt &= wt - 1, we &= we - 1) {
            const int k = wt ? low_bit(wt) : 0, j = we ? low_bit(we) : 0;
            const int i1 = (kTriS1 >> (4 * k)) & 15, i2 = (kTriS2 >> (4 * k)) & 15;
            const int ia = (j < 8) ? (int)((kTriS1 >> (4 * j)) & 15) : 8;
            const int ib = (j < 8) ? (int)((kTriS2 >> (4 * j)) & 15) : j - 8;
            const float ca = ch[ia * stride], cb = ch[ib * stride];
            const EdgeF ef = load_consts(f.ef[j]);
            const TriF tf = load_consts(f.tri[k]);
            const bool fall = ((mask >> (8 + j)) & 1u) && (odd || fmaf(fabsf(Eb), 4e-7f, Eb) + cb > ef.K);
            float Ee = Eb, Et = ((mask >> k) & 1u) ? Eb : -HUGE_VALF;
            const unsigned ve = edge_may(Ee, ca, cb, ef, f);
            const unsigned vt = tri_may(Et, ch[i1 * stride], ch[i2 * stride], tf, f);
            need |= ((vt & 1u) << k) | ((ve & 1u) << (8 + j));
            in |= ((vt >> 1) << k) | ((ve >> 1) << (8 + j));
            if ((mask >> k) & 1u) Eb = fminf(Eb, Et);
            if (fall) {  // the edge's fall-back, :99-113
                const SurfK &sk = t.surf[f.surf_at[j & 7]];
                const EdgeK &e = (j < 8) ? sk.nest : t.edge[f.edge_at[j & 7]];
                const double sa = sh[ia * stride], sb = sh[ib * stride], v = sb + e.K;
                const bool closed = (j < 8) ? nest_closed(st, sa, sb, sk) : ((e.early != 0) & (sb > st));
                if ((e.fb_ok != 0) & !closed & (tn > sb) & (v < tn)) {
                    tn = v;
                    const float En = (float)(tn - st);
                    Eb = fminf(Eb, fmaf(fabsf(En), 1e-6f, En));
                }
            }
        }
        if (odd) need = mask;
        need &= mask;
        while (lanes_any((need & 0xffu) != 0)) {
            if (need & 0xffu) {
                const int k = low_bit(need);
                need &= need - 1;
                const double s1 = sh[((kTriS1 >> (4 * k)) & 15) * stride], s2 = sh[((kTriS2 >> (4 * k)) & 15) * stride];
                const SurfK &sk = t.surf[f.surf_at[k]];
                if (!surf_closed(st, s1, s2, sk)) surf_body(tn, st, s1, s2, sk, t, (in >> k) & 1u);
            }
        }
        while (lanes_any(need != 0)) {
            if (need) {
                const int k = low_bit(need) - 8;
                need &= need - 1;
                const int ia = (k < 8) ? (int)((kTriS1 >> (4 * k)) & 15) : 8;
                const int ib = (k < 8) ? (int)((kTriS2 >> (4 * k)) & 15) : k - 8;
                const double sa = sh[ia * stride], sb = sh[ib * stride];
                const SurfK &sk = t.surf[f.surf_at[k & 7]];
                const EdgeK &e = (k < 8) ? sk.nest : t.edge[f.edge_at[k & 7]];
                const bool closed = (k < 8) ? nest_closed(st, sa, sb, sk) : ((e.early != 0) & (sb > st));
                if (!closed) edge_body(tn, sa, sb, e, t.F, (in >> (8 + k)) & 1u);
            }
        }
    }
    return ((told > 0) ? 1.0 : -1.0) * tn;
}

// A direction's table into shared memory, by all `n` threads.
__device__ __forceinline__ void copy_table(DirTable &dst, const DirTable &tab, int tid, int n)
{
    static_assert(sizeof(DirTable) % 16 == 0, "copied in 16-byte words");
    for (int i = tid; i < (int)(sizeof(DirTable) / 16); i += n)
        reinterpret_cast<int4 *>(&dst)[i] = reinterpret_cast<const int4 *>(&tab)[i];
}

// The same for one point with its sources named as in the reference
// (:195-204); host code only (one point is not a warp).
inline double point_update_fast(double told, double st, double xt, double yt, double xnt, double ynt, double txy,
                                double txm, double tym, double txnyn, const DirTable *tab)
{
    const double s[9] = {xt, txy, yt, tym, xnt, txnyn, ynt, txm, st};
    double sh[9];
    float ch[9];
    return point_update_fan(true, told, s, *tab, sh, ch, 1);
}

// ---------------------------------------------------------------------------
// Candidate values for the compacted kernel.  Each function returns the
// smallest candidate its reference call would accept when entered with the
// current time `th` -- or +infinity -- instead of updating a running time.
// Every value returned is below th, so folding them with min gives the same
// result as the reference's sequence of calls (see the header comment).  The
// caller has already applied the call's entry gates.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double edge_cand(double th, double s0, double s1, const EdgeK &k, double F)
{
    double best = th;
    const double d = div_by_const(s1 - s0, k.hx, k.rhx);
    double c = (1.0 - d * k.ax);
    double q = k.g * (c * c - d * d * k.ga);
    if (0.0 < q) {
        c = div_by_const(-k.az * c + sqrt(q), k.ga, k.rga);
        q = s0 + k.hz * c;
        if (q < best && q > kmin(s0, s1)) {
            const double g = sqrt(div_by_const((d * d + c * c) * F * F, k.g, k.rg));
            const double xe = -k.hz * (d + k.ax * g) / (c + k.az * g);
            if (0.0 < xe && xe < k.hx) best = q;
        }
    }
    if (best > s1 && k.fb_ok) best = kmin(best, s1 + k.K);
    return best;
}

__device__ __forceinline__ double surf_cand(double th, double s0, double s1, double s2, const SurfK &k,
                                            const SideTable &t)
{
    double best = th;
    const double dx = div_by_const(s1 - s0, k.hx, k.rhx);
    const double dy = div_by_const(s2 - s1, k.hy, k.rhy);
    double dd = dx * dx + dy * dy;
    double al = 1.0 - k.ax * dx - k.ay * dy;
    double q = al * al - dd * t.g;
    if (q > 0.0) {
        al = div_by_const(-t.az * al + t.F * sqrt(q), t.g, t.rg);
        const double g = s0 + t.hz * al;
        if (g < best && g > kmin(kmin(s0, s1), s2)) {
            q = sqrt(dd + al * al);
            dd = -t.hz / (t.F * al + t.az * q);
            const double xe = dd * (t.F * dx + k.ax * q);
            const double ye = dd * (t.F * dy + k.ay * q);
            if (0.0 <= kmin(xe, ye) && ye * k.hx <= xe * k.hy && xe <= k.hx) best = g;
        }
    }
    return best;
}
#endif  // __CUDACC__

}  // namespace fold3d
