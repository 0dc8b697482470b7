// fold3d_wavefront.cu -- the WAVEFRONT engine: one persistent launch per
// directional pass, tile dataflow between consecutive planes, and tiles
// skipped when their inputs did not change.
//
// Work items are (plane step p, tile t) pairs of a pass, tiles being 32 points
// by a few rows of a plane, numbered plane-major.  A worker -- a warp in the
// drift medium's passes, a CTA in the elliptical medium's -- claims the next
// item from an atomic counter.  Item (p, t) reads the source plane written by
// step p-1 only within t's 1-point halo, i.e. from the 3 x 3 tiles around t,
// so it waits for exactly those items (their completion flags), not for the
// whole previous plane: consecutive planes overlap and no plane-wide barrier
// or launch separates them.  Items are claimed in increasing order and a worker
// processes its claims in order, so the lowest unfinished item is always held
// by a running worker that is at it; the waits always end.  They are bounded
// anyway: after a time limit the worker raises the status word and every
// worker leaves (FOLD3D_ERR_TIMEOUT).
//
// Skipping.  A point update is min(T_old, M(nine source values, side)) (see
// fold3d_fast.cuh), so re-evaluating a tile whose source neighbourhood has
// not changed since its previous evaluation in the same direction leaves
// every target value unchanged, bit for bit.  Each orientation (plane normal
// x, y or z) keeps a map with, per plane and tile, the last pass in which any
// of its points changed; a pass writes the maps of all three orientations for
// the points it changes.  From the second sweep of a solve on, item (p, t)
// of pass e is skipped when no tile of the 3 x 3 neighbourhood of its source
// plane changed in passes e-5 .. e (the previous evaluation of that tile in
// this direction was in pass e-6, after the source plane's update of that
// pass).
//
// The change marks of earlier passes are final when a pass starts; whether
// step p-1 of the current pass changed the source plane comes with its
// completion flags, which hold (pass << 1) | changed.
//
// Synchronisation: an item is published with a barrier of its worker's threads
// (__syncwarp or __syncthreads) and a gpu-scope release of the item's flag; nine
// lanes of the waiting worker poll the nine neighbour flags in parallel with
// acquire loads before a barrier.  Field values written inside the launch are
// read with L2-cached loads (ld.global.cg), never through the non-coherent
// read-only path.
#include <cstring>

#include "fold3d_ellip.cuh"
#include "fold3d_fast.cuh"
#include "fold3d_internal.h"
#include "fold3d_sync.cuh"

namespace fold3d {

namespace {

__device__ __forceinline__ double ld_cg(const double *p) { return __ldcg(p); }
__device__ __forceinline__ float ld_cg(const float *p) { return __ldcg(p); }

// Whether a stored value changes (bit patterns, so -0 vs +0 counts).
__device__ __forceinline__ bool bits_differ(double a, double b) { return __double_as_longlong(a) != __double_as_longlong(b); }
__device__ __forceinline__ bool bits_differ(float a, float b) { return __float_as_int(a) != __float_as_int(b); }

}  // namespace

constexpr int kWaveThreads = 128;           // the drift medium's CTAs: four warps
constexpr int kEllipThreads = 32 * kWaveTV;  // the elliptical medium's: a warp per row of the tile

template <class R> constexpr int wave_min_blocks()
{
    return (sizeof(R) == 8 ? FOLD3D_WAVE_MINB_ELLIP : FOLD3D_WAVE_MINB_ELLIP_F32) * 4 / kWaveTV;
}

// A lane's point (u, v) of the target plane src + sg: update it from the source
// plane and store it; whether it changed.  All lanes of the warp call this
// together; points outside the plane are left out.  sh: the thread's scratch
// (ell_update_fan), `stride` doubles apart; unused by float fields.
template <class R>
__device__ __forceinline__ bool ellip_point(R *__restrict__ T, const WaveArgs &a, const EllipParam &tab, int src, int u,
                                            int v, double *sh, int stride, double &dmax, unsigned &evaluated)
{
    const PlaneGeom &g = a.pg;
    const bool active = u <= g.nu && v <= g.nv;
    const long long s = (long long)src * g.s_nrm + (long long)u * g.su + (long long)v * g.sv, d = s + g.sn;
    R told = R(0), tnew = R(0), fan[9] = {};
    int win = -1;
    if constexpr (sizeof(R) == 8) {
        double m[6] = {};
        if (active) {
            ell_values(tab.med, tab.dir, d, m);
            told = ld_cg(T + d);
            fan[8] = fabs(ld_cg(T + s));
#pragma unroll
            for (int r = 0; r < 8; ++r) fan[r] = fabs(ld_cg(T + s + ell_ri(r) * g.sx + ell_rj(r) * g.sy));
        }
        tnew = ell_update_fan(active, told, fan, m, tab.med.kind, tab.dir, sh, stride, win);
        if (!active) return false;
    } else {
        if (!active) return false;
        told = ld_cg(T + d);
        fan[8] = fabs(ld_cg(T + s));
        R nb[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) nb[r] = fabs(ld_cg(T + s + ell_ri(r) * g.sx + ell_rj(r) * g.sy));
        tnew = point_update_ellip(told, fan[8], nb, ell_local<R>(tab.med, tab.dir, d), win);
    }
    ++evaluated;
    if (!bits_differ(tnew, told)) return false;
    if (a.winners) a.winners[d] = (win < 0) ? (unsigned char)kNoWinner : (unsigned char)(a.dir * kEllipCands + win);
    T[d] = tnew;
    dmax = fmax(dmax, (double)fabs(tnew - told));
    return true;
}

// Marks the tile of changed point (u, v) of plane tgt in an in-plane
// orientation: Q = 1, planes u of normal axis ua; Q = 2, planes v of va.
template <int Q, int TV>
__device__ __forceinline__ void wave_mark(const WaveArgs &a, int u, int v, int tgt)
{
    const int other = (Q == 1) ? v : u;
    const bool first = a.nrm < ((Q == 1) ? a.va : a.ua);  // the pass's normal is that orientation's faster axis
    const int cu = first ? tgt : other, cv = first ? other : tgt;
    a.mod[Q][(long long)(Q == 1 ? u : v) * a.mod_ntiles[Q] + ((cv - 1) / TV) * a.mod_ntu[Q] + ((cu - 1) >> 5)] = a.epoch;
}

// x / n and the remainder r for 0 <= x, n > 0; inv = 1/n rounded.  The product
// is off by at most one for quotients below 2^22, and corrected from the
// remainder (in as many steps as it takes beyond that).
__device__ __forceinline__ int wave_div(int x, int n, float inv, int &r)
{
    int q = (int)((float)x * inv);
    r = x - q * n;
    while (r < 0) {
        --q;
        r += n;
    }
    while (r >= n) {
        ++q;
        r -= n;
    }
    return q;
}

// One work item (step p, tile t) of one grid, for all threads of the CTA:
// wait for the 3 x 3 tiles of step p-1, then skip or update the tile, then
// publish its flag.  Adds each changed point's |dT| into dmax and the
// evaluated points into evaluated.  Returns false if a wait gave up (the
// item is then left unpublished and the caller must leave).
template <class R, int TV>
__device__ __forceinline__ bool wave_item(R *__restrict__ T, const WaveArgs &a,
                                          const EllipParam &tab, int item, double *sh,
                                          double &dmax, unsigned &evaluated)
{
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const PlaneGeom &g = a.pg;
    const int ntiles = a.ntu * a.ntv;
    const unsigned want = a.epoch << 1;  // flags hold (pass << 1) | changed
    const bool may_skip = a.epoch >= a.skip_from;
    const int p = item / ntiles, t = item - p * ntiles;
    const int tu = t % a.ntu, tv = t / a.ntu;
    const int src = a.first_src + p * a.sg;
    const int tgt = src + a.sg;

    // Threads 0..8 each watch one tile of the 3 x 3 neighbourhood: its change
    // mark from earlier passes, and its step p-1 flag (which also says whether
    // that item changed the source plane).
    int timed_out = 0, recent = 0;
    if (tid < 9) {
        const int nu = tu + tid % 3 - 1, nv = tv + tid / 3 - 1;
        if (nu >= 0 && nu < a.ntu && nv >= 0 && nv < a.ntv) {
            const int nt = nv * a.ntu + nu;
            if (may_skip) recent = (__ldcg(a.mod[0] + (long long)src * ntiles + nt) + 5u >= a.epoch);
            if (p > 0) {
                const unsigned f = wait_flag(a.flags + (((long long)(p - 1) * ntiles + nt) << a.fshift), want, a.status, a.timeout_ns);
                timed_out = f == 0;
                recent |= (int)(f & 1u);
            }
        }
    }
    if (__syncthreads_or(timed_out)) return false;
    const int skip = may_skip && !__syncthreads_or(recent);

    int changed = 0;
    if (!skip) {
        const int u = tu * 32 + lane + 1;
        const int v = tv * TV + warp + 1;
        if (ellip_point<R>(T, a, tab, src, u, v, sh, 32 * TV, dmax, evaluated)) {
            changed = 1;
            wave_mark<1, TV>(a, u, v, tgt);
            wave_mark<2, TV>(a, u, v, tgt);
        }
        changed = __syncthreads_or(changed);
        if (changed && tid == 0) a.mod[0][(long long)tgt * ntiles + t] = a.epoch;
    }
    // publish: the barrier makes every thread's stores precede thread 0's
    // release store, which orders them (cumulatively) before the flag
    __syncthreads();
    if (tid == 0) st_release(a.flags + ((long long)item << a.fshift), want | (unsigned)changed);
    return true;
}

// Block-wide maximum of d into *out (IEEE bits) and sum of e into *sum.
template <int TV>
__device__ __forceinline__ void wave_flush(double d, unsigned long long e, unsigned long long *out,
                                           unsigned long long *sum)
{
    __shared__ double wmax[TV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d = fmax(d, __shfl_xor_sync(0xffffffffu, d, o));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (lane == 0) {
        wmax[warp] = d;
        if (e) atomicAdd(sum, e);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0;
        for (int w = 0; w < TV; ++w) m = fmax(m, wmax[w]);
        if (m > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
    }
    __syncthreads();
}

// The items of a pass whose warps work alone: every warp claims and publishes
// whole items of 32 x TV points, each with one fence; no warp waits at a CTA
// barrier for another's rows.  rows(src, u, v0, last, active, prefetch) updates
// the lane's points (u, v0 .. v0 + last - 1) of a tile (lanes that are not
// active only keep company), calls prefetch() once its first loads are under
// way, and returns the changed ones of the lane's points as bits.  The change
// marks of the other orientations (32 scattered stores) come after the item is
// published, for the fence would wait for them.
template <int TV, class Rows> __device__ __forceinline__ void warp_items(const WaveArgs &a, Rows rows)
{
    const int lane = threadIdx.x & 31;
    const int ntiles = a.ntu * a.ntv;
    const unsigned total = (unsigned)(a.steps * ntiles);
    const float inv_tiles = 1.0f / (float)ntiles, inv_ntu = 1.0f / (float)a.ntu;
    const unsigned want = a.epoch << 1;  // flags hold (pass << 1) | changed
    const bool may_skip = a.epoch >= a.skip_from;
    // Lanes 0..8 each watch one tile of an item's 3 x 3 neighbourhood: its
    // change mark from earlier passes, and its step p-1 flag (which also says
    // whether that item changed the source plane).  watch() gives the lane's
    // flag, or NULL where there is nothing to wait for.
    auto watch = [&](unsigned item, int &p, int &t, int &tu, int &tv, bool &recent) -> const unsigned * {
        p = wave_div((int)item, ntiles, inv_tiles, t);
        tv = wave_div(t, a.ntu, inv_ntu, tu);
        const int nu = tu + lane % 3 - 1, nv = tv + lane / 3 - 1, nt = nv * a.ntu + nu;
        const bool in = lane < 9 && nu >= 0 && nu < a.ntu && nv >= 0 && nv < a.ntv;
        recent = in && may_skip && __ldcg(a.mod[0] + (long long)(a.first_src + p * a.sg) * ntiles + nt) + 5u >= a.epoch;
        return (in && p > 0) ? a.flags + (((long long)(p - 1) * ntiles + nt) << a.fshift) : nullptr;
    };
    // The warp holds two claimed items: the flags of the second are read while
    // the first is worked on, and the fence that publishes the first also
    // orders that read before the second's loads (with the warp barrier after it,
    // which carries the nine watching lanes' order to all lanes).
    unsigned ahead = 0;
    if (lane == 0) ahead = atomicAdd(a.work, 1u);
    unsigned item = __shfl_sync(0xffffffffu, ahead, 0);
    if (lane == 0) ahead = atomicAdd(a.work, 1u);
    int p = 0, t = 0, tu = 0, tv = 0;
    bool recent = false;
    const unsigned *fl = item < total ? watch(item, p, t, tu, tv, recent) : nullptr;
    unsigned f = 0;
    while (item < total) {
        bool gave_up = false;
        if (fl && f < want) {
            f = wait_flag(fl, want, a.status, a.timeout_ns);
            gave_up = f == 0;
        }
        recent |= fl && (f & 1u);
        if (__any_sync(0xffffffffu, gave_up)) break;
        const bool skip = may_skip && !__any_sync(0xffffffffu, recent);
        __syncwarp();  // the watching lanes' acquire comes before every lane's loads (votes order no memory)
        const unsigned next = __shfl_sync(0xffffffffu, ahead, 0);
        if (lane == 0) ahead = atomicAdd(a.work, 1u);
        const int src = a.first_src + p * a.sg, tgt = src + a.sg, u = tu * 32 + lane + 1, v0 = tv * TV + 1;
        const int t0 = t;
        auto prefetch = [&] {
            if (next < total) {
                fl = watch(next, p, t, tu, tv, recent);
                f = fl ? ld_relaxed(fl) : 0u;
            }
        };
        unsigned changed = 0, any = 0;
        if (!skip) {
            changed = rows(src, u, v0, min(TV, a.pg.nv - v0 + 1), u <= a.pg.nu, prefetch);
            any = __any_sync(0xffffffffu, changed != 0) ? 1u : 0u;
        } else {
            prefetch();
        }
        __syncwarp();
        fence_acq_rel();
        if (lane == 0) st_relaxed(a.flags + ((long long)item << a.fshift), want | any);
        __syncwarp();
        if (changed) {
            wave_mark<1, TV>(a, u, v0, tgt);
#pragma unroll
            for (int r = 0; r < TV; ++r)
                if ((changed >> r) & 1u) wave_mark<2, TV>(a, u, v0 + r, tgt);
        }
        if (any && lane == 0) a.mod[0][(long long)tgt * ntiles + t0] = a.epoch;
        item = next;
    }
}

// A pass of the drift medium.  Every warp claims and processes whole items
// of 32 x TV points on its own, the tile's rows one after another, and
// publishes them with one fence; no warp waits at a CTA barrier for another's
// rows.  A row's nine source values are the last row's shifted by one, with
// three new ones read while the last row is worked on.
//
// What bounds it: the latency of a point's update and of the exchange between
// plane steps, not bytes (10 DRAM bytes per update) and not issue alone (59% of the
// cycles at 1280^2 planes).  Per row of 32 points it runs 450 to 940 warp
// instructions (930 to 1360 before the float filter).  In a settled field (no tile skipped)
// a plane step takes 6.6, 9.6, 12.6 and 61 us at 64, 256, 512 and 1280 points
// per axis, of which the claims, waits and publishing alone 2.5, 4.0, 5.7 and 9.
// ms before (a CTA per 32 x 4 tile, FP64 gates) and now: 64^3, 8 sweeps 36.8 ->
// 19.4; 512^3, 8 sweeps 453 -> 350; 1280^3, 2 sweeps 1518 -> 1135.
template <int TV>
__global__ void __launch_bounds__(kWaveThreads, FOLD3D_WAVE_MINB_DRIFT)
    drift_pass_kernel(double *__restrict__ T, WaveArgs a, const __grid_constant__ DirTable tab)
{
    __shared__ DirTable s_tab;
    __shared__ double s_fan[9 * kWaveThreads];
    __shared__ float s_dif[9 * kWaveThreads];
    copy_table(s_tab, tab, threadIdx.x, kWaveThreads);
    __syncthreads();
    double dmax = 0.0;
    unsigned evaluated = 0;
    warp_items<TV>(a, [&](int src, int u, int v0, int last, bool active, auto prefetch) -> unsigned {
        const PlaneGeom &g = a.pg;
        const double *s = T + ((long long)src * g.s_nrm + (long long)u * g.su + (long long)v0 * g.sv);
        // source rows v0 - 1 .. v0 + 1, and the target
        double w[3][3] = {}, told = 0.0;
        if (active) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) w[i][j] = fabs(ld_cg(s + (i - 1) * g.sv + (j - 1) * g.su));
            told = ld_cg(s + g.sn);
        }
        prefetch();
        unsigned any = 0;
#pragma unroll 1
        for (int r = 0; r < last; ++r, s += g.sv) {
            double w3[3] = {}, told3 = 0.0;  // the next row's new sources and target
            if (TV > 1 && active && r + 1 < last) {
#pragma unroll
                for (int j = 0; j < 3; ++j) w3[j] = fabs(ld_cg(s + 2 * g.sv + (j - 1) * g.su));
                told3 = ld_cg(s + g.sv + g.sn);
            }
            const double fan[9] = {w[1][2], w[2][2], w[2][1], w[2][0], w[1][0], w[0][0], w[0][1], w[0][2], w[1][1]};
            const double tnew =
                point_update_fan(active, told, fan, s_tab, &s_fan[threadIdx.x], &s_dif[threadIdx.x], kWaveThreads);
            const bool changed = active && bits_differ(tnew, told);
            evaluated += active;
            if (changed) {
                const_cast<double *>(s)[g.sn] = tnew;
                dmax = fmax(dmax, fabs(tnew - told));
            }
            any |= (unsigned)changed << r;
            if (TV > 1) {
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    w[0][j] = w[1][j];
                    w[1][j] = w[2][j];
                    w[2][j] = w3[j];
                }
                told = told3;
            }
        }
        return any;
    });
    __syncthreads();
    wave_flush<kWaveThreads / 32>(dmax, evaluated, a.maxd, a.evaluated);
}

// A pass of the elliptical medium: the warps of a CTA share each item's rows.
// (Its update is 700 instructions of mostly straight code; warps that run it
// together fetch it together.  With items of their own, as in the drift
// medium's passes, 512^3 to 1e-10 took 437 ms instead of 312.)
//
// wave_pass_kernel is for planes of kLargePlaneTiles tiles or more, where a CTA
// has several items of a step: two barriers per item.  Before the first, warp 0
// watches the item's dependencies and the last warp claims the next item; the
// rows run between them; after the second, warp 1 publishes the item while the
// others go on.  On smaller planes, and for float fields, the plane-to-plane
// chain binds and wave_item_kernel is faster, where thread 0 publishes before
// anything of the next item begins (ms; two barriers, this, one source each:
// 128^3 to 1e-10 12.7, 12.2; 512^3 312, 339; float32 380x319x257 72.4, 69.8).  What bounds
// both is the chain from step to step, and on x-normal planes loads of which
// every lane's is a sector of its own (2 to 3 times a k pass at 512^3).
template <class R>
__global__ void __launch_bounds__(kEllipThreads, wave_min_blocks<R>())
    wave_item_kernel(R *__restrict__ T, WaveArgs a, const __grid_constant__ EllipParam tab)
{
    __shared__ int s_next;
    __shared__ double s_fan[sizeof(R) == 8 ? 9 * kEllipThreads : 1];
    const long long total = (long long)a.steps * a.ntu * a.ntv;
    double dmax = 0.0;
    unsigned evaluated = 0;
    if (threadIdx.x == 0) {
        const unsigned w = atomicAdd(a.work, 1u);
        s_next = (w < total) ? (int)w : -1;
    }
    __syncthreads();
    for (;;) {
        const int item = s_next;
        if (item < 0) break;
        __syncthreads();  // every thread has read s_next
        if (threadIdx.x == 0) {  // claim the next item now; it is processed after this one
            const unsigned w = atomicAdd(a.work, 1u);
            s_next = (w < total) ? (int)w : -1;
        }
        if (!wave_item<R, kWaveTV>(T, a, tab, item, s_fan + threadIdx.x, dmax, evaluated)) break;
    }
    wave_flush<kWaveTV>(dmax, evaluated, a.maxd, a.evaluated);
}

__global__ void __launch_bounds__(kEllipThreads, wave_min_blocks<double>())
    wave_pass_kernel(double *__restrict__ T, WaveArgs a, const __grid_constant__ EllipParam tab)
{
    constexpr int TV = kWaveTV, kWarps = TV, kPublisher = TV > 1 ? 32 : 0;  // a warp other than 0, where there is one
    __shared__ int s_item[2];           // the CTA's items, by parity; -1 for none
    __shared__ int s_state;             // 0 update, 1 skip, 2 a wait gave up
    __shared__ double s_fan[9 * kEllipThreads];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ntiles = a.ntu * a.ntv;
    const unsigned total = (unsigned)(a.steps * ntiles);
    const float inv_tiles = 1.0f / (float)ntiles, inv_ntu = 1.0f / (float)a.ntu;
    const unsigned want = a.epoch << 1;  // flags hold (pass << 1) | changed
    const bool may_skip = a.epoch >= a.skip_from;
    double dmax = 0.0;
    unsigned evaluated = 0;
    if (threadIdx.x == 0) {
        const unsigned w = atomicAdd(a.work, 1u);
        s_item[0] = (w < total) ? (int)w : -1;
    }
    __syncthreads();
    for (int q = 0;; ++q) {
        const int slot = q & 1, item = s_item[slot];
        if (item < 0) break;
        int t, tu;
        const int p = wave_div(item, ntiles, inv_tiles, t), tv = wave_div(t, a.ntu, inv_ntu, tu);
        const int src = a.first_src + p * a.sg, tgt = src + a.sg, u = tu * 32 + lane + 1;
        if (warp == 0) {
            // lanes 0..8 each watch one tile of the 3 x 3 neighbourhood: its
            // change mark from earlier passes, and its step p-1 flag (which
            // also says whether that item changed the source plane)
            const int nu = tu + lane % 3 - 1, nv = tv + lane / 3 - 1;
            bool gave_up = false, recent = false;
            if (lane < 9 && nu >= 0 && nu < a.ntu && nv >= 0 && nv < a.ntv) {
                const int nt = nv * a.ntu + nu;
                if (may_skip) recent = __ldcg(a.mod[0] + (long long)src * ntiles + nt) + 5u >= a.epoch;
                if (p > 0) {
                    const unsigned f =
                        wait_flag(a.flags + (((long long)(p - 1) * ntiles + nt) << a.fshift), want, a.status, a.timeout_ns);
                    gave_up = f == 0;
                    recent |= f & 1u;
                }
            }
            gave_up = __any_sync(0xffffffffu, gave_up);
            recent = __any_sync(0xffffffffu, recent);
            if (lane == 0) s_state = gave_up ? 2 : (may_skip && !recent) ? 1 : 0;
        }
        unsigned claim = 0;  // the next item; looked at only after this one's rows
        const bool claims = threadIdx.x == 32 * (kWarps - 1);
        if (claims) claim = atomicAdd(a.work, 1u);
        __syncthreads();
        const int state = s_state;
        if (state == 2) break;
        bool changed = false;
        if (state == 0)
            changed = ellip_point<double>(T, a, tab, src, u, tv * TV + warp + 1, s_fan + threadIdx.x, kEllipThreads,
                                          dmax, evaluated);
        if (changed) {
            wave_mark<1, TV>(a, u, tv * TV + warp + 1, tgt);
            wave_mark<2, TV>(a, u, tv * TV + warp + 1, tgt);
        }
        if (claims) s_item[slot ^ 1] = (claim < total) ? (int)claim : -1;
        const bool any = __syncthreads_or(changed);  // precedes the release: every thread's stores come before the flag
        if (threadIdx.x == kPublisher) {
            st_release(a.flags + ((long long)item << a.fshift), want | (any ? 1u : 0u));
            if (any) a.mod[0][(long long)tgt * ntiles + t] = a.epoch;
        }
    }
    __syncthreads();
    wave_flush<kWarps>(dmax, evaluated, a.maxd, a.evaluated);
}

// ---------------------------------------------------------------------------
// Batched passes: the items of one pass of many independent grids (the
// elliptical medium) in one launch.  Items are ordered step-major across the
// instances (step p of every instance that has one, then step p+1), the
// instances sorted by their number of steps, so that the active instances of
// a step are a prefix of the list; every item's predecessors (step p-1 of the
// same instance) come earlier in that order, and the launch's claimed items
// spread over many instances at once.
// ---------------------------------------------------------------------------
// Resident CTAs per SM the batched kernel is compiled for, by tile height: the
// option's warps, rounded up to whole CTAs.  FP64 at 8 rows gets 3 CTAs and 80
// registers per thread, at 2 and 4 rows 20 warps and 96; rounded down it had 16
// warps (ms at 8 rows, 2 and 3 CTAs: 24 instances of 96 to 200 points per axis
// 328, 299; 48 of 64 to 176 395, 341; at 4 rows 280 and 323).
template <class R, int TV> constexpr int batch_min_blocks()
{
    return ((sizeof(R) == 8 ? FOLD3D_WAVE_MINB_BATCH : FOLD3D_WAVE_MINB_BATCH_F32) * 4 + TV - 1) / TV;
}

template <class R, int TV>
__global__ void __launch_bounds__(32 * TV, batch_min_blocks<R, TV>()) batch_pass_kernel(BatchArgs b)
{
    // A CTA claims b.chunk consecutive items at a time, and the first
    // lanes of warp 0 locate them in parallel (two binary searches each over
    // the launch's tables): consecutive items mostly belong to one instance
    // (its tiles of a step come together), so the instance is staged once for
    // several items, and the searches' dependent loads are paid once per
    // chunk.  Claims stay in increasing order and a chunk's items run in
    // order, so the lowest unfinished item always runs and every wait ends.
    __shared__ int s_next;  // first item of the CTA's next chunk, -1 for none
    __shared__ int s_loc[kBatchChunk][2];
    __shared__ int s_n;     // items of the current chunk
    __shared__ int s_cur;   // the active slot staged in s_inst, -1 for none
    __shared__ BatchInst s_inst;
    __shared__ double s_fan[sizeof(R) == 8 ? 9 * 32 * TV : 1];
    const unsigned total = *b.total;
    if (threadIdx.x == 0) {
        const unsigned w = atomicAdd(b.work, (unsigned)b.chunk);
        s_next = (w < total) ? (int)w : -1;
        s_n = 0;
        s_cur = -1;
    }
    __syncthreads();
    // The instance stays staged, and its largest change and evaluated points
    // are flushed only when the CTA moves to another one.
    double dmax = 0.0;
    unsigned evaluated = 0;
    for (int q = 0;; ++q) {
        if (q == s_n) {  // the same for every thread
            const int c0 = s_next;
            if (c0 < 0) break;
            __syncthreads();  // every thread has read s_n and s_next
            if (threadIdx.x < 32) {
                const int n = (int)min((unsigned)b.chunk, total - (unsigned)c0);
                if ((int)threadIdx.x < n)
                    batch_locate(b.step_off, b.step_k, b.tile_pre, b.max_steps, c0 + (int)threadIdx.x,
                                 s_loc[threadIdx.x][0], s_loc[threadIdx.x][1]);
                if (threadIdx.x == 0) {
                    const unsigned w = atomicAdd(b.work, (unsigned)b.chunk);
                    s_next = (w < total) ? (int)w : -1;
                    s_n = n;
                }
            }
            __syncthreads();
            q = 0;
        }
        const int slot = s_loc[q][0];
        if (slot != s_cur) {  // the same for every thread
            if (s_cur >= 0) {
                wave_flush<TV>(dmax, evaluated, s_inst.a.maxd, s_inst.a.evaluated);
                dmax = 0.0;
                evaluated = 0;
            }
            const unsigned *src = reinterpret_cast<const unsigned *>(b.inst + b.act[slot]);
            unsigned *dst = reinterpret_cast<unsigned *>(&s_inst);
            for (int w = threadIdx.x; w < (int)(sizeof(BatchInst) / 4); w += blockDim.x) dst[w] = src[w];
            __syncthreads();
            if (threadIdx.x == 0) {  // the pass number is per launch, not per staged instance
                s_inst.a.epoch = *b.epoch_base + (unsigned)b.dir + 1u;
                s_inst.a.skip_from = b.skip_from;
                s_cur = slot;
            }
            __syncthreads();
        }
        if (!wave_item<R, TV>(static_cast<R *>(s_inst.T), s_inst.a, s_inst.p, s_loc[q][1],
                                            s_fan + threadIdx.x, dmax, evaluated))
            break;
    }
    if (s_cur >= 0) wave_flush<TV>(dmax, evaluated, s_inst.a.maxd, s_inst.a.evaluated);
}

// The batch's state after a sweep and the next sweep's tables (BatchCtl).
// One block: the instances are folded in parallel, then one thread per
// direction rebuilds that direction's tables (a few thousand steps).
__global__ void __launch_bounds__(256) batch_restage_kernel(BatchCtl c, int first)
{
    __shared__ int s_left;
    if (threadIdx.x == 0) s_left = 0;
    __syncthreads();
    if (first) {
        for (int i = threadIdx.x; i < c.n; i += blockDim.x) {
            c.active[i] = 1;
            c.sweeps[i] = 0;
            c.delta[i] = 0.0;
            c.maxd[i] = 0ull;
        }
        if (threadIdx.x == 0) {
            *c.epoch_base = c.epoch0;
            c.sweep[0] = 0;
            c.sweep[1] = c.n;
        }
    } else {
        int left = 0;
        for (int i = threadIdx.x; i < c.n; i += blockDim.x) {
            if (c.active[i]) {
                c.sweeps[i] += 1;
                const double d = __longlong_as_double((long long)c.maxd[i]);
                c.delta[i] = d;
                if (!c.fixed && d <= c.tol) c.active[i] = 0;
                else ++left;
            }
            c.maxd[i] = 0ull;
        }
        atomicAdd(&s_left, left);
    }
    __syncthreads();
    if (!first && threadIdx.x == 0) {
        *c.epoch_base += 6u;
        c.sweep[0] += 1;
        c.sweep[1] = s_left;
    }
    if (threadIdx.x < 6) c.total[threadIdx.x] = batch_tables(c.dir[threadIdx.x], c.active, c.n, c.max_steps);
    if (!first && threadIdx.x == 0) {
        const int more = (*(volatile const unsigned *)c.status == 0) && c.sweep[0] < c.max_sweeps && s_left > 0;
        cudaGraphSetConditional((cudaGraphConditionalHandle)c.cond, more ? 1u : 0u);
    }
}

cudaError_t launch_batch_restage(const BatchCtl &ctl, bool first, cudaStream_t s)
{
    batch_restage_kernel<<<1, 256, 0, s>>>(ctl, first ? 1 : 0);
    return cudaGetLastError();
}

template <int TV> static cudaError_t launch_batch_tv(const BatchArgs &b, bool f32, int grid, cudaStream_t s)
{
    if (f32) batch_pass_kernel<float, TV><<<grid, 32 * TV, 0, s>>>(b);
    else batch_pass_kernel<double, TV><<<grid, 32 * TV, 0, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_batch_pass(const BatchArgs &b, bool f32, int tv, int grid, cudaStream_t s)
{
    switch (tv) {
    case 2: return launch_batch_tv<2>(b, f32, grid, s);
    case 4: return launch_batch_tv<4>(b, f32, grid, s);
    case 8: return launch_batch_tv<8>(b, f32, grid, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int TV> static int batch_occupancy(bool f32)
{
    int n = 0;
    const cudaError_t e =
        f32 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_pass_kernel<float, TV>, 32 * TV, 0)
            : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_pass_kernel<double, TV>, 32 * TV, 0);
    if (e != cudaSuccess) return 1;
    return n > 0 ? n : 1;
}

int batch_blocks_per_sm(bool f32, int tv)
{
    return tv == 2 ? batch_occupancy<2>(f32) : tv == 8 ? batch_occupancy<8>(f32) : batch_occupancy<4>(f32);
}

cudaError_t launch_wave_pass(double *T, const WaveArgs &a, const DirTable &tab, int tv, int grid, cudaStream_t s)
{
    switch (tv) {
    case 1: drift_pass_kernel<1><<<grid, kWaveThreads, 0, s>>>(T, a, tab); break;
    case 2: drift_pass_kernel<2><<<grid, kWaveThreads, 0, s>>>(T, a, tab); break;
    case 4: drift_pass_kernel<4><<<grid, kWaveThreads, 0, s>>>(T, a, tab); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_wave_pass_ellip(void *T, bool f32, const WaveArgs &a, const EllipParam &p, int grid, cudaStream_t s,
                                   bool large)
{
    if (f32) wave_item_kernel<float><<<grid, kEllipThreads, 0, s>>>(static_cast<float *>(T), a, p);
    else if (large) wave_pass_kernel<<<grid, kEllipThreads, 0, s>>>(static_cast<double *>(T), a, p);
    else wave_item_kernel<double><<<grid, kEllipThreads, 0, s>>>(static_cast<double *>(T), a, p);
    return cudaGetLastError();
}

template <class K> static int occupancy(K kernel, int threads)
{
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0) != cudaSuccess) return 1;
    return n > 0 ? n : 1;
}

int wave_blocks_per_sm(bool f32, bool large)
{
    return f32     ? occupancy(wave_item_kernel<float>, kEllipThreads)
           : large ? occupancy(wave_pass_kernel, kEllipThreads)
                   : occupancy(wave_item_kernel<double>, kEllipThreads);
}

int drift_blocks_per_sm(int tv)
{
    return tv == 1   ? occupancy(drift_pass_kernel<1>, kWaveThreads)
           : tv == 2 ? occupancy(drift_pass_kernel<2>, kWaveThreads)
                     : occupancy(drift_pass_kernel<4>, kWaveThreads);
}

}  // namespace fold3d
