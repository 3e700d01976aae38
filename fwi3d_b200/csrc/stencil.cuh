// stencil.cuh -- the two hot kernels of the wave-propagation path.
//
//   fd_forward_kernel   every leapfrog step of every shot of a batch:
//                       Q <- d (dt^2 v^2 lap(A) + 2 A - d Q)   [+ source]
//                       and the receiver samples of A
//                       (reference: compute_pressure + compute_seismogram,
//                        src/modeling/modeling.cu:324-393)
//   fd_backward_kernel  every step of the fused back-propagation:
//                       Ps    <- dt^2 v^2 lap(Psold) + 2 Psold - Ps  (source rebuilt)
//                       Prold <- dt^2 v^2 lap(Pr) + 2 Pr - Prold      (adjoint)
//                       illum += Ps^2 ; image += Ps Pr  or  the gradient term
//                       (reference: cross_correlation, src/migration/migration.cu:134-202;
//                        build_gradient, src/inversion/inversion.cu:400-468)
//
// Data layout in HBM: every field of one shot is a pitched [nyy][nxx][ldz] FP32
// array (z fastest, ldz = nzz rounded up to 8); the shots of a batch follow
// one another at a stride of `vol` elements.  Cells with an index < 4 or >= n-4
// on any axis are never written and stay 0 (the reference's stencil guard,
// src/modeling/modeling.cu:350).
//
// Tiling: a CTA takes a TZ x TX (z, x) column of one step of one shot and walks
// its y planes.  A thread owns 4 consecutive z cells of R neighbouring x rows.
//   - Arithmetic is on packed pairs of z cells; the y derivative is kept as
//     eight partial sums per cell (push_y).
//   - Stencil fields arrive plane by plane as (TZ+8) x (TX+8) halo tiles,
//     TMA-loaded into a ring of SH shared-memory slots (plane y needs the slots
//     of planes y and y+4, and so those between; the rest is load-ahead).
//   - Centre-only fields (old time level, coefficient) arrive as TZ x TX tiles
//     in a second ring of SH - 4 slots.
//   - One thread issues every TMA copy; completion is tracked with mbarriers
//     whose waits are bounded (kWaitLimitNs) and report through g_status
//     instead of hanging.
#pragma once

#include <type_traits>

#include "device.cuh"
#include "loop_order.h"

namespace fwi {

__device__ unsigned int g_status;

template <int TZ4_, int TX_, int R_>
struct Tile {
    static constexpr int TZ4 = TZ4_, TX = TX_, R = R_;
    static constexpr int NT = TZ4 * TX / R;      // threads: 4 z cells of R x rows each
    static_assert(TX % R == 0, "a thread owns R whole rows");
    static constexpr int TZ = 4 * TZ4;           // z cells
    static constexpr int HZ = TZ + 8, HX = TX + 8;
    static constexpr int HALO_BYTES = HZ * HX * 4;
    static constexpr int HSLOT = (HALO_BYTES + 127) / 128 * 128;
    static constexpr int CTR_BYTES = TZ * TX * 4;
    static constexpr int CSLOT = (CTR_BYTES + 127) / 128 * 128;
    static_assert((HZ * 4) % 16 == 0, "TMA inner box must be a multiple of 16 bytes");
    static_assert(HZ <= 256 && HX <= 256, "TMA box dimension limit");
};

__device__ __forceinline__ void raise_status(unsigned bits) { atomicOr(&g_status, bits); }

// A launch after a failed wait does no work: a time loop whose copies stopped
// completing ends after one bounded wait instead of one per step.
__device__ __forceinline__ bool status_failed() { return *(volatile unsigned int *)&g_status != 0; }

// Exercises the bounded-wait path without any fault: an mbarrier that expects
// two arrivals gets one, so its phase never completes; the wait gives up after
// limit_ns and reports through g_status exactly like the stencil kernels.
__global__ void bounded_wait_probe_kernel(uint64_t limit_ns)
{
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 2);
        fence_mbar_init();
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(&bar)) : "memory");
        if (!mbar_wait(&bar, 0, limit_ns)) raise_status(kErrTimeout);
    }
}

// ---------------------------------------------------------------------------
// Stencil on packed pairs of z cells (fma.rn.f32x2).
// ---------------------------------------------------------------------------
struct f2 {
    unsigned long long v;
};

__device__ __forceinline__ f2 pk(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo(f2 a) { return __uint_as_float((unsigned)a.v); }
__device__ __forceinline__ float hi(f2 a) { return __uint_as_float((unsigned)(a.v >> 32)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ f2 dup2(float x) { return pk(x, x); }

// Four consecutive z cells.
struct q4 {
    f2 a, b;
};
__device__ __forceinline__ q4 ldq(const float *p)
{
    const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(p);
    q4 r;
    r.a.v = u.x;
    r.b.v = u.y;
    return r;
}
__device__ __forceinline__ void stq(float *p, const q4 &x)
{
    *reinterpret_cast<ulonglong2 *>(p) = make_ulonglong2(x.a.v, x.b.v);
}
__device__ __forceinline__ q4 fma4(f2 w, const q4 &x, const q4 &c) { return {fma2(w, x.a, c.a), fma2(w, x.b, c.b)}; }
__device__ __forceinline__ q4 fma4(const q4 &w, const q4 &x, const q4 &c)
{
    return {fma2(w.a, x.a, c.a), fma2(w.b, x.b, c.b)};
}
__device__ __forceinline__ q4 mul4(f2 w, const q4 &x) { return {mul2(w, x.a), mul2(w, x.b)}; }
__device__ __forceinline__ q4 mul4(const q4 &x, const q4 &y) { return {mul2(x.a, y.a), mul2(x.b, y.b)}; }
__device__ __forceinline__ q4 add4(const q4 &x, const q4 &y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ float get(const q4 &x, int e)
{
    return e == 0 ? lo(x.a) : (e == 1 ? hi(x.a) : (e == 2 ? lo(x.b) : hi(x.b)));
}
__device__ __forceinline__ q4 mk4(float e0, float e1, float e2, float e3) { return {pk(e0, e1), pk(e2, e3)}; }

// Adds the cells in `mask` of a quad of the image and of the illumination; the
// others keep their values.  A reduction in L2, which nothing waits for, unless
// `direct`.  It takes addends and sums below 2^-126 for 0, where FP32 still has
// digits, so the caller's addends are scaled up for it (kAccScale).  Time of a
// step against reductions without a scale (301^3 cells, 1000 steps: 146 us): at
// most 1 % more with it, 5 % on 88^3 cells; 20 % with loads a plane ahead, adds
// and stores; 14 % with small quads in an accumulator of their own; 22 % with a
// choice per quad between the reduction and a load and a store; `direct` 38 %.
__device__ __forceinline__ void accumulate4(float *image, float *illum, const q4 &im, const q4 &il, int mask, int direct)
{
    float i[4], l[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        i[e] = (mask >> e) & 1 ? get(im, e) : 0.0f;
        l[e] = (mask >> e) & 1 ? get(il, e) : 0.0f;
    }
    if (!direct) {
        red_add4(image, i[0], i[1], i[2], i[3]);
        red_add4(illum, l[0], l[1], l[2], l[3]);
    } else {
        float4 *pi = reinterpret_cast<float4 *>(image), *pl = reinterpret_cast<float4 *>(illum);
        const float4 oi = __ldcg(pi), ol = __ldcg(pl);
        __stcg(pi, make_float4(oi.x + i[0], oi.y + i[1], oi.z + i[2], oi.w + i[3]));
        __stcg(pl, make_float4(ol.x + l[0], ol.y + l[1], ol.z + l[2], ol.w + l[3]));
    }
}

// *p += v with the digits that FP32 has below 2^-126.  Where |v| >= 2^-101 the
// reduction has them too: an old value below 2^-126 is less than half a unit in
// the last place of v, and a sum that cancels is 0 or a multiple of 2^-125.
__device__ __forceinline__ void accumulate(float *p, float v)
{
    if (!(fabsf(v) < 0x1p-101f))
        red_add(p, v);
    else if (v != 0.0f)
        __stcg(p, __ldcg(p) + v);
}

// The y derivatives of the planes in the making: when plane p arrives, its
// value v enters the sums of planes p-4 .. p+4 with their tap weights.  s[k]
// is the sum of plane p-4+k so far; the call returns the finished plane p-4
// and moves every sum down by one plane, which costs nothing: each
// multiply-add reads s[k+1] and writes s[k].
__device__ __forceinline__ q4 push_y(q4 (&s)[8], const q4 &v)
{
    const q4 done = fma4(dup2(-W4), v, s[0]);
    s[0] = fma4(dup2(W3), v, s[1]);
    s[1] = fma4(dup2(-W2), v, s[2]);
    s[2] = fma4(dup2(W1), v, s[3]);
    s[3] = fma4(dup2(-W0), v, s[4]);
    s[4] = fma4(dup2(W1), v, s[5]);
    s[5] = fma4(dup2(-W2), v, s[6]);
    s[6] = fma4(dup2(W3), v, s[7]);
    s[7] = mul4(dup2(-W4), v);
    return done;
}

// d += the z derivative of 4 cells c whose neighbours are m (4 below) and p (4
// above).  Even distances are packed; odd distances straddle the pairs and
// stay scalar, since building the straddling pairs would cost as many moves
// (the packed ones first: one switch between pairs and scalars, 2 % fewer
// instructions than outer to inner, and 7 % fewer than all scalar).
__device__ __forceinline__ void add_dz(q4 &d, const q4 &m, const q4 &c, const q4 &p)
{
    const float w[12] = {lo(m.a), hi(m.a), lo(m.b), hi(m.b), lo(c.a), hi(c.a),
                         lo(c.b), hi(c.b), lo(p.a), hi(p.a), lo(p.b), hi(p.b)};
    float y[4];
    q4 x = fma4(dup2(-W4), m, d);
    x = fma4(dup2(-W4), p, x);
    x.a = fma2(dup2(-W2), c.b, fma2(dup2(-W2), m.b, x.a));
    x.b = fma2(dup2(-W2), p.a, fma2(dup2(-W2), c.a, x.b));
    x = fma4(dup2(-W0), c, x);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        y[e] = fmaf(W3, w[e + 7], fmaf(W3, w[e + 1], get(x, e)));
        y[e] = fmaf(W1, w[e + 5], fmaf(W1, w[e + 3], y[e]));
    }
    d = mk4(y[0], y[1], y[2], y[3]);
}

// x + z derivatives d of R neighbouring x rows (4 z cells each) of one plane,
// and the rows' own values c.  H: the thread's first cell in the halo tile.
template <class T>
__device__ __forceinline__ void xz_d2(const float *H, q4 (&c)[T::R], q4 (&d)[T::R])
{
    constexpr int R = T::R;
    // row by row, so that few of them are live at once
    constexpr float w[9] = {-W4, W3, -W2, W1, -W0, W1, -W2, W3, -W4};
#pragma unroll
    for (int k = 0; k < R + 8; ++k) {  // row k - 4
        const q4 v = ldq(H + (k - 4) * T::HZ);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (k < r || k > r + 8) continue;
            d[r] = k == r ? mul4(dup2(w[0]), v) : fma4(dup2(w[k - r]), v, d[r]);
            if (k == r + 4) c[r] = v;
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) add_dz(d[r], ldq(H + r * T::HZ - 4), c[r], ldq(H + r * T::HZ + 4));
}

// ---------------------------------------------------------------------------
// Time-loop kernels: roles and hand-over.
//
// One launch runs every step of every shot of a batch.  A work item is one
// step of one column (a TZ x TX tile over all y planes); CTAs take items in
// the order (shot, step, column) from a ticket counter, so every item that an
// item waits for has been taken before it, by a CTA that is running: the waits
// end whatever the number of resident CTAs.  Step t+1 of a column follows step
// t a few planes behind: it may read plane p once its own column and the four
// columns beside it have stored plane p of step t.  Several steps are thus in
// flight at once, each a window of planes apart, and a plane that one step
// stores is read by the next from L2.
//
// The same waits order the overwrites.  Step t overwrites plane y of u^(t-1)
// after the plane y + 4 of u^t has arrived, so the neighbours have stored
// plane y + 4 of step t-1 and therefore read all of plane y.  A halo box also
// covers corner cells of diagonal neighbours, which the stencil never uses.
// Receiver samples are a reader of their own, beside the stencil: the
// publisher keeps its lead over them within kSampleLead planes.  (The rules
// are in loop_order.h.)
//
// Warps of a CTA: NW compute warps; one producer (tickets, waits for the other
// columns, TMA); one publisher (tells the other columns which planes are in
// memory, and samples receivers).  Stage g of a CTA carries halo plane p of
// its current item and the centre tiles of plane y = p - 4; planes 0..3 hold
// only zeros and are not loaded.
// ---------------------------------------------------------------------------
constexpr int kItemRing = 4;      // items described in shared memory at once
// Stages are counted modulo 2^32 and compared by differences, since a CTA of a
// very long loop takes more than 2^31; starting here, every loop wraps.
constexpr unsigned kFirstStage = 0u - 1000u;
constexpr unsigned kNoMoreItems = 1u << 30;   // added to the count of a warp that is through

// FIELDS: fields that advance side by side, each with its own compute warps.
template <class T, int FIELDS>
struct Loop {
    static constexpr int NWF = (T::NT + 31) / 32;  // compute warps of a field
    static constexpr int NW = FIELDS * NWF;
    static constexpr int THREADS = NW * 32 + 64;
};

// State of the CTA's roles in shared memory.
template <int NW>
struct LoopShared {
    long long item[kItemRing];    // tickets of the items in flight, -1 ends
    unsigned staged[NW];          // stages finished by each compute warp, from kFirstStage on
    int items_read;               // items the publisher has looked up
    int abort;
};

__device__ __forceinline__ bool aborted(const int *flag) { return *(const volatile int *)flag != 0; }

__device__ __forceinline__ void loop_fail(int *flag)
{
    *(volatile int *)flag = 1;
    raise_status(kErrTimeout);
}

// Bounded wait until *p >= v (shared memory).
__device__ __forceinline__ bool wait_shared(const int *p, int v, const int *abort_flag)
{
    if (ld_acquire_cta(p) >= v) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i) {
            if (ld_acquire_cta(p) >= v) return true;
            __nanosleep(64);
        }
        if (aborted(abort_flag) || global_ns() - t0 > kWaitLimitNs) return false;
    }
}

__device__ __forceinline__ long long *counter(const LoopProgress &prog, int ncol, int shot, int t, int col)
{
    return prog.done + (((long long)shot * prog.ring + t % prog.ring) * ncol + col) * kCounterStride;
}

// Bounded wait of a warp until every lane's counter has reached `need`; `seen`
// is the lane's last reading.
__device__ __forceinline__ bool wait_columns(const long long *p, long long need, long long &seen,
                                             const int *abort_flag)
{
    if (__all_sync(0xffffffffu, seen >= need)) return true;  // ordered by the fence below, earlier
    const uint64_t t0 = global_ns();
    for (int i = 0;; ++i) {
        if (seen < need) seen = ld_acquire_gpu(p);
        if (__all_sync(0xffffffffu, seen >= need)) break;
        if ((i & 63) == 63) {
            const bool late = aborted(abort_flag) || status_failed() || global_ns() - t0 > kWaitLimitNs;
            if (__any_sync(0xffffffffu, late)) return false;
        }
    }
    __syncwarp();
    fence_proxy_async_global();  // what was acquired, before the copies that follow
    return true;
}

// Smallest number of stages beyond s0 that the compute warps have finished.
template <int NW>
__device__ __forceinline__ int stages_done(const LoopShared<NW> &sh, unsigned s0, int lane)
{
    int v = kNoMoreItems;
    for (int w = lane; w < NW; w += 32) v = min(v, (int)(ld_acquire_cta(&sh.staged[w]) - s0));
    return __reduce_min_sync(0xffffffffu, v);
}

// The receiver cells of a column in plane order, for the warp that follows the
// planes.  Lane l holds cell u + l of the list and the list's place at plane
// base + l, both fetched ahead of the planes.
struct CellCursor {
    const int *below;             // null: nothing to do
    const long long *cells;
    int u, last, base, ahead, nyy;
    long long cell;

    __device__ __forceinline__ void open(const CellLists &lists, int column, int planes, int lane)
    {
        cells = lists.cell;
        below = lists.below + (long long)column * (planes + 1);
        nyy = planes;
        base = 0;
        ahead = below[min(lane, nyy)];
        u = __shfl_sync(0xffffffffu, ahead, 0);
        last = below[nyy];
        if (u == last) below = nullptr;
        fetch(lane);
    }
    __device__ __forceinline__ void fetch(int lane)
    {
        if (u + lane < last) cell = cells[u + lane];
    }
    // End of the list's part below plane n.
    __device__ __forceinline__ int end_below(int n, int lane)
    {
        if (n - base > 31) {
            base = n;
            ahead = below[min(n + lane, nyy)];
        }
        return __shfl_sync(0xffffffffu, ahead, n - base);
    }
};

// Further cells of a plane are taken in bursts of kBurst per lane, whose loads
// are in flight together: a warp that takes 32 at a time is latency-bound, and
// with it the steps that wait for its publications.  201^3 cells with a 50-cell
// pad, 404010 receivers on ten layers: forward 245 us a step by 32, 84 now (94
// with 16 per lane; 61 without receivers), backward 279 and 137; receivers in
// every cell of 44^3, 8-cell pad: forward 35 and 11, backward 162 and 13.
constexpr int kBurst = 8;

// What the roles of a CTA need to know of the loop.
struct LoopGeo {
    int nshot, nsteps, ncol, ntz, nyy;
};

// Producer warp: takes tickets, waits until the planes an item reads are
// stored, and issues the loads of each stage.  start(it) returns the state of
// an item; issue(state, p, hs, cs, centre) runs in lane 0: it announces the
// bytes on full[hs] and starts the copies of halo plane p and, if centre, of
// centre plane p - 4.
template <int SH, int NW, class Start, class Issue>
__device__ __forceinline__ void loop_producer(LoopShared<NW> &sh, uint64_t *full, uint64_t *done, const LoopGeo &geo,
                                              const LoopProgress &prog, int lane, Start start, Issue issue)
{
    constexpr int SC = SH - 4;
    const long long total = (long long)geo.nshot * geo.nsteps * geo.ncol;
    int hs = 0, cs = 0, cph = 1;  // cph: parity of the previous use of done[cs]
    long long g = 0;              // stages issued
    bool ok = true;
    for (int item = 0; ok; ++item) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(prog.ticket, 1ull);
        tk = __shfl_sync(0xffffffffu, tk, 0);
        const bool end = (long long)tk >= total;
        ok = wait_shared(&sh.items_read, item - (kItemRing - 1), &sh.abort) && (g < SC || mbar_wait(&done[cs], cph));
        if (!__all_sync(0xffffffffu, ok)) {
            ok = false;
            break;
        }
        if (lane == 0) *(volatile long long *)&sh.item[item % kItemRing] = end ? -1 : (long long)tk;
        if (end) {
            if (lane == 0) mbar_arrive(&full[hs]);
            break;
        }
        const Item it = item_of((long long)tk, geo.nshot, prog.shots, geo.nsteps, geo.ncol);
        const int dep = it.t > 0 ? dependency_column(lane, it.col, geo.ntz, geo.ncol) : -1;
        const long long *dp = counter(prog, geo.ncol, it.shot, it.t + prog.ring - 1, max(dep, 0));
        long long seen = dep >= 0 ? 0 : 0x7fffffffffffffffll;
        const long long base = (long long)(it.t - 1) * geo.nyy;
        const auto state = start(it);
        for (int p = 4; p < geo.nyy; ++p) {
            if (p > 4 && g >= SC) ok = mbar_wait(&done[cs], cph);
            if (const int need = planes_awaited(p, geo.nyy)) ok = wait_columns(dp, base + need, seen, &sh.abort) && ok;
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            if (lane == 0) issue(state, p, hs, cs, p >= 8);
            ++g;
            if (++hs == SH) hs = 0;
            if (++cs == SC) {
                cs = 0;
                cph ^= 1;
            }
        }
    }
    if (!ok && lane == 0) {
        loop_fail(&sh.abort);  // (the compute warps wait for the same stage and give up as well)
        // no copy may land after the CTA has gone: only the newest use of
        // each slot can still be in flight
        for (int k = 1; k <= SH && k <= g; ++k) {
            const long long st = g - k;
            mbar_wait(&full[st % SH], (st / SH) & 1);
        }
    }
}

// Publisher warp: follows the compute warps and tells the other columns which
// planes of an item are stored.  start(it) returns the state of an item;
// work(state, n) does its work on the planes below n: before they are published
// (LEAD 0), or after LEAD planes at most have been published without it.
template <int LEAD, int NW, class Start, class Work>
__device__ __forceinline__ void loop_publisher(LoopShared<NW> &sh, const LoopGeo &geo, const LoopProgress &prog,
                                               int lane, Start start, Work work)
{
    const int nstage = geo.nyy - 4;  // stages of an item: p = 4 .. nyy-1, y = p - 4
    // stages of the item finished by every compute warp, once there are more
    // than s; -1 when the wait gave up
    unsigned s0 = kFirstStage;  // stages before the item
    auto more_than = [&](int s) {
        int n = stages_done(sh, s0, lane);
        if (n > s) return n;
        const uint64_t t0 = global_ns();
        for (;;) {
            for (int i = 0; i < 64; ++i) {
                __nanosleep(20);
                if ((n = stages_done(sh, s0, lane)) > s) return n;
            }
            const bool late = aborted(&sh.abort) || global_ns() - t0 > 2 * kWaitLimitNs;
            if (__any_sync(0xffffffffu, late)) return -1;
        }
    };
    for (int item = 0;; ++item, s0 += nstage) {
        if (more_than(0) < 0) return;
        // (the compute warps can be through with the last items when the
        // publisher still has some of them ahead, so the item says what is left)
        const long long tk = *(volatile long long *)&sh.item[item % kItemRing];
        if (tk < 0) return;
        __syncwarp();
        if (lane == 0) st_release_cta(&sh.items_read, item + 1);
        const Item it = item_of(tk, geo.nshot, prog.shots, geo.nsteps, geo.ncol);
        long long *dp = counter(prog, geo.ncol, it.shot, it.t, it.col);
        const long long base = (long long)it.t * geo.nyy;
        auto state = start(it);
        int published = 4, stored = 4;  // the first four planes are never written
        while (published < nstage) {
            if (stored == published) {
                const int n = more_than(published);
                if (n < 0) return;
                stored = min(n, nstage);
            }
            published = next_publication(published, stored, LEAD);
            const bool first = work_first(published, nstage, LEAD);
            if (first) work(state, published);
            __syncwarp();
            if (lane == 0) st_release_gpu(dp, base + published);
            __syncwarp();
            if (!first) work(state, published);
        }
    }
}

// ---------------------------------------------------------------------------
// Forward time loop.
//   mh: halo-box maps over the field pair (read with the stencil)
//   mq: centre-box maps over the field pair (the old level, overwritten)
//   mv: centre-box map over the stencil coefficients dt^2 v^2 / dh^2 of the
//       velocity slots (one slot shared by every shot, or one slot per shot
//       when every shot has its own random pad).  They are 0 on the cells
//       that are never updated, which keeps those cells at 0.
// Bound: shared-memory wavefronts (70 % of the L1 pipe: 10 halo rows read for
// 8 cells) together with HBM.  301^3 cells, random pad, one shot, per step:
// 86.1 us as one launch per step with a register queue per cell, 60.7 us now;
// 13.7 bytes per cell from HBM instead of 14.9, since a plane that one step
// stores is often still in L2 when the next reads it; 16 bytes per cell at the
// 6.55 TB/s of a copy take 67 us.  Small grids were bound by the launches and
// by few planes per CTA: 56 x 60 x 58 cells with the Cerjan pad 29 us, now 6.2 us.
// The Cerjan factors per row instead of a branch per cell: 201^3 cells 73 us,
// now 20 us.
// ---------------------------------------------------------------------------
struct FwdMaps {
    CUtensorMap mh[2], mq[2], mv;
};

template <class T, int SH, bool ABC, int CTAS>
__global__ void __launch_bounds__(Loop<T, 1>::THREADS, CTAS)
    fd_forward_kernel(const __grid_constant__ FwdMaps maps, const FwdArgs a)
{
    static_assert(SH >= 6, "plane y needs halo slots y..y+4, and one more to load ahead");
    constexpr int R = T::R, NW = Loop<T, 1>::NW;
    constexpr int SC = SH - 4;  // centre slots: a stage's loads run SC stages ahead of its end
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *hring = smem;
    unsigned char *cring = smem + SH * T::HSLOT;
    uint64_t *full = reinterpret_cast<uint64_t *>(cring + SC * 2 * T::CSLOT);  // [SH] stage loaded
    uint64_t *done = full + SH;                                                // [SC] stage computed
    __shared__ LoopShared<NW> sh;
    __shared__ float b1s[ABC ? kMaxPad : 1];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (status_failed()) return;
    if constexpr (ABC) {
        for (int i = tid; i < a.nb; i += Loop<T, 1>::THREADS) b1s[i] = a.b1d[i];
    }
    if (tid < NW) sh.staged[tid] = kFirstStage;
    if (tid == 0) {
        sh.items_read = 0;
        sh.abort = 0;
        for (int s = 0; s < SH; ++s) mbar_init(&full[s], 1);
        for (int s = 0; s < SC; ++s) mbar_init(&done[s], NW);
        fence_mbar_init();
    }
    __syncthreads();

    const LoopGeo geo{a.binfo->nshot, a.nsteps, a.ncol, a.ntz, a.nyy};
    const long long plane = (long long)a.ldz * a.nxx;

    if (warp == NW) {
        if (lane == 0) {
            prefetch_tmap(&maps.mh[0]);
            prefetch_tmap(&maps.mh[1]);
            prefetch_tmap(&maps.mq[0]);
            prefetch_tmap(&maps.mq[1]);
            prefetch_tmap(&maps.mv);
        }
        struct State {
            const CUtensorMap *mh, *mq;
            int z0, x0, shot, vshot;
        };
        loop_producer<SH>(
            sh, full, done, geo, a.prog, lane,
            [&](const Item &it) {
                return State{&maps.mh[it.t & 1], &maps.mq[1 - (it.t & 1)], 4 + it.col % a.ntz * T::TZ,
                             4 + it.col / a.ntz * T::TX, it.shot, a.vel_slots > 1 ? it.shot : 0};
            },
            [&](const State &st, int p, int hs, int cs, bool centre) {
                uint64_t *bar = &full[hs];
                mbar_expect_tx(bar, T::HALO_BYTES + (centre ? 2 * T::CTR_BYTES : 0));
                tma_load_4d(hring + hs * T::HSLOT, st.mh, bar, st.z0 - 4, st.x0 - 4, p, st.shot);
                if (centre) {
                    unsigned char *c = cring + 2 * cs * T::CSLOT;
                    tma_load_4d(c, st.mq, bar, st.z0, st.x0, p - 4, st.shot);
                    tma_load_4d(c + T::CSLOT, &maps.mv, bar, st.z0, st.x0, p - 4, st.vshot);
                }
            });
    } else if (warp == NW + 1) {
        // Samples of the level the item stores, u^(t+1), a few planes behind the
        // publication where they can be.
        struct State {
            CellCursor at;
            const float *F;
            float *dst;
        };
        const int ncell = a.binfo->ncell;
        loop_publisher<kSampleLead>(
            sh, geo, a.prog, lane,
            [&](const Item &it) {
                const int sample = it.t + 1 - a.tlag;
                State st;
                st.at.below = nullptr;
                if (sample > 0 && it.t + 1 < a.nsteps) {
                    st.at.open(a.rec, it.shot * a.ncol + it.col, a.nyy, lane);
                    st.F = a.F[1 - (it.t & 1)];
                    st.dst = a.seis_tm + (long long)sample * ncell;
                }
                return st;
            },
            [&](State &st, int n) {
                if (!st.at.below) return;
                const int end = st.at.end_below(n, lane);
                if (st.at.u == end) return;
                if (st.at.u + lane < end) st.dst[st.at.u + lane] = __ldcg(st.F + st.at.cell);
                for (int e0 = st.at.u + 32 + lane; e0 < end; e0 += 32 * kBurst) {
                    float v[kBurst];
#pragma unroll
                    for (int k = 0; k < kBurst; ++k)
                        if (e0 + 32 * k < end) v[k] = __ldcg(st.F + st.at.cells[e0 + 32 * k]);
#pragma unroll
                    for (int k = 0; k < kBurst; ++k)
                        if (e0 + 32 * k < end) st.dst[e0 + 32 * k] = v[k];
                }
                __syncwarp();
                st.at.u = end;
                st.at.fetch(lane);
            });
    } else {
        // ---- compute ----
        const int ct = min(tid, T::NT - 1);  // the last warp's spare lanes repeat its last thread
        const int lz = ct % T::TZ4, lx = ct / T::TZ4 * R;
        const int ho = (lx + 4) * T::HZ + 4 + 4 * lz, co = lx * T::TZ + 4 * lz;
        int hs = 0, hph = 0, cs = 0;
        unsigned g = kFirstStage;  // stages finished
        for (int item = 0;; ++item) {
            bool ok = __all_sync(0xffffffffu, mbar_wait(&full[hs], hph) && !aborted(&sh.abort));
            if (!ok) {
                loop_fail(&sh.abort);
                break;
            }
            const long long tk = *(volatile long long *)&sh.item[item % kItemRing];
            if (tk < 0) {
                __syncwarp();
                if (lane == 0) st_release_cta(&sh.staged[warp], g + kNoMoreItems);
                break;
            }
            const Item it = item_of(tk, geo.nshot, a.prog.shots, a.nsteps, a.ncol);
            const int zc = 4 + it.col % a.ntz * T::TZ + 4 * lz, xc = 4 + it.col / a.ntz * T::TX + lx;

            // Cerjan factors of the thread's z cells and x rows, constant over the plane loop
            float bz[4] = {1.f, 1.f, 1.f, 1.f};
            float bx[R];
            int zpad = 0;
#pragma unroll
            for (int r = 0; r < R; ++r) bx[r] = -1.0f;  // outside the x pad
            if constexpr (ABC) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int d = zc + e < a.nzz ? pad_depth(zc + e, a.nzz, a.nb) : -1;
                    if (d >= 0) {
                        bz[e] = b1s[d];
                        zpad |= 1 << e;
                    }
                }
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int d = xc + r < a.nxx ? pad_depth(xc + r, a.nxx, a.nb) : -1;
                    if (d >= 0) bx[r] = b1s[d];
                }
            }
            // source cell among this thread's cells: element se of row sr on plane ys
            const int sz = a.binfo->src[it.shot][0], sx = a.binfo->src[it.shot][1];
            const int se = (sz >= zc && sz < zc + 4) ? sz - zc : -1;
            const int sr = (se >= 0 && sx >= xc && sx < xc + R) ? sx - xc : -1;
            const int ys = sr >= 0 && it.t + 1 < a.nt ? a.binfo->src[it.shot][2] : -1;
            // rows this thread writes
            const int nrow = zc < a.nzz - 4 && tid < T::NT ? min(R, a.nxx - 4 - xc) : 0;
            float *Qp = a.F[1 - (it.t & 1)] + (long long)it.shot * a.vol + 4 * plane + (long long)xc * a.ldz + zc;

            q4 s[R][8];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int m = 0; m < 8; ++m) s[r][m] = mk4(0.f, 0.f, 0.f, 0.f);

            for (int p = 4; p < a.nyy; ++p) {
                const int y = p - 4;
                if (p > 4) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&full[hs], hph));
                    if (!ok) break;
                }
                const float *Hp = reinterpret_cast<const float *>(hring + hs * T::HSLOT) + ho;
                q4 dy[R];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    dy[r] = push_y(s[r], ldq(Hp + r * T::HZ));
                }
                if (y >= 4) {
                    const int hy = hs >= 4 ? hs - 4 : hs + SH - 4;
                    const float *Hy = reinterpret_cast<const float *>(hring + hy * T::HSLOT) + ho;
                    const float *Cq = reinterpret_cast<const float *>(cring + (2 * cs) * T::CSLOT) + co;
                    const float *Cv = reinterpret_cast<const float *>(cring + (2 * cs + 1) * T::CSLOT) + co;
                    q4 c[R], d[R];
                    xz_d2<T>(Hy, c, d);
                    float by = -1.0f;
                    if constexpr (ABC) {
                        const int dep = pad_depth(y, a.nyy, a.nb);
                        if (dep >= 0) by = b1s[dep];
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const q4 lap = add4(d[r], dy[r]);
                        const q4 old = ldq(Cq + r * T::TZ), cv = ldq(Cv + r * T::TZ);
                        q4 out;
                        if constexpr (ABC) {
                            // b2d / b3d of the reference (modeling.cu:101-127) from
                            // the 1-D table; which axes are in the pad is the same
                            // for the whole row except along z
                            float f[4];
                            const bool px = bx[r] >= 0.0f, py = by >= 0.0f;
                            if (px && py) {
                                const float bxy = __fadd_rn(bx[r], by), n2 = __fsub_rn(bxy, 1.0f);
#pragma unroll
                                for (int e = 0; e < 4; ++e)
                                    f[e] = (zpad >> e) & 1
                                               ? __fsub_rn(__fadd_rn(__fadd_rn(__fadd_rn(bz[e], bx[r]), bxy),
                                                                     __fadd_rn(bz[e], by)), 5.0f)
                                               : n2;
                            } else if (px || py) {
                                const float b1 = px ? bx[r] : by;
#pragma unroll
                                for (int e = 0; e < 4; ++e)
                                    f[e] = (zpad >> e) & 1 ? __fsub_rn(__fadd_rn(bz[e], b1), 1.0f) : b1;
                            } else {
#pragma unroll
                                for (int e = 0; e < 4; ++e) f[e] = bz[e];
                            }
                            const q4 f4 = mk4(f[0], f[1], f[2], f[3]), n4 = mk4(-f[0], -f[1], -f[2], -f[3]);
                            out = fma4(cv, lap, fma4(n4, old, add4(c[r], c[r])));
                            out = {mul2(f4.a, out.a), mul2(f4.b, out.b)};
                        } else {
                            out = fma4(cv, lap, fma4(dup2(-1.0f), old, add4(c[r], c[r])));
                        }
                        // Source sample t+1 goes into the new field, which is exactly where
                        // the reference adds it at the start of the next step
                        // (src/modeling/modeling.cu:347-348).
                        if (y == ys && r == sr) {
                            const float add = a.idh3 * a.wavelet[it.t + 1];
                            out = mk4(lo(out.a) + (se == 0 ? add : 0.f), hi(out.a) + (se == 1 ? add : 0.f),
                                      lo(out.b) + (se == 2 ? add : 0.f), hi(out.b) + (se == 3 ? add : 0.f));
                        }
                        if (r < nrow) stq(Qp + r * a.ldz, out);
                    }
                    Qp += plane;
                }
                ++g;
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&done[cs]);
                    st_release_cta(&sh.staged[warp], g);
                }
                if (++hs == SH) {
                    hs = 0;
                    hph ^= 1;
                }
                if (++cs == SC) cs = 0;
            }
            if (!ok) {
                loop_fail(&sh.abort);
                break;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Backward time loop: the source field is rebuilt backwards, the adjoint field
// propagates, and the image (or gradient) and the illumination accumulate.
//   mhs, mhr: halo maps over the source and adjoint field pairs
//   mcs, mcr: centre maps over the same (old time levels, overwritten)
//   mv:       centre map over the stencil coefficients (0 on the cells that
//             are never updated)
// GRAD: gradient imaging condition (with GRAD_DY the d2y term is kept).  Its
// factor dt v^2 / dh^2 is the coefficient times 1/dt.
// The accumulators are updated by vector reductions in L2 (accumulate4): they
// take no shared memory, so the rings run a stage deeper, and nothing waits for
// them.  The steps of a column follow one another, so every cell adds its steps
// in order.  The sums of a loop have a volume of their own and join the
// caller's accumulators after it.
// Each field has its own compute warps, since one thread with the sums of both
// for two rows would need more than 200 registers, and with one row each
// 14 loads per 4 cells (301^3 cells, 4 shots: 0.694 ms per step, by field
// 0.665, with the accumulators out of shared memory 0.573 and the ring that
// this makes room for 0.543).
// Bound: HBM.  301^3 cells, random pad, one shot: 32.1 bytes per cell and step
// at 6.5 TB/s, the rate of a copy (the old levels and the coefficients arrive
// in 148 x 8 boxes, the halos of the two fields are read 2.1 times, from L2).
// 185 us per step as one launch per step, 136 us now; 88^3 cells,
// 4 shots: 35 and 12.1 us.
// ---------------------------------------------------------------------------
struct BwdMaps {
    CUtensorMap mhs[2], mhr[2], mcs[2], mcr[2], mv;
};

template <class T, int SH, bool GRAD, bool GRAD_DY, int CTAS>
__global__ void __launch_bounds__(Loop<T, 2>::THREADS, CTAS)
    fd_backward_kernel(const __grid_constant__ BwdMaps maps, const BwdArgs a)
{
    static_assert(SH >= 6, "plane y needs halo slots y..y+4, and one more to load ahead");
    constexpr int R = T::R, NW = Loop<T, 2>::NW;
    constexpr int SC = SH - 4, NCF = 3;  // centre fields: Ps, Prold, coefficient
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *hring = smem;                      // SH x {Psold, Pr}
    unsigned char *cring = smem + SH * 2 * T::HSLOT;  // SC x {Ps, Prold, coefficient}
    uint64_t *full = reinterpret_cast<uint64_t *>(cring + SC * NCF * T::CSLOT);
    uint64_t *done = full + SH;
    __shared__ LoopShared<NW> sh;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (status_failed()) return;
    if (tid < NW) sh.staged[tid] = kFirstStage;
    if (tid == 0) {
        sh.items_read = 0;
        sh.abort = 0;
        for (int s = 0; s < SH; ++s) mbar_init(&full[s], 1);
        for (int s = 0; s < SC; ++s) mbar_init(&done[s], NW);
        fence_mbar_init();
    }
    __syncthreads();

    const LoopGeo geo{a.binfo->nshot, a.nsteps, a.ncol, a.ntz, a.nyy};
    const long long plane = (long long)a.ldz * a.nxx;
    if (warp == NW) {
        if (lane == 0) {
            for (int b = 0; b < 2; ++b) {
                prefetch_tmap(&maps.mhs[b]);
                prefetch_tmap(&maps.mhr[b]);
                prefetch_tmap(&maps.mcs[b]);
                prefetch_tmap(&maps.mcr[b]);
            }
            prefetch_tmap(&maps.mv);
        }
        struct State {
            const CUtensorMap *mhs, *mhr, *mcs, *mcr;
            int z0, x0, shot, vshot;
        };
        loop_producer<SH>(
            sh, full, done, geo, a.prog, lane,
            [&](const Item &it) {
                const int sc = (a.s0 + it.t) & 1, rc = it.t & 1;
                return State{&maps.mhs[sc], &maps.mhr[rc], &maps.mcs[1 - sc], &maps.mcr[1 - rc],
                             4 + it.col % a.ntz * T::TZ, 4 + it.col / a.ntz * T::TX, it.shot,
                             a.vel_slots > 1 ? it.shot : 0};
            },
            [&](const State &st, int p, int hs, int cs, bool centre) {
                uint64_t *bar = &full[hs];
                mbar_expect_tx(bar, 2 * T::HALO_BYTES + (centre ? NCF * T::CTR_BYTES : 0));
                unsigned char *h = hring + 2 * hs * T::HSLOT;
                tma_load_4d(h, st.mhs, bar, st.z0 - 4, st.x0 - 4, p, st.shot);
                tma_load_4d(h + T::HSLOT, st.mhr, bar, st.z0 - 4, st.x0 - 4, p, st.shot);
                if (centre) {
                    unsigned char *c = cring + cs * NCF * T::CSLOT;
                    tma_load_4d(c + 0 * T::CSLOT, st.mcs, bar, st.z0, st.x0, p - 4, st.shot);
                    tma_load_4d(c + 1 * T::CSLOT, st.mcr, bar, st.z0, st.x0, p - 4, st.shot);
                    tma_load_4d(c + 2 * T::CSLOT, &maps.mv, bar, st.z0, st.x0, p - 4, st.vshot);
                }
            });
    } else if (warp == NW + 1) {
        // Before publishing: the adjoint source of step t+1 is added to the level
        // the item stores.  Lane l has that of its cell at hand, too.
        struct State {
            CellCursor at;
            const float *src;
            float *Pr;
            float f;
        };
        const int ncell = a.binfo->ncell;
        auto fetch = [&](State &st) {
            st.at.fetch(lane);
            if (st.at.u + lane < st.at.last) st.f = st.src[st.at.u + lane];
        };
        loop_publisher<0>(
            sh, geo, a.prog, lane,
            [&](const Item &it) {
                State st;
                st.at.below = nullptr;
                if (it.t + 1 < a.nt) {
                    st.Pr = a.Rf[1 - (it.t & 1)];
                    st.src = a.data_tm + (long long)(a.nt - 2 - it.t) * ncell;
                    st.at.open(a.inj, it.shot * a.ncol + it.col, a.nyy, lane);
                    fetch(st);
                }
                return st;
            },
            [&](State &st, int n) {
                if (!st.at.below) return;
                const int end = st.at.end_below(n, lane);
                if (st.at.u == end) return;
                if (st.at.u + lane < end) accumulate(st.Pr + st.at.cell, st.f);
                for (int e0 = st.at.u + 32 + lane; e0 < end; e0 += 32 * kBurst) {
                    float f[kBurst];
                    long long cell[kBurst];
#pragma unroll
                    for (int k = 0; k < kBurst; ++k)
                        if (e0 + 32 * k < end) {
                            f[k] = st.src[e0 + 32 * k];
                            cell[k] = st.at.cells[e0 + 32 * k];
                        }
#pragma unroll
                    for (int k = 0; k < kBurst; ++k)
                        if (e0 + 32 * k < end) accumulate(st.Pr + cell[k], f[k]);
                }
                __syncwarp();
                st.at.u = end;
                fetch(st);
            });
    } else {
        // ---- compute: the first NWF warps advance the source field and
        // accumulate, the others advance the adjoint field ----
        auto compute = [&](auto source_field) {
            constexpr bool SRC = decltype(source_field)::value;
            constexpr int CF = T::CSLOT / 4;  // floats per centre slot
            const int ft = SRC ? tid : tid - Loop<T, 2>::NWF * 32;
            const int ct = min(ft, T::NT - 1);  // the last warp's spare lanes repeat its last thread
            const int lz = ct % T::TZ4, lx = ct / T::TZ4 * R;
            const int ho = (lx + 4) * T::HZ + 4 + 4 * lz, co = lx * T::TZ + 4 * lz;
            int hs = 0, hph = 0, cs = 0;
            unsigned g = kFirstStage;  // stages finished
            for (int item = 0;; ++item) {
                bool ok = __all_sync(0xffffffffu, mbar_wait(&full[hs], hph) && !aborted(&sh.abort));
                if (!ok) {
                    loop_fail(&sh.abort);
                    break;
                }
                const long long tk = *(volatile long long *)&sh.item[item % kItemRing];
                if (tk < 0) {
                    __syncwarp();
                    if (lane == 0) st_release_cta(&sh.staged[warp], g + kNoMoreItems);
                    break;
                }
                const Item it = item_of(tk, geo.nshot, a.prog.shots, a.nsteps, a.ncol);
                const int zc = 4 + it.col % a.ntz * T::TZ + 4 * lz, xc = 4 + it.col / a.ntz * T::TX + lx;
                const int nrow = zc < a.nzz - 4 && ft < T::NT ? min(R, a.nxx - 4 - xc) : 0;  // rows this thread writes
                const long long off = (long long)it.shot * a.vol + 4 * plane + (long long)xc * a.ldz + zc;
                float *out = (SRC ? a.F[1 - ((a.s0 + it.t) & 1)] : a.Rf[1 - (it.t & 1)]) + off;
                float *image = a.image + it.shot * a.acc_shot + 4 * a.acc_plane + (long long)xc * a.acc_ld + zc;
                // source cell among this thread's cells: element se of row sr on
                // plane ys.  Stored field A_{N-t} carried source sample N-t; the
                // exact rebuild adds it back.
                int se = -1, sr = -1, ys = -1;
                int zmask = 0;  // cells of the thread's quad that accumulate
                if constexpr (SRC) {
                    const int sz = a.binfo->src[it.shot][0], sx = a.binfo->src[it.shot][1];
                    if (sz >= zc && sz < zc + 4) se = sz - zc;
                    if (se >= 0 && sx >= xc && sx < xc + R) sr = sx - xc;
                    if (sr >= 0 && a.subtract_src && a.nsteps - it.t < a.nt) ys = a.binfo->src[it.shot][2];
#pragma unroll
                    for (int e = 0; e < 4; ++e) zmask |= (zc + e >= a.acc_z0 && zc + e < a.acc_z1) ? 1 << e : 0;
                }

                q4 s[R][8];  // y derivatives in the making
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int m = 0; m < 8; ++m) s[r][m] = mk4(0.f, 0.f, 0.f, 0.f);

                for (int p = 4; p < a.nyy; ++p) {
                    const int y = p - 4;
                    if (p > 4) {
                        ok = __all_sync(0xffffffffu, mbar_wait(&full[hs], hph));
                        if (!ok) break;
                    }
                    const float *Hp =
                        reinterpret_cast<const float *>(hring + (2 * hs + (SRC ? 0 : 1)) * T::HSLOT) + ho;
                        q4 dy[R];
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        dy[r] = push_y(s[r], ldq(Hp + r * T::HZ));
                    }
                    if (y >= 4) {
                        const int hy = hs >= 4 ? hs - 4 : hs + SH - 4;
                        const float *Hy =
                            reinterpret_cast<const float *>(hring + (2 * hy + (SRC ? 0 : 1)) * T::HSLOT) + ho;
                        const float *C = reinterpret_cast<const float *>(cring + cs * NCF * T::CSLOT);
                        const bool acc = SRC && zmask && y >= a.acc_y0 && y < a.acc_y1;
                        q4 c[R], d[R];
                        xz_d2<T>(Hy, c, d);
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            const q4 cv = ldq(C + 2 * CF + co + r * T::TZ);
                            const q4 old = ldq(C + (SRC ? 0 : CF) + co + r * T::TZ);
                            const q4 lap = add4(d[r], dy[r]);
                            q4 nv = fma4(cv, lap, fma4(dup2(-1.0f), old, add4(c[r], c[r])));
                            if (SRC && y == ys && r == sr) {
                                const float add = a.idh3 * a.wavelet[a.nsteps - it.t];
                                nv = mk4(lo(nv.a) + (se == 0 ? add : 0.f), hi(nv.a) + (se == 1 ? add : 0.f),
                                         lo(nv.b) + (se == 2 ? add : 0.f), hi(nv.b) + (se == 3 ? add : 0.f));
                            }
                            if (r >= nrow) continue;
                            stq(out + r * a.ldz, nv);
                            // (the box lies inside the updated cells)
                            if (acc && xc + r >= a.acc_x0 && xc + r < a.acc_x1) {
                                const q4 pr = ldq(Hy + T::HSLOT / 4 + r * T::HZ);  // the adjoint field's own value
                                const q4 sv = mul4(dup2(a.acc_scale), nv);
                                const q4 il = mul4(sv, nv);
                                const q4 im = GRAD ? mul4(mul4(mul4(dup2(a.gscale), cv), pr), GRAD_DY ? lap : d[r])
                                                   : mul4(sv, pr);
                                float *to = image + r * a.acc_ld;
                                accumulate4(to, to + a.to_illum, im, il, zmask, a.acc_direct);
                            }
                        }
                        out += plane;
                        if (SRC) image += a.acc_plane;
                    }
                    ++g;
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&done[cs]);
                        st_release_cta(&sh.staged[warp], g);
                    }
                    if (++hs == SH) {
                        hs = 0;
                        hph ^= 1;
                    }
                    if (++cs == SC) cs = 0;
                }
                if (!ok) {
                    loop_fail(&sh.abort);
                    break;
                }
            }
        };
        if (warp < Loop<T, 2>::NWF)
            compute(std::true_type{});
        else
            compute(std::false_type{});
    }
}

}  // namespace fwi
