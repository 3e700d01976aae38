// stencil.cuh -- the two hot kernels of the wave-propagation path.
//
//   fd_forward_kernel   one leapfrog step of every shot of a batch:
//                       Q <- d (dt^2 v^2 lap(A) + 2 A - d Q)   [+ source]
//                       and the receiver samples of A
//                       (reference: compute_pressure + compute_seismogram,
//                        src/modeling/modeling.cu:324-393)
//   fd_backward_kernel  the fused back-propagation step:
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
// Tiling: a CTA owns a TZ x TX (z, x) column of one shot and walks a chunk of
// y planes.  Thread (lz, lx) owns 4 consecutive z cells of row lx.
//   - The forward kernel works on packed pairs of z cells and two x rows per
//     thread, and keeps the y derivative as eight partial sums instead of a
//     queue of nine values (push_y).
//   - Stencil fields arrive plane by plane as (TZ+8) x (TX+8) halo tiles,
//     TMA-loaded into a ring of SH shared-memory slots (plane y needs slots
//     y..y+4 resident; the rest is prefetch).  z and x neighbours come from the
//     tile of plane y, y neighbours from a 9-deep register queue fed with the
//     centre of plane y+4.
//   - Centre-only fields (old time level, velocity, accumulators) arrive as
//     TZ x TX tiles in a second ring of SC slots; the accumulators only
//     where the tile meets the box of accumulated cells, and then only over
//     the z range that meets it.
//   - One elected thread issues every TMA copy; completion is tracked with
//     mbarriers whose waits are bounded (kWaitLimitNs) and report through
//     g_status instead of hanging.
#pragma once

#include "device.cuh"

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

// Second derivative along one axis, without the 1/dh^2 factor, summed from the
// outer taps inwards like the reference (src/modeling/modeling.cu:354-358).
__device__ __forceinline__ float d2(float c, float m1, float p1, float m2, float p2, float m3,
                                    float p3, float m4, float p4)
{
    float acc = -W4 * (m4 + p4);
    acc = fmaf(W3, m3 + p3, acc);
    acc = fmaf(-W2, m2 + p2, acc);
    acc = fmaf(W1, m1 + p1, acc);
    acc = fmaf(-W0, c, acc);
    return acc;
}

// Per-axis second derivatives of 4 consecutive z cells of one thread.
// H: halo tile of the plane (row stride HZ); q: register queue (q[4] = centre).
template <class T>
__device__ __forceinline__ void axis_d2(const float *H, int ro, int zo, const float4 (&q)[9],
                                        float (&ax)[4], float (&ay)[4], float (&az)[4])
{
    const float4 zm = lds4(H + ro + zo - 4);
    const float4 zp = lds4(H + ro + zo + 4);
    const float4 c = q[4];
    const float w[12] = {zm.x, zm.y, zm.z, zm.w, c.x, c.y, c.z, c.w, zp.x, zp.y, zp.z, zp.w};
    float4 xm[4], xp[4];
#pragma unroll
    for (int m = 1; m <= 4; ++m) {
        xm[m - 1] = lds4(H + ro - m * T::HZ + zo);
        xp[m - 1] = lds4(H + ro + m * T::HZ + zo);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float c0 = w[4 + e];
        ax[e] = d2(c0, comp(xm[0], e), comp(xp[0], e), comp(xm[1], e), comp(xp[1], e),
                   comp(xm[2], e), comp(xp[2], e), comp(xm[3], e), comp(xp[3], e));
        ay[e] = d2(c0, comp(q[3], e), comp(q[5], e), comp(q[2], e), comp(q[6], e), comp(q[1], e),
                   comp(q[7], e), comp(q[0], e), comp(q[8], e));
        az[e] = d2(c0, w[3 + e], w[5 + e], w[2 + e], w[6 + e], w[1 + e], w[7 + e], w[e], w[8 + e]);
    }
}

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
__device__ __forceinline__ q4 add4(const q4 &x, const q4 &y) { return {add2(x.a, y.a), add2(x.b, y.b)}; }
__device__ __forceinline__ float get(const q4 &x, int e)
{
    return e == 0 ? lo(x.a) : (e == 1 ? hi(x.a) : (e == 2 ? lo(x.b) : hi(x.b)));
}
__device__ __forceinline__ q4 mk4(float e0, float e1, float e2, float e3) { return {pk(e0, e1), pk(e2, e3)}; }

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
// stay scalar, since building the straddling pairs would cost as many moves.
__device__ __forceinline__ void add_dz(q4 &d, const q4 &m, const q4 &c, const q4 &p)
{
    q4 x = fma4(dup2(-W4), m, d);
    x = fma4(dup2(-W4), p, x);
    const float w[12] = {lo(m.a), hi(m.a), lo(m.b), hi(m.b), lo(c.a), hi(c.a),
                         lo(c.b), hi(c.b), lo(p.a), hi(p.a), lo(p.b), hi(p.b)};
    float y[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = fmaf(W3, w[e + 7], fmaf(W3, w[e + 1], get(x, e)));
    x = mk4(y[0], y[1], y[2], y[3]);
    x.a = fma2(dup2(-W2), c.b, fma2(dup2(-W2), m.b, x.a));
    x.b = fma2(dup2(-W2), p.a, fma2(dup2(-W2), c.a, x.b));
#pragma unroll
    for (int e = 0; e < 4; ++e) y[e] = fmaf(W1, w[e + 5], fmaf(W1, w[e + 3], get(x, e)));
    d = fma4(dup2(-W0), c, mk4(y[0], y[1], y[2], y[3]));
}

// x + z derivatives d of R neighbouring x rows (4 z cells each) of one plane,
// and the rows' own values c.  H: the thread's first cell in the halo tile.
template <class T>
__device__ __forceinline__ void xz_d2(const float *H, q4 (&c)[T::R], q4 (&d)[T::R])
{
    constexpr int R = T::R;
    q4 row[R + 8];  // rows -4 .. R+3
#pragma unroll
    for (int r = 0; r < R + 8; ++r) row[r] = ldq(H + (r - 4) * T::HZ);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        c[r] = row[r + 4];
        q4 x = mul4(dup2(-W4), row[r]);
        x = fma4(dup2(-W4), row[r + 8], x);
        x = fma4(dup2(W3), row[r + 1], x);
        x = fma4(dup2(W3), row[r + 7], x);
        x = fma4(dup2(-W2), row[r + 2], x);
        x = fma4(dup2(-W2), row[r + 6], x);
        x = fma4(dup2(W1), row[r + 3], x);
        x = fma4(dup2(W1), row[r + 5], x);
        d[r] = fma4(dup2(-W0), c[r], x);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) add_dz(d[r], ldq(H + r * T::HZ - 4), c[r], ldq(H + r * T::HZ + 4));
}

// ---------------------------------------------------------------------------
// Forward leapfrog step.
// Bound by HBM: 4 shots of 301^3 padded cells take 0.282 ms a step, 6.19 TB/s
// of 16 B per cell, 94 % of the 6.55 TB/s that a copy reaches (0.324 ms with
// scalar arithmetic, one row per thread and a nine-deep y queue, which were
// limited by instruction issue: 285 instead of about 110 instructions per 128
// cells).  With damping, 201^3 cells take 36 us (73 us with the Cerjan factor
// branched on per cell; here its z part sits in registers and the branch is on
// the row).
//   mh: halo-box map over A (the field read with the stencil)
//   mq: centre-box map over Q (the field overwritten)
//   mv: centre-box map over the stencil coefficients dt^2 v^2 / dh^2 of the
//       velocity slots (one slot shared by every shot, or one slot per shot
//       when every shot has its own random pad).  They are 0 on the cells
//       that are never updated, which keeps those cells at 0.
// ---------------------------------------------------------------------------
template <class T, int SH, int SC, bool ABC>
__global__ void __launch_bounds__(T::NT)
    fd_forward_kernel(const __grid_constant__ CUtensorMap mh, const __grid_constant__ CUtensorMap mq,
                      const __grid_constant__ CUtensorMap mv, const FwdArgs a)
{
    static_assert(SH >= 5, "plane y needs halo slots y..y+4");
    constexpr int R = T::R;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *hring = smem;
    unsigned char *cring = smem + SH * T::HSLOT;
    uint64_t *hbar = reinterpret_cast<uint64_t *>(cring + SC * 2 * T::CSLOT);
    uint64_t *cbar = hbar + SH;
    __shared__ int abort_flag;

    const int tid = threadIdx.x;
    const int shot = blockIdx.y;
    if (status_failed()) return;

    // Receiver samples of A at this step (before the guard below, so that
    // every launched thread takes part).  The reference records P after its
    // in-place damping, i.e. d * A (src/modeling/modeling.cu:378, 391-392).
    if (a.t > a.tlag) {
        const int nrec = a.binfo->R;
        const long long total = (long long)gridDim.x * gridDim.y * T::NT;
        for (long long g = ((long long)blockIdx.y * gridDim.x + blockIdx.x) * T::NT + tid; g < nrec;
             g += total)
            a.seis_tm[(long long)(a.t - a.tlag) * nrec + g] = a.rec_damp[g] * a.A[a.rec_cell[g]];
    }

    int b = blockIdx.x;
    const int zt = b % a.ntz;
    b /= a.ntz;
    const int xt = b % a.ntx;
    const int ch = b / a.ntx;
    const int z0 = 4 + zt * T::TZ, x0 = 4 + xt * T::TX;
    const int ya = 4 + ch * a.ylen;
    const int yb = min(ya + a.ylen, a.nyy - 4);
    if (ya >= yb || shot >= a.binfo->nshot) return;  // uniform per CTA

    const int lz = tid % T::TZ4, lx = tid / T::TZ4 * R;
    const int zc = z0 + 4 * lz, xc = x0 + lx;
    const int vshot = a.vel_slots > 1 ? shot : 0;

    if (tid == 0) {
        abort_flag = 0;
        prefetch_tmap(&mh);
        prefetch_tmap(&mq);
        prefetch_tmap(&mv);
        for (int s = 0; s < SH; ++s) mbar_init(&hbar[s], 1);
        for (int s = 0; s < SC; ++s) mbar_init(&cbar[s], 1);
        fence_mbar_init();
    }
    __syncthreads();

    const int pf = ya - 4, pl = yb + 3;  // halo planes loaded: [pf, pl]
    int h_issued = pf - 1, c_issued = ya - 1;  // meaningful in thread 0 only
    auto issue_h = [&](int p, int s) {
        mbar_expect_tx(&hbar[s], T::HALO_BYTES);
        tma_load_4d(hring + s * T::HSLOT, &mh, &hbar[s], z0 - 4, x0 - 4, p, shot);
        h_issued = p;
    };
    auto issue_c = [&](int y, int s) {
        mbar_expect_tx(&cbar[s], 2 * T::CTR_BYTES);
        tma_load_4d(cring + (2 * s) * T::CSLOT, &mq, &cbar[s], z0, x0, y, shot);
        tma_load_4d(cring + (2 * s + 1) * T::CSLOT, &mv, &cbar[s], z0, x0, y, vshot);
        c_issued = y;
    };
    if (tid == 0) {
        for (int p = pf; p < pf + SH && p <= pl; ++p) issue_h(p, p - pf);
        for (int y = ya; y < ya + SC && y < yb; ++y) issue_c(y, y - ya);
    }

    // Cerjan factors of the thread's z cells, constant over the plane loop.
    float bz[4] = {1.f, 1.f, 1.f, 1.f};
    int zpad = 0;
    if constexpr (ABC) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int d = zc + e < a.nzz ? pad_depth(zc + e, a.nzz, a.nb) : -1;
            if (d >= 0) {
                bz[e] = a.b1d[d];
                zpad |= 1 << e;
            }
        }
    }
    float bx[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        bx[r] = -1.0f;  // outside the x pad
        if constexpr (ABC) {
            const int d = xc + r < a.nxx ? pad_depth(xc + r, a.nxx, a.nb) : -1;
            if (d >= 0) bx[r] = a.b1d[d];
        }
    }

    const int3 src = make_int3(a.binfo->src[shot][0], a.binfo->src[shot][1], a.binfo->src[shot][2]);
    const int se = (src.x >= zc && src.x < zc + 4) ? src.x - zc : -1;  // source cell among this thread's
    const int sr = (se >= 0 && src.y >= xc && src.y < xc + R) ? src.y - xc : -1;
    const int ys = sr >= 0 && a.t + 1 < a.nt ? src.z : -1;
    const int ho = (lx + 4) * T::HZ + 4 + 4 * lz, co = lx * T::TZ + 4 * lz;
    const int nrow = zc < a.nzz - 4 ? min(R, a.nxx - 4 - xc) : 0;  // rows this thread writes
    const long long plane = (long long)a.ldz * a.nxx;
    float *Qp = a.Q + (long long)shot * a.vol + (long long)ya * plane + (long long)xc * a.ldz + zc;

    q4 s[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int m = 0; m < 8; ++m) s[r][m] = mk4(0.f, 0.f, 0.f, 0.f);

    // Ring positions: hs, hph = slot and phase parity of halo plane p; hy =
    // slot of plane y = p - 4; cs, cph = slot and phase parity of centre plane y.
    int hs = 0, hph = 0, hy = 0, cs = 0, cph = 0;
    for (int p = pf; p <= pl; ++p) {
        const int y = p - 4;
        bool ok = mbar_wait(&hbar[hs], hph);
        if (y >= ya) ok = mbar_wait(&cbar[cs], cph) && ok;
        if (!ok) abort_flag = 1;

        const float *Hp = reinterpret_cast<const float *>(hring + hs * T::HSLOT) + ho;
        q4 dy[R];
#pragma unroll
        for (int r = 0; r < R; ++r) dy[r] = push_y(s[r], ldq(Hp + r * T::HZ));

        if (y >= ya) {
            const float *Hy = reinterpret_cast<const float *>(hring + hy * T::HSLOT) + ho;
            const float *Cq = reinterpret_cast<const float *>(cring + (2 * cs) * T::CSLOT) + co;
            const float *Cv = reinterpret_cast<const float *>(cring + (2 * cs + 1) * T::CSLOT) + co;
            q4 c[R], d[R];
            xz_d2<T>(Hy, c, d);
            float by = -1.0f;
            if constexpr (ABC) {
                const int dep = pad_depth(y, a.nyy, a.nb);
                if (dep >= 0) by = a.b1d[dep];
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
                    const float add = a.idh3 * a.wavelet[a.t + 1];
                    out = mk4(lo(out.a) + (se == 0 ? add : 0.f), hi(out.a) + (se == 1 ? add : 0.f),
                              lo(out.b) + (se == 2 ? add : 0.f), hi(out.b) + (se == 3 ? add : 0.f));
                }
                if (r < nrow) stq(Qp + (long long)r * a.ldz, out);
            }
            Qp += plane;
        }
        __syncthreads();
        if (abort_flag) break;
        if (tid == 0) {
            fence_proxy_async();
            if (p < ya) {
                if (p + SH <= pl) issue_h(p + SH, hs);
            } else if (y >= ya) {
                if (y + SH <= pl) issue_h(y + SH, hy);
                if (y + SC < yb) issue_c(y + SC, cs);
            }
        }
        if (++hs == SH) {
            hs = 0;
            hph ^= 1;
        }
        if (y >= ya) {
            if (++hy == SH) hy = 0;
            if (++cs == SC) {
                cs = 0;
                cph ^= 1;
            }
        } else if (y == ya - 1) {
            hy = 4 % SH;
        }
    }

    if (abort_flag && tid == 0) {
        raise_status(kErrTimeout);
        // Drain copies still in flight into this CTA's shared memory.
        // (only the newest use of each slot can still be in flight)
        for (int p = max(pf, h_issued - SH + 1); p <= h_issued; ++p)
            mbar_wait(&hbar[(p - pf) % SH], ((p - pf) / SH) & 1);
        for (int y = max(ya, c_issued - SC + 1); y <= c_issued; ++y)
            mbar_wait(&cbar[(y - ya) % SC], ((y - ya) / SC) & 1);
    }
}

// ---------------------------------------------------------------------------
// Fused backward step.
//   mhs, mhr: halo maps over Psold and Pr
//   mcs, mcr: centre maps over Ps and Prold (old time levels, overwritten)
//   mv:       centre map over the velocity slots (shared, or one per shot);
//             with the image condition over their stencil coefficient
//             dt^2 v^2 / dh^2 instead (the gradient condition also needs v^2)
//   mim, mil: maps over the image/gradient and illumination slots, with a box
//             of acc_zbox x TX cells (the widest z range of a tile that meets
//             the accumulated box)
// GRAD: gradient imaging condition (with GRAD_DY the d2y term is kept).
// ---------------------------------------------------------------------------
template <class T, int SH, int SC, bool GRAD, bool GRAD_DY>
__global__ void __launch_bounds__(T::NT)
    fd_backward_kernel(const __grid_constant__ CUtensorMap mhs, const __grid_constant__ CUtensorMap mhr,
                       const __grid_constant__ CUtensorMap mcs, const __grid_constant__ CUtensorMap mcr,
                       const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mim,
                       const __grid_constant__ CUtensorMap mil, const BwdArgs a)
{
    static_assert(SH >= 5, "plane y needs halo slots y..y+4");
    constexpr int NCF = 5;  // centre fields: Ps, Prold, v, image, illum
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *hring = smem;                            // SH x {Psold, Pr}
    unsigned char *cring = smem + SH * 2 * T::HSLOT;        // SC x {Ps, Prold, v, img, ill}
    uint64_t *hbar = reinterpret_cast<uint64_t *>(cring + SC * NCF * T::CSLOT);
    uint64_t *cbar = hbar + SH;
    __shared__ int abort_flag;

    const int tid = threadIdx.x;
    const int shot = blockIdx.y;
    if (status_failed()) return;
    int b = blockIdx.x;
    const int zt = b % a.ntz;
    b /= a.ntz;
    const int xt = b % a.ntx;
    const int ch = b / a.ntx;
    const int z0 = 4 + zt * T::TZ, x0 = 4 + xt * T::TX;
    const int ya = 4 + ch * a.ylen;
    const int yb = min(ya + a.ylen, a.nyy - 4);
    if (ya >= yb || shot >= a.binfo->nshot) return;

    const int lz = tid % T::TZ4, lx = tid / T::TZ4;
    const int zc = z0 + 4 * lz, xc = x0 + lx;
    const int vshot = a.vel_slots > 1 ? shot : 0;
    // Accumulator box: a CTA whose tile misses it in z or x, and every plane
    // outside it in y, moves no accumulator bytes at all.
    const bool acc_tile = z0 < a.acc_z1 && z0 + T::TZ > a.acc_z0 && x0 < a.acc_x1 && x0 + T::TX > a.acc_x0;
    const bool acc_row = xc >= a.acc_x0 && xc < a.acc_x1 && zc < a.acc_z1 && zc + 4 > a.acc_z0;
    auto acc_plane = [&](int y) { return acc_tile && y >= a.acc_y0 && y < a.acc_y1; };
    // Accumulator tiles cover z in [za, za + acc_zbox) only: the part of the
    // tile's z range that reaches the box, widened to float4 boundaries (the
    // TMA start stays 16-byte aligned).
    const int za = max(z0, a.acc_z0) & ~3;
    const int acc_bytes = a.acc_zbox * T::TX * 4;

    if (tid == 0) {
        abort_flag = 0;
        prefetch_tmap(&mhs);
        prefetch_tmap(&mhr);
        for (int s = 0; s < SH; ++s) mbar_init(&hbar[s], 1);
        for (int s = 0; s < SC; ++s) mbar_init(&cbar[s], 1);
        fence_mbar_init();
    }
    __syncthreads();

    const int pf = ya - 4, pl = yb + 3;
    int h_issued = pf - 1, c_issued = ya - 1;
    auto issue_h = [&](int p, int s) {
        mbar_expect_tx(&hbar[s], 2 * T::HALO_BYTES);
        tma_load_4d(hring + (2 * s) * T::HSLOT, &mhs, &hbar[s], z0 - 4, x0 - 4, p, shot);
        tma_load_4d(hring + (2 * s + 1) * T::HSLOT, &mhr, &hbar[s], z0 - 4, x0 - 4, p, shot);
        h_issued = p;
    };
    auto issue_c = [&](int y, int s) {
        unsigned char *base = cring + s * NCF * T::CSLOT;
        const bool acc = acc_plane(y);
        mbar_expect_tx(&cbar[s], (NCF - 2) * T::CTR_BYTES + (acc ? 2 * acc_bytes : 0));
        tma_load_4d(base + 0 * T::CSLOT, &mcs, &cbar[s], z0, x0, y, shot);
        tma_load_4d(base + 1 * T::CSLOT, &mcr, &cbar[s], z0, x0, y, shot);
        tma_load_4d(base + 2 * T::CSLOT, &mv, &cbar[s], z0, x0, y, vshot);
        if (acc) {
            tma_load_4d(base + 3 * T::CSLOT, &mim, &cbar[s], za, x0, y, shot);
            tma_load_4d(base + 4 * T::CSLOT, &mil, &cbar[s], za, x0, y, shot);
        }
        c_issued = y;
    };
    if (tid == 0) {
        for (int p = pf; p < pf + SH && p <= pl; ++p) issue_h(p, p - pf);
        for (int y = ya; y < ya + SC && y < yb; ++y) issue_c(y, y - ya);
    }

    const int3 src = make_int3(a.binfo->src[shot][0], a.binfo->src[shot][1], a.binfo->src[shot][2]);
    // Stored field A_{N-t} carried source sample N-t; the exact rebuild adds it back.
    const float scorr = (a.subtract_src && a.nsteps - a.t < a.nt)
                            ? a.idh3 * a.wavelet[a.nsteps - a.t] : 0.0f;
    const int ro = (lx + 4) * T::HZ, zo = 4 + 4 * lz;
    const bool row_ok = xc < a.nxx - 4 && zc < a.nzz - 4;
    const long long plane = (long long)a.ldz * a.nxx;
    const long long sh_off = (long long)shot * a.vol;

    float4 qs[9], qr[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) {
        qs[m] = make_float4(0.f, 0.f, 0.f, 0.f);
        qr[m] = qs[m];
    }

    // Ring positions as counters (no division by the ring depths per plane):
    // hs, hph = slot and phase parity of halo plane p; hy = slot of plane
    // y = p - 4; cs, cph = slot and phase parity of centre plane y.
    int hs = 0, hph = 0, cs = 0, cph = 0;
    for (int p = pf; p <= pl; ++p) {
        const int y = p - 4;
        const int hy = hs >= 4 ? hs - 4 : hs + SH - 4;
        bool ok = mbar_wait(&hbar[hs], hph);
        if (y >= ya) ok = mbar_wait(&cbar[cs], cph) && ok;
        if (!ok) abort_flag = 1;

        const float *Hs = reinterpret_cast<const float *>(hring + (2 * hs) * T::HSLOT);
        const float *Hr = reinterpret_cast<const float *>(hring + (2 * hs + 1) * T::HSLOT);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            qs[m] = qs[m + 1];
            qr[m] = qr[m + 1];
        }
        qs[8] = lds4(Hs + ro + zo);
        qr[8] = lds4(Hr + ro + zo);

        if (y >= ya) {
            const float *Hys = reinterpret_cast<const float *>(hring + (2 * hy) * T::HSLOT);
            const float *Hyr = reinterpret_cast<const float *>(hring + (2 * hy + 1) * T::HSLOT);
            const float *C = reinterpret_cast<const float *>(cring + cs * NCF * T::CSLOT);
            constexpr int CF = T::CSLOT / 4;  // floats per centre slot
            const int co = lx * T::TZ + 4 * lz;
            const float4 ps_old = lds4(C + 0 * CF + co);
            const float4 pr_old = lds4(C + 1 * CF + co);
            const float4 vv = lds4(C + 2 * CF + co);
            const bool acc = acc_plane(y);
            float4 img = make_float4(0.f, 0.f, 0.f, 0.f), ill = img;
            if (acc && acc_row) {  // then za <= zc and zc + 4 <= za + acc_zbox
                const int ao = lx * a.acc_zbox + (zc - za);
                img = lds4(C + 3 * CF + ao);
                ill = lds4(C + 4 * CF + ao);
            }

            float sx[4], sy[4], sz[4];
            axis_d2<T>(Hys, ro, zo, qs, sx, sy, sz);
            float4 ps_new, pr_new;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float v = comp(vv, e);
                const float cv = GRAD ? v * v * a.cvel : v;
                float s = fmaf(cv, sx[e] + sy[e] + sz[e], 2.0f * comp(qs[4], e) - comp(ps_old, e));
                set_comp(ps_new, e, s);
            }
            if (y == src.z && xc == src.y) {
                const int e = src.x - zc;
                if (e >= 0 && e < 4) set_comp(ps_new, e, comp(ps_new, e) + scorr);
            }
            float rx[4], ry[4], rz[4];
            axis_d2<T>(Hyr, ro, zo, qr, rx, ry, rz);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float v = comp(vv, e);
                const float v2 = v * v;  // used by the gradient condition only
                const float cv = GRAD ? v2 * a.cvel : v;
                const float prc = comp(qr[4], e);
                set_comp(pr_new, e, fmaf(cv, rx[e] + ry[e] + rz[e], 2.0f * prc - comp(pr_old, e)));
                const float psn = comp(ps_new, e);
                const int ze = zc + e;
                if (ze >= a.nzz - 4) {
                    set_comp(ps_new, e, comp(ps_old, e));
                    set_comp(pr_new, e, comp(pr_old, e));
                }
                // (the box lies inside the updated cells: acc_z1 <= nzz - 4)
                if (acc && acc_row && ze >= a.acc_z0 && ze < a.acc_z1) {
                    float im = comp(img, e), il = comp(ill, e);
                    il = fmaf(psn, psn, il);
                    if constexpr (GRAD) {
                        const float lz2 = GRAD_DY ? (sx[e] + sz[e] + sy[e]) : (sx[e] + sz[e]);
                        im += a.gscale * prc * lz2 * v2;
                    } else {
                        im = fmaf(psn, prc, im);
                    }
                    set_comp(img, e, im);
                    set_comp(ill, e, il);
                }
            }
            if (row_ok) {
                const long long off = sh_off + y * plane + (long long)xc * a.ldz + zc;
                *reinterpret_cast<float4 *>(a.Ps + off) = ps_new;
                *reinterpret_cast<float4 *>(a.Prold + off) = pr_new;
                if (acc && acc_row) {
                    *reinterpret_cast<float4 *>(a.image + off) = img;
                    *reinterpret_cast<float4 *>(a.illum + off) = ill;
                }
            }
        }
        __syncthreads();
        if (abort_flag) break;
        if (tid == 0) {
            fence_proxy_async();
            if (p < ya) {
                if (p + SH <= pl) issue_h(p + SH, hs);
            } else if (y >= ya) {
                if (y + SH <= pl) issue_h(y + SH, hy);
                if (y + SC < yb) issue_c(y + SC, cs);
            }
        }
        if (++hs == SH) {
            hs = 0;
            hph ^= 1;
        }
        if (y >= ya && ++cs == SC) {
            cs = 0;
            cph ^= 1;
        }
    }

    if (abort_flag && tid == 0) {
        raise_status(kErrTimeout);
        // (only the newest use of each slot can still be in flight)
        for (int p = max(pf, h_issued - SH + 1); p <= h_issued; ++p)
            mbar_wait(&hbar[(p - pf) % SH], ((p - pf) / SH) & 1);
        for (int y = max(ya, c_issued - SC + 1); y <= c_issued; ++y)
            mbar_wait(&cbar[(y - ya) % SC], ((y - ya) / SC) & 1);
    }
}

}  // namespace fwi
