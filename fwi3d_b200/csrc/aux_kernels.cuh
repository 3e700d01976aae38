// aux_kernels.cuh -- the small kernels around the two stencil kernels:
// padding, source start, adjoint injection, seismogram transposes, image and
// gradient post-processing, FP64 reductions and the random boundary.
#pragma once

#include "device.cuh"

namespace fwi {

// f(i, j, k, row) for every cell of nz x nx x ny, a warp to a z row.  The kernels
// built on it are copies that HBM bounds; with a thread to a cell, two 64-bit
// divisions per cell took longer than the copy.  Now a lane divides once per
// row.  301^3 cells: coefficients 135 -> 39 us (33 us at the rate of a copy),
// largest velocity 63 -> 31 us (18 us to read), edge padding 94 -> 32 us;
// image of 201^3 cells from dense accumulators, with 32 MB to the host, 806 ->
// 732 us.  Rows shorter than a warp leave lanes idle, which costs less than
// the divisions (88^3 cells: no difference), given a grid by rows: with one by
// cells, warps took several short rows in turn (image of 5^3 cells, the call:
// 32 us, 23 now).  LANES 256: a block to a row, for few and long rows, where the
// passes of a warp over its row wait for one another (image kernel, 500 x 16 x 16
// cells: 14.5 us with warps, 4.1 with blocks; 4.0 with a thread per cell).  Parts of
// rows to a warp take a division more (201^3 cells: 33 us, 48 with it).
template <int LANES = 32, class F>
__device__ __forceinline__ void for_cells(int nz, int nx, int ny, F f)
{
    const long long rows = (long long)nx * ny, step = (long long)gridDim.x * (blockDim.x / LANES);
    for (long long r = blockIdx.x * (long long)(blockDim.x / LANES) + threadIdx.x / LANES; r < rows; r += step) {
        const int k = (int)(r / nx), j = (int)(r - (long long)k * nx);
#pragma unroll 4
        for (int i = threadIdx.x % LANES; i < nz; i += LANES) f(i, j, k, r);
    }
}

// ---------------------------------------------------------------------------
// Edge-replication padding of an unpadded [nz,nx,ny] model into a pitched
// padded field: every padded cell copies the nearest model cell
// (same result as expand_boundary, src/modeling/modeling.cu:181-228).
// ---------------------------------------------------------------------------
__global__ void pad_edges_kernel(const float *__restrict__ in, int nz, int nx, int ny, int nb,
                                 int nzz, int nxx, int nyy, int ldz, float *__restrict__ out)
{
    for_cells(ldz, nxx, nyy, [&](int i, int j, int k, long long r) {
        const int is = min(max(i - nb, 0), nz - 1);
        const int js = min(max(j - nb, 0), nx - 1);
        const int ks = min(max(k - nb, 0), ny - 1);
        out[r * ldz + i] = i < nzz ? in[is + (long long)js * nz + (long long)ks * nx * nz] : 0.0f;
    });
}

// Dense padded [nzz,nxx,nyy] <-> pitched [nyy][nxx][ldz].
__global__ void dense_to_pitched_kernel(const float *__restrict__ in, int nzz, int nxx, int nyy,
                                        int ldz, float *__restrict__ out)
{
    for_cells(ldz, nxx, nyy,
              [&](int i, int, int, long long r) { out[r * ldz + i] = i < nzz ? in[r * nzz + i] : 0.0f; });
}

__global__ void pitched_to_dense_kernel(const float *__restrict__ in, int nzz, int nxx, int nyy,
                                        int ldz, float *__restrict__ out)
{
    for_cells(nzz, nxx, nyy, [&](int i, int, int, long long r) { out[r * nzz + i] = in[r * ldz + i]; });
}

// Sum the accumulator slots of a batch into slot 0.
__global__ void sum_slots_kernel(float *__restrict__ acc, long long vol, int nslot)
{
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < vol;
         c += (long long)gridDim.x * blockDim.x) {
        float s = acc[c];
        for (int k = 1; k < nslot; ++k) {
            s += acc[c + k * vol];
            acc[c + k * vol] = 0.0f;
        }
        acc[c] = s;
    }
}

// Accumulators of one time loop: z x x x y cells of the box per shot with z pitch
// ld, image and illumination by blockIdx.y, times kAccScale.  A value that is not
// finite has left the range that the scale leaves and sets *over.
__global__ void check_loop_sums_kernel(const float *__restrict__ sums, long long n, unsigned *__restrict__ over)
{
    bool bad = false;
    const float4 *s = reinterpret_cast<const float4 *>(sums);
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n / 4; c += (long long)gridDim.x * blockDim.x) {
        const float4 v = s[c];
        bad |= !isfinite(v.x) || !isfinite(v.y) || !isfinite(v.z) || !isfinite(v.w);
    }
    if (bad) *over = 1u;
}

// Adds them to the accumulators, whose box starts at `box`, unless *over, and
// leaves them at 0.
__global__ void fold_loop_sums_kernel(float *__restrict__ sums, long long to_illum, int ld, int nx, int ny, int nshot,
                                      float *__restrict__ image, float *__restrict__ illum, long long box,
                                      long long vol, int ldz, int nxx, const unsigned *__restrict__ over)
{
    sums += blockIdx.y * to_illum;
    float *acc = (blockIdx.y ? illum : image) + box;
    const bool drop = *over != 0u;
    for_cells(ld, nx, ny * nshot, [&](int i, int j, int ks, long long r) {
        const float v = sums[r * ld + i];
        if (v == 0.0f) return;
        if (!drop) acc[ks / ny * vol + ((long long)(ks % ny) * nxx + j) * ldz + i] += v * (1.0f / kAccScale);
        sums[r * ld + i] = 0.0f;
    });
}

// First source sample of every shot: A[src] = idh3 * w[0]
// (src/modeling/modeling.cu:347-348 at t = 0).
__global__ void start_source_kernel(float *__restrict__ A, long long vol, int ldz, int nxx,
                                    const BatchInfo *__restrict__ bi, const float *__restrict__ w,
                                    float idh3)
{
    const int s = threadIdx.x;
    if (s < bi->nshot) {
        const long long c = (long long)s * vol + bi->src[s][0] + (long long)bi->src[s][1] * ldz +
                            (long long)bi->src[s][2] * ldz * nxx;
        A[c] += idh3 * w[0];
    }
}

// ---------------------------------------------------------------------------
// Adjoint sources: the sum of idh3 * d(receiver) over the receivers on a cell
// (inject_seismogram / inject_residuo, src/migration/migration.cu:119-132,
// src/inversion/inversion.cu:385-398), in receiver order, which keeps it
// deterministic where the reference uses atomicAdd.  Data [R][nt] -> [nt][ncell]
// in the order of the cell lists, 32x32 tiles through shared memory; the
// receivers of cell u are rid[first[u]] .. rid[first[u+1]-1].  A grid has 65535
// blocks along the times, which go on beyond 2097120 of them.
// ---------------------------------------------------------------------------
__global__ void gather_data_kernel(const float *__restrict__ in, int nt, int ncell, const int *__restrict__ first,
                                   const int *__restrict__ rid, float idh3, float *__restrict__ out)
{
    __shared__ float tile[32][33];
    const int u0 = blockIdx.x * 32;
    for (long long t0 = blockIdx.y * 32; t0 < nt; t0 += gridDim.y * 32) {
        for (int k = threadIdx.y; k < 32; k += blockDim.y) {
            const long long t = t0 + threadIdx.x;
            const int u = u0 + k;
            if (u < ncell && t < nt) {
                float v = 0.0f;
                for (int q = first[u]; q < first[u + 1]; ++q) v += idh3 * in[(long long)rid[q] * nt + t];
                tile[k][threadIdx.x] = v;
            }
        }
        __syncthreads();
        for (int k = threadIdx.y; k < 32; k += blockDim.y) {
            const long long t = t0 + k;
            const int u = u0 + threadIdx.x;
            if (u < ncell && t < nt) out[t * ncell + u] = tile[threadIdx.x][k];
        }
        __syncthreads();
    }
}

// Adjoint source of step 0, before the time loop adds the others.
__global__ void inject_adjoint_kernel(float *__restrict__ Pr, const BatchInfo *__restrict__ bi,
                                      const long long *__restrict__ cell, const float *__restrict__ data)
{
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < bi->ncell; u += gridDim.x * blockDim.x)
        Pr[cell[u]] += data[u];
}

// Samples of the receiver cells [nt][ncell] -> seismograms [R][nt].  The
// reference records P after its in-place damping (src/modeling/modeling.cu:378,
// 391-392), so every receiver has its factor (1 without a damping boundary).
__global__ void scatter_seis_kernel(const float *__restrict__ in, int nt, int ncell, const int *__restrict__ first,
                                    const int *__restrict__ rid, const float *__restrict__ damp, float *__restrict__ out)
{
    __shared__ float tile[32][33];
    const int u0 = blockIdx.x * 32, t0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int t = t0 + k, u = u0 + threadIdx.x;
        if (u < ncell && t < nt) tile[k][threadIdx.x] = in[(long long)t * ncell + u];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int u = u0 + k, t = t0 + threadIdx.x;
        if (u < ncell && t < nt)
            for (int q = first[u]; q < first[u + 1]; ++q)
                out[(long long)rid[q] * nt + t] = damp[rid[q]] * tile[threadIdx.x][k];
    }
}

// ---------------------------------------------------------------------------
// RTM image: crop, divide by illumination, -d2/dz2 * idh2 with the first and
// last depth sample 0 (Migration::export_seismic,
// src/migration/migration.cu:90-117), FP32 like the reference.
// ---------------------------------------------------------------------------
// Image or gradient over illumination.  A cell the source field never
// reached has illumination 0 and no image either; the reference's 0/0 there
// is NaN (src/migration/migration.cu:100, src/inversion/inversion.cu:150), the
// project defines it as 0.
__device__ __forceinline__ float ratio(float a, float ill) { return ill != 0.0f ? a / ill : 0.0f; }

template <int LANES>
__global__ void rtm_image_kernel(const float *__restrict__ img, const float *__restrict__ ill,
                                 int nz, int nx, int ny, int nb, int nxx, int ldz, float idh2,
                                 float *__restrict__ out)
{
    for_cells<LANES>(nz, nx, ny, [&](int i, int j, int k, long long r) {
        float v = 0.0f;
        if (i > 0 && i < nz - 1) {
            const long long p = (i + nb) + (long long)(j + nb) * ldz + (long long)(k + nb) * ldz * nxx;
            const float sm = ratio(img[p - 1], ill[p - 1]);
            const float s0 = ratio(img[p], ill[p]);
            const float sp = ratio(img[p + 1], ill[p + 1]);
            v = -1.0f * (sm - 2.0f * s0 + sp) * idh2;
        }
        out[r * nz + i] = v;
    });
}

// Gradient post-processing, first pass: crop, divide, -d2/dz2 below the mask
// and the running max |g| (src/inversion/inversion.cu:142-165).  max|g| of
// non-negative floats is taken with an integer atomicMax on their bits, which
// is exact and order independent.
template <int LANES>
__global__ void grad_post_kernel(const float *__restrict__ g, const float *__restrict__ ill, int nz,
                                 int nx, int ny, int nb, int nxx, int ldz, float idh2, int imask,
                                 float *__restrict__ out, unsigned int *__restrict__ gmax_bits)
{
    float lmax = 0.0f;
    for_cells<LANES>(nz, nx, ny, [&](int i, int j, int k, long long r) {
        float v = 0.0f;
        if (i > imask && i < nz - 1) {
            const long long p = (i + nb) + (long long)(j + nb) * ldz + (long long)(k + nb) * ldz * nxx;
            const float sm = ratio(g[p - 1], ill[p - 1]);
            const float s0 = ratio(g[p], ill[p]);
            const float sp = ratio(g[p + 1], ill[p + 1]);
            v = -1.0f * (sm - 2.0f * s0 + sp) * idh2;
        }
        out[r * nz + i] = v;
        lmax = fmaxf(lmax, fabsf(v));
    });
    for (int o = 16; o > 0; o >>= 1) lmax = fmaxf(lmax, __shfl_xor_sync(0xffffffffu, lmax, o));
    // (most warps see a larger maximum already: 16 x 16 x 500 cells, 9.2 us with an
    // atomic for each of the 8000 warps, 6.4 now)
    if ((threadIdx.x & 31) == 0 && __float_as_uint(lmax) > *(volatile unsigned int *)gmax_bits)
        atomicMax(gmax_bits, __float_as_uint(lmax));
}

// Second pass: g *= 1/gmax (src/inversion/inversion.cu:167-169).
__global__ void scale_by_inverse_kernel(float *__restrict__ g, long long n,
                                        const unsigned int *__restrict__ gmax_bits)
{
    const float m = __uint_as_float(*gmax_bits);
    const float s = m > 0.0f ? 1.0f / m : 0.0f;  // an all-zero gradient stays zero
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
         c += (long long)gridDim.x * blockDim.x)
        g[c] *= s;
}

// ---------------------------------------------------------------------------
// FP64 reductions.  Every block writes one partial; the block that finishes
// last adds the partials in a fixed order, so the result does not depend on
// scheduling, and stores the total in mapped host memory: one launch and no
// copy back.
// ---------------------------------------------------------------------------
template <int NT>
__device__ __forceinline__ double block_sum(double v)
{
    __shared__ double red[NT / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < NT / 32; ++w) s += red[w];
    return s;
}

// The block's value into partial[]; the last block to get here adds up.
// arrived counts blocks and is left at 0.
template <int NT>
__device__ __forceinline__ void finish_sum(double acc, double *partial, unsigned *arrived, double *out)
{
    __shared__ bool last;
    const double s = block_sum<NT>(acc);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    for (int c = threadIdx.x; c < (int)gridDim.x; c += NT) t += __ldcg(partial + c);
    t = block_sum<NT>(t);
    if (threadIdx.x == 0) {
        *out = t;
        *arrived = 0u;
    }
}

// Four consecutive elements from index 4 q, as one load where the pointer is
// 16-byte aligned.
template <bool VEC>
__device__ __forceinline__ float4 load4(const float *__restrict__ p, long long q)
{
    if constexpr (VEC) return __ldcs(reinterpret_cast<const float4 *>(p) + q);
    return make_float4(__ldcs(p + 4 * q), __ldcs(p + 4 * q + 1), __ldcs(p + 4 * q + 2), __ldcs(p + 4 * q + 3));
}

// The two reductions below stream their inputs once and are bound by HBM, so
// what counts is bytes in flight: each thread has kQuads independent quads of
// both inputs outstanding.  45.6 M residual samples with the residual stored:
// the whole call takes 0.101 ms (0.160 ms with scalar loads, two blocks per SM,
// a second launch for the total and a copy of it).  The order of the sum depends
// on n and the grid alone, not on the alignment.
constexpr int kQuads = 4;

// res = obs - cal (FP32, as the reference stores it) and sum(res^2) in FP64
// (src/inversion/inversion.cu:194-198).
template <int NT, bool VEC>
__global__ void __launch_bounds__(NT)
    residual_partial_kernel(const float *__restrict__ obs, const float *__restrict__ cal,
                            long long n, float *__restrict__ res, double *__restrict__ partial,
                            unsigned *__restrict__ arrived, double *__restrict__ out)
{
    double acc = 0.0;
    const long long nq = n / 4, stride = (long long)gridDim.x * NT;
    long long q = blockIdx.x * (long long)NT + threadIdx.x;
    auto quad = [&](long long i, const float4 &o, const float4 &c) {
        const float r0 = o.x - c.x, r1 = o.y - c.y, r2 = o.z - c.z, r3 = o.w - c.w;
        if (res) {
            if constexpr (VEC) {
                __stcs(reinterpret_cast<float4 *>(res) + i, make_float4(r0, r1, r2, r3));
            } else {
                res[4 * i] = r0;
                res[4 * i + 1] = r1;
                res[4 * i + 2] = r2;
                res[4 * i + 3] = r3;
            }
        }
        acc += (double)r0 * (double)r0;
        acc += (double)r1 * (double)r1;
        acc += (double)r2 * (double)r2;
        acc += (double)r3 * (double)r3;
    };
    for (; q + (kQuads - 1) * stride < nq; q += kQuads * stride) {
        float4 o[kQuads], c[kQuads];
#pragma unroll
        for (int k = 0; k < kQuads; ++k) {
            o[k] = load4<VEC>(obs, q + k * stride);
            c[k] = load4<VEC>(cal, q + k * stride);
        }
#pragma unroll
        for (int k = 0; k < kQuads; ++k) quad(q + k * stride, o[k], c[k]);
    }
    for (; q < nq; q += stride) quad(q, load4<VEC>(obs, q), load4<VEC>(cal, q));
    if (blockIdx.x == 0 && 4 * nq + threadIdx.x < n) {  // the last n % 4 elements
        const float r = obs[4 * nq + threadIdx.x] - cal[4 * nq + threadIdx.x];
        if (res) res[4 * nq + threadIdx.x] = r;
        acc += (double)r * (double)r;
    }
    finish_sum<NT>(acc, partial, arrived, out);
}

template <int NT, bool VEC>
__global__ void __launch_bounds__(NT)
    dot_partial_kernel(const float *__restrict__ a, const float *__restrict__ b, long long n,
                       double *__restrict__ partial, unsigned *__restrict__ arrived, double *__restrict__ out)
{
    double acc = 0.0;
    const long long nq = n / 4, stride = (long long)gridDim.x * NT;
    long long q = blockIdx.x * (long long)NT + threadIdx.x;
    auto quad = [&](const float4 &x, const float4 &y) {
        acc += (double)x.x * (double)y.x;
        acc += (double)x.y * (double)y.y;
        acc += (double)x.z * (double)y.z;
        acc += (double)x.w * (double)y.w;
    };
    for (; q + (kQuads - 1) * stride < nq; q += kQuads * stride) {
        float4 x[kQuads], y[kQuads];
#pragma unroll
        for (int k = 0; k < kQuads; ++k) {
            x[k] = load4<VEC>(a, q + k * stride);
            y[k] = load4<VEC>(b, q + k * stride);
        }
#pragma unroll
        for (int k = 0; k < kQuads; ++k) quad(x[k], y[k]);
    }
    for (; q < nq; q += stride) quad(load4<VEC>(a, q), load4<VEC>(b, q));
    if (blockIdx.x == 0 && 4 * nq + threadIdx.x < n)
        acc += (double)a[4 * nq + threadIdx.x] * (double)b[4 * nq + threadIdx.x];
    finish_sum<NT>(acc, partial, arrived, out);
}

// ---------------------------------------------------------------------------
// Deterministic random boundary.
// Counter-based generator: the SplitMix64 output function (Steele, Lea and
// Flood, "Fast splittable pseudorandom number generators", OOPSLA 2014)
// applied to (seed, stream, counter); uniforms take the top 24 bits and
// normals come from the Box-Muller transform.
// ---------------------------------------------------------------------------
__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x)
{
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__device__ __forceinline__ float uniform01(uint64_t seed, uint64_t stream, uint64_t ctr)
{
    const uint64_t h = splitmix64(seed ^ splitmix64(stream * 0x632BE59BD9B4E019ull + ctr));
    return ((float)(h >> 40) + 0.5f) * (1.0f / 16777216.0f);
}

// Box-Muller in FP64, rounded once to FP32: the deviate is then the FP32
// rounding of a value any FP64 restatement computes to within a few FP64
// ulps, so a host restatement reproduces it bit for bit.
__device__ __forceinline__ float normal01(uint64_t seed, uint64_t stream, uint64_t ctr)
{
    const double u1 = (double)uniform01(seed, stream, 2 * ctr);
    const double u2 = (double)uniform01(seed, stream, 2 * ctr + 1);
    return (float)(sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2));
}

// Pad background.  For every pad cell take the nearest model-edge value, then
//   kind 0: add ramp_a * varVp * N(0,1) for every axis a in the pad, with
//           ramp_a = 1 - depth_a/nb  (random_boundary_bg,
//           src/modeling/modeling.cu:617-666)
//   kind 1: scale by 1 + ratio * ramp * U(-1,1), ramp = max_a ramp_a
// and clamp to [vlo, vhi].
__global__ void rbc_background_kernel(float *__restrict__ vp, int nzz, int nxx, int nyy, int ldz,
                                      int nb, int kind, float ratio, float varVp, float vlo,
                                      float vhi, uint64_t seed)
{
    const long long n = (long long)ldz * nxx * nyy;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
         c += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(c % ldz);
        const long long r = c / ldz;
        const int j = (int)(r % nxx), k = (int)(r / nxx);
        if (i >= nzz) continue;
        const bool inside = i >= nb && i < nzz - nb && j >= nb && j < nxx - nb && k >= nb && k < nyy - nb;
        if (inside) continue;
        const int ii = min(max(i, nb), nzz - nb - 1);
        const int jj = min(max(j, nb), nxx - nb - 1);
        const int kk = min(max(k, nb), nyy - nb - 1);
        float v = vp[ii + (long long)jj * ldz + (long long)kk * ldz * nxx];
        const int dz = pad_depth(i, nzz, nb), dx = pad_depth(j, nxx, nb), dy = pad_depth(k, nyy, nb);
        const uint64_t cell = (uint64_t)i + (uint64_t)nzz * ((uint64_t)j + (uint64_t)nxx * k);
        const float fnb = (float)nb;
        // every product and sum rounded on its own (no contraction), so that
        // FP32 arithmetic on the host reproduces the pad exactly
        if (kind == 0) {
            if (dx >= 0) v = __fadd_rn(v, __fmul_rn(__fmul_rn(1.0f - dx / fnb, varVp), normal01(seed, 1, cell)));
            if (dy >= 0) v = __fadd_rn(v, __fmul_rn(__fmul_rn(1.0f - dy / fnb, varVp), normal01(seed, 2, cell)));
            if (dz >= 0) v = __fadd_rn(v, __fmul_rn(__fmul_rn(1.0f - dz / fnb, varVp), normal01(seed, 3, cell)));
        } else {
            float ramp = 0.0f;
            if (dx >= 0) ramp = fmaxf(ramp, 1.0f - dx / fnb);
            if (dy >= 0) ramp = fmaxf(ramp, 1.0f - dy / fnb);
            if (dz >= 0) ramp = fmaxf(ramp, 1.0f - dz / fnb);
            const float u = __fsub_rn(__fmul_rn(2.0f, uniform01(seed, 4, cell)), 1.0f);
            v = __fmul_rn(v, __fadd_rn(1.0f, __fmul_rn(__fmul_rn(ratio, ramp), u)));
        }
        vp[c] = fminf(fmaxf(v, vlo), vhi);
    }
}

// Gaussian blobs (random_boundary_gp, src/modeling/modeling.cu:594-615): every
// cell outside the strict inner box visits, in order, the blobs near it and
// applies v += s A exp(-|x-c|^2 / (2 r^2)) followed by the clamp.  Blobs
// are truncated at 5 r (the omitted tail is below 4e-6 A).
struct Blob {
    float x, y, z, r, amp;  // centre [m], radius [m], signed amplitude [m/s]
};

// A block owns a brick of 32 x bx x by cells.  It keeps the blobs whose 5 r ball reaches the
// brick, in blob order, in shared memory; a warp then goes through its patches
// of 8 x 4 (z, x) cells and drops, 32 blobs at a time, those that do not reach
// the patch.
// Bound by instruction issue: about 60 blobs act on a cell.  301^3 cells, 8000
// blobs: 1.83 ms (2.32 ms with rows of 32 z cells as patches, 4.45 ms with a
// thread per cell going through host-built bins).
constexpr int kBrickZ = 32, kBrickThreads = 256, kBrickBlobs = 1024;

// Whether the 5 r ball of a blob reaches a box, with a margin for rounding.
__device__ __forceinline__ bool blob_reaches(const Blob &b, float z0, float z1, float x0, float x1, float y0, float y1)
{
    const float dz = fmaxf(fmaxf(z0 - b.z, b.z - z1), 0.0f), dx = fmaxf(fmaxf(x0 - b.x, b.x - x1), 0.0f),
                dy = fmaxf(fmaxf(y0 - b.y, b.y - y1), 0.0f), e = 5.001f * b.r;
    return dz * dz + dx * dx + dy * dy <= e * e;
}

__global__ void __launch_bounds__(kBrickThreads)
    rbc_blobs_kernel(float *__restrict__ vp, int nzz, int nxx, int nyy, int ldz, int nb, float dh,
                     const Blob *__restrict__ blobs, int nblob, float vlo, float vhi, int bx, int by)
{
    __shared__ Blob list[kBrickBlobs];
    __shared__ float inv_r[kBrickBlobs];
    __shared__ int warp_count[kBrickThreads / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int i0 = blockIdx.x * kBrickZ, j0 = blockIdx.y * bx, k0 = blockIdx.z * by;
    const int i1 = min(i0 + kBrickZ, nzz) - 1, j1 = min(j0 + bx, nxx) - 1, k1 = min(k0 + by, nyy) - 1;
    const float fnb = nb * dh;
    const float xmax = (nxx - 1) * dh, ymax = (nyy - 1) * dh, zmax = (nzz - 1) * dh;
    if (i0 * dh > fnb && i1 * dh < zmax - fnb && j0 * dh > fnb && j1 * dh < xmax - fnb && k0 * dh > fnb &&
        k1 * dh < ymax - fnb)
        return;  // no cell outside the strict inner box

    int n = 0;  // blobs in the list
    for (int b0 = 0; b0 < nblob; b0 += kBrickThreads) {
        // append the blobs of this pass that reach the brick
        Blob b;
        bool in = false;
        if (b0 + tid < nblob) {
            b = blobs[b0 + tid];
            in = blob_reaches(b, i0 * dh, i1 * dh, j0 * dh, j1 * dh, k0 * dh, k1 * dh);
        }
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) warp_count[warp] = __popc(m);
        __syncthreads();
        int at = n;
        for (int w = 0; w < kBrickThreads / 32; ++w) {
            if (w < warp) at += warp_count[w];
            n += warp_count[w];
        }
        if (in) {
            at += __popc(m & ((1u << lane) - 1u));
            list[at] = b;
            inv_r[at] = 1.0f / b.r;
        }
        __syncthreads();
        if (n <= kBrickBlobs - kBrickThreads && b0 + kBrickThreads < nblob) continue;
        // apply the list, patch by patch
        const int px = bx / 4;
        for (int patch = warp; patch < kBrickZ / 8 * px * by; patch += kBrickThreads / 32) {
            const int pi = i0 + patch % (kBrickZ / 8) * 8, pj = j0 + patch / (kBrickZ / 8) % px * 4,
                      k = k0 + patch / (kBrickZ / 8 * px);
            const int i = pi + (lane & 7), j = pj + (lane >> 3);
            const float X = j * dh, Y = k * dh, Z = i * dh;
            const bool mine = i <= i1 && j <= j1 && k <= k1 &&
                              !(X > fnb && X < xmax - fnb && Y > fnb && Y < ymax - fnb && Z > fnb && Z < zmax - fnb);
            if (!__any_sync(0xffffffffu, mine)) continue;
            const long long c = i + (long long)j * ldz + (long long)k * ldz * nxx;
            float v = mine ? vp[c] : 0.0f;
            for (int q0 = 0; q0 < n; q0 += 32) {
                const bool near = q0 + lane < n && blob_reaches(list[q0 + lane], pi * dh, (pi + 7) * dh, pj * dh,
                                                                (pj + 3) * dh, Y, Y);
                for (unsigned todo = __ballot_sync(0xffffffffu, near); todo; todo &= todo - 1) {
                    const int q = q0 + __ffs(todo) - 1;
                    const Blob bl = list[q];
                    const float ir = inv_r[q];
                    const float ex = (X - bl.x) * ir, ey = (Y - bl.y) * ir, ez = (Z - bl.z) * ir;
                    const float e2 = ex * ex + ey * ey + ez * ez;
                    if (e2 > 25.0f) continue;
                    v += bl.amp * expf(-0.5f * e2);
                    v = fminf(fmaxf(v, vlo), vhi);
                }
            }
            if (mine) vp[c] = v;
        }
        n = 0;
        __syncthreads();
    }
}

// Stencil coefficient (v * v) * cvel = dt^2 v^2 / dh^2 of every updated cell of
// the velocity slots, 0 on the 4-cell shell that is never updated.
__global__ void coeff_kernel(const float *__restrict__ vp, float *__restrict__ out, int nzz, int nxx, int nyy,
                             int ldz, int nslot, float cvel)
{
    for_cells(ldz, nxx, nyy * nslot, [&](int i, int j, int ks, long long r) {
        const int k = ks % nyy;
        const bool upd = i >= 4 && i < nzz - 4 && j >= 4 && j < nxx - 4 && k >= 4 && k < nyy - 4;
        const float v = vp[r * ldz + i];
        out[r * ldz + i] = upd ? v * v * cvel : 0.0f;
    });
}

// Range of a velocity model and its first value that is not a positive number.
// Positive floats order like their bits.
struct VelocityRange {
    unsigned long long bad;  // index, ~0 when there is none
    unsigned lo, hi;         // bits
};

__global__ void velocity_range_kernel(const float *__restrict__ v, long long n, VelocityRange *__restrict__ out)
{
    unsigned lo = 0x7f800000u, hi = 0u;
    unsigned long long bad = ~0ull;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
         c += (long long)gridDim.x * blockDim.x) {
        const float x = v[c];
        if (!isfinite(x) || x <= 0.0f) {
            bad = min(bad, (unsigned long long)c);
        } else {
            lo = min(lo, __float_as_uint(x));
            hi = max(hi, __float_as_uint(x));
        }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&out->lo, lo);
        atomicMax(&out->hi, hi);
    }
    if (bad != ~0ull) atomicMin(&out->bad, bad);
}

// Largest |v| in a pitched field restricted to the real cells (CFL check).
__global__ void max_abs_kernel(const float *__restrict__ v, int nzz, int nxx, int nplane, int ldz,
                               unsigned int *__restrict__ out_bits)
{
    float m = 0.0f;
    for_cells(nzz, nxx, nplane, [&](int i, int, int, long long r) { m = fmaxf(m, fabsf(v[r * ldz + i])); });
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out_bits, __float_as_uint(m));
}

}  // namespace fwi
