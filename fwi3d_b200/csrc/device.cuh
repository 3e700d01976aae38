// device.cuh -- PTX helpers (TMA, mbarrier), constants and argument structs
// shared by the stencil kernels.  sm_100a only.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fwi {

// 8th-order second-derivative weights, FP32 images of the reference's double
// literals (src/modeling/modeling.cuh:9-13): centre, then taps m = 1..4.
// The operator is  -W0 f0 + W1 (f1+f-1) - W2 (f2+f-2) + W3 (f3+f-3) - W4 (f4+f-4).
constexpr float W0 = 2.847222222222f;
constexpr float W1 = 1.600000000000f;
constexpr float W2 = 0.200000000000f;
constexpr float W3 = 0.025396825396f;
constexpr float W4 = 0.001785714285f;

constexpr int kMaxBatch = 64;      // shots per launch
constexpr int kMaxPad = 1024;      // largest pad width the damper table holds
// Image and illumination accumulate in reductions, which take what is below
// 2^-126 for 0.  Times 2^24 an addend that FP32 holds, the least being 2^-149, stays
// above that, and what a sum loses is below half of the least.
constexpr float kAccScale = 0x1p24f;
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s cap on any device wait

// Error bits the kernels raise in g_status (read back by the host).
constexpr unsigned kErrTimeout = 1u;

// Per-batch shot description, copied to the device once per batch.
struct BatchInfo {
    int nshot;                    // shots in this batch
    int R;                        // receivers of all shots together
    int ncell;                    // distinct receiver cells of all shots together
    int pad_;
    int src[kMaxBatch][3];        // source cell (i=z, j=x, k=y), padded indices
};

// Distinct receiver cells of a batch, sorted by the column (shot, col) of the
// tiling that owns them and by y plane.
struct CellLists {
    const int *below;             // [shots * columns][nyy + 1] place in the list of a column's first cell at or above a plane
    const long long *cell;        // [ncell] batch-flat cell index
};

// Progress of the items of a time-loop kernel: an item is one step of one
// column of one shot; it publishes the y planes it has stored.
// Every counter has a 128-byte line to itself: up to five columns poll it, and
// the line of several counters was what the hand-over between steps waited for
// (146 x 123 x 101 cells, forward: 10.4 us a step with counters side by side,
// 7.3 with one per 32-byte sector, 7.0 with one per line).
constexpr int kCounterStride = 16;

struct LoopProgress {
    unsigned long long *ticket;   // next item
    long long *done;              // [shot][step % ring][column] (kCounterStride apart): step * nyy + planes stored
    int ring;
    int shots;                    // shots whose steps interleave in the ticket order
};

// Forward time loop arguments (all leapfrog steps of every shot of a batch).
struct FwdArgs {
    int nzz, nxx, nyy, ldz;
    long long vol;                // device elements of one shot's field (pitched)
    int ntz, ncol;                // z tiles, columns (z tiles x x tiles)
    int nsteps, nt, tlag;         // steps, wavelet length, recording lag
    float idh3;                   // source / adjoint scaling 1/dh^3
    int nb;                       // pad width (damper tables)
    int vel_slots;                // 1: every shot reads velocity slot 0; B: shot s reads slot s
    float *F[2];                  // field pair (batch base): step t reads F[t & 1], overwrites the other
    const float *b1d;             // Cerjan 1-D table (ABC only)
    const float *wavelet;         // [nt]
    const BatchInfo *binfo;
    CellLists rec;
    float *seis_tm;               // [nt][ncell] samples of the receiver cells
    LoopProgress prog;
};

// Backward time loop arguments (source rebuild + adjoint + imaging).
struct BwdArgs {
    int nzz, nxx, nyy, ldz;
    long long vol;
    int ntz, ncol;
    int nsteps, nt;               // N = nt + tlag, wavelet and data length
    float gscale;                 // acc_scale / dt (gradient imaging condition)
    float idh3;
    int subtract_src;             // remove the source while rebuilding Ps
    int vel_slots;                // 1: every shot reads velocity slot 0; B: shot s reads slot s
    int acc_z0, acc_z1;           // box [acc_z0, acc_z1) x [acc_x0, acc_x1) x [acc_y0, acc_y1)
    int acc_x0, acc_x1;           // of the cells whose image and illumination accumulate;
    int acc_y0, acc_y1;           // the accumulators of every other cell keep their values
    int s0;                       // F[s0] holds the older of the two forward levels
    float *F[2];                  // source field: step t reads F[(s0 + t) & 1], overwrites the other
    float *Rf[2];                 // adjoint field: step t reads Rf[t & 1], overwrites the other
    float *image;                 // image or gradient accumulator, of cell (0, 0, 0) of the first shot
    long long to_illum;           // from there to the illumination
    int acc_ld;                   // pitches of the accumulators: x rows,
    long long acc_plane;          // y planes
    long long acc_shot;           // and shots
    float acc_scale;              // what is added is scaled by this
    int acc_direct;               // loads and stores instead of reductions in L2
    const float *wavelet;
    const BatchInfo *binfo;
    CellLists inj;
    const float *data_tm;         // [nt][ncell] adjoint sources of the receiver cells
    LoopProgress prog;
};

// ---------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ void fence_mbar_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Generic-proxy accesses of global memory (another CTA's stores, made visible
// by an acquire) before the TMA copies that follow.
__device__ __forceinline__ void fence_proxy_async_global()
{
    asm volatile("fence.proxy.async.global;" ::: "memory");
}

__device__ __forceinline__ long long ld_acquire_gpu(const long long *p)
{
    long long v;
    asm volatile("ld.acquire.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void red_add(float *p, float v)
{
    asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(p), "f"(v) : "memory");
}

__device__ __forceinline__ void red_add4(float *p, float a, float b, float c, float d)
{
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

__device__ __forceinline__ void st_release_gpu(long long *p, long long v)
{
    asm volatile("st.release.gpu.global.s64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

template <class T>
__device__ __forceinline__ T ld_acquire_cta(const T *p)
{
    static_assert(sizeof(T) == 4, "32-bit counters");
    T v;
    asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}

template <class T>
__device__ __forceinline__ void st_release_cta(T *p, T v)
{
    static_assert(sizeof(T) == 4, "32-bit counters");
    asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(p)), "r"(v) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for phase `parity` of an mbarrier, giving up after limit_ns.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint64_t limit_ns = kWaitLimitNs)
{
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_ns();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) return false;
    }
}

// 4-D tiled TMA load (z, x, y, shot) into shared memory, completing on bar.
// No multicast: every CTA fetches its own tiles from this GPU's memory.
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar,
                                            int c0, int c1, int c2, int c3)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(c0), "r"(c1), "r"(c2),
        "r"(c3)
        : "memory");
}

// 3-D tiled TMA load, completing on bar.  No multicast.
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1,
                                            int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}

// 2-D tiled TMA load, completing on bar.  No multicast.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(c0), "r"(c1)
        : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// ---------------------------------------------------------------------------
// tcgen05 (5th-generation tensor core) wrappers, cta_group::1.
// ---------------------------------------------------------------------------
// Tensor-memory allocation by one full warp; the address lands in *slot.
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor.  Bit 46 is the tcgen05 descriptor version.
// No swizzle: core matrices are 128 contiguous bytes.  K-major: 8 M/N rows x
// 16 bytes of K; lbo = byte stride between K halves, sbo = byte stride
// between 8-row groups.  MN-major: 8 K rows x 16 bytes of M/N; lbo = byte
// stride between 8-row K groups, sbo = byte stride between 8-element M/N
// groups.
// 32-byte swizzle (the pattern a SWIZZLE_32B TMA load writes: the 16-byte
// half of each 32-byte row flips with address bit 7): rows of 32 bytes.
// K-major (K = 16 BF16 per row): sbo = stride between 8-row groups, lbo
// unused.  MN-major (16 M/N elements per row, K along rows): lbo = stride
// between 16-element M/N groups, sbo = stride between 8-row K groups.
constexpr uint64_t kSwizzleNone = 0, kSwizzle32B = 6;  // layout type, bits 61..63

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo,
                                              uint64_t layout = kSwizzleNone)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (layout << 61);
}

// Instruction descriptor of kind::f16: D FP32, A and B BF16; a_mn / b_mn
// select the MN-major operand layout (bits 15 / 16), K-major otherwise.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n, bool a_mn = false, bool b_mn = false)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T, issued by one thread.
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrive on bar once every tcgen05 operation this thread issued has completed.
__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_addr(bar))
                 : "memory");
}

// 16 consecutive FP32 columns of the calling thread's TMEM lane; the
// registers are valid after tmem_wait_ld().
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Named barrier over `count` threads that also ANDs a predicate across them.
__device__ __forceinline__ bool bar_and(int id, int count, bool pred)
{
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred), "r"(id), "r"(count)
        : "memory");
    return r != 0;
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap *map)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// Distance into the pad along one axis, -1 inside (src/modeling/modeling.cu:408-431).
__device__ __forceinline__ int pad_depth(int i, int n, int nb)
{
    return i < nb ? i : (i >= n - nb ? n - 1 - i : -1);
}

}  // namespace fwi
