// tcgen05 BF16 implicit-GEMM 3x3 convolutions of the learned-AO U-Net:
// forward / backward-data (k_conv3x3) and backward-weights (k_wgrad).
//
// Both kernels are persistent and warp-specialised (192 threads):
//   warp 0      TMA producer (one lane): halo tiles into a shared-memory ring
//   warp 1      MMA issuer (the warp waits, one elected lane issues) and TMEM owner
//   warps 2..5  epilogue: TMEM -> registers -> global
#include <cfloat>
#include <cuda_bf16.h>

#include "fr_aonet_conv.cuh"
#include "fr_aonet_ew.cuh"
#include "fr_tc.cuh"

namespace fra
{
namespace
{

constexpr uint64_t kWaitNs = 2000000000ull;  // 2 s: far above any legitimate wait
constexpr uint32_t kSleepHintNs = 100000;     // longest hardware sleep of one poll
constexpr int kHeadParamsMax = 68;            // 1x1 head: w[4][16], b[4]

struct SyncState
{
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t tfull[2];
    uint64_t tempty[2];
    uint64_t wbar;
    uint64_t done;
    uint32_t tmem;
    int abort;
};

// Bounded wait. Gives up when another thread of the CTA aborted, or after kWaitNs
// (then it aborts the CTA and sets status bit 2).
__device__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort, int* status)
{
    if (frtc::mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = frtc::global_timer_ns();
    // sleep in hardware between polls so waiting threads leave the issue slots to the others
    while (!frtc::mbar_try_wait_sleep(bar, parity, kSleepHintNs))
    {
        if (*abort) return false;
        if (frtc::global_timer_ns() - t0 > kWaitNs)
        {
            *abort = 1;
            atomicOr(status, 2);
            return false;
        }
    }
    return true;
}

// The same for a converged warp whose lanes all wait (uniform result).
__device__ __forceinline__ bool warp_wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort, int* status)
{
    return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort, status));
}

// Barriers of one CTA: the halo ring, the two TMEM buffers, weights, done.
__device__ __forceinline__ void init_sync(SyncState& sy)
{
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < kMaxStages; ++s)
        {
            frtc::mbar_init(&sy.full[s], 1);
            frtc::mbar_init(&sy.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b)
        {
            frtc::mbar_init(&sy.tfull[b], 1);
            frtc::mbar_init(&sy.tempty[b], 4);
        }
        frtc::mbar_init(&sy.wbar, 1);
        frtc::mbar_init(&sy.done, 1);
        sy.abort = 0;
        frtc::fence_mbar_init();
    }
}

__device__ __forceinline__ uint32_t tmem_cols(int cols)
{
    return cols <= 32 ? 32u : cols <= 64 ? 64u : cols <= 128 ? 128u : cols <= 256 ? 256u : 512u;
}

__device__ __forceinline__ void decode_tile(int tile, int tilesX, int tilesY, int& b, int& tx, int& ty)
{
    const int per = tilesX * tilesY;
    b = tile / per;
    const int r = tile - b * per;
    ty = r / tilesX;
    tx = r - ty * tilesX;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Tiles are 8 x (16 * mb) pixels: mb M-blocks of 128 rows share one halo load,
// one pipeline stage and one accumulator buffer (mb * cout TMEM columns).

// The shared-memory ring of halo tiles, after the weight region.
struct ConvRing
{
    unsigned char* sW;      // the layer's packed weights
    unsigned char* sStage;  // ring slot i at sStage + i * stageBytes
    uint32_t stageBytes;
    int stages;
};

// Each role's running count of tiles (ring slots, TMEM buffers and barrier
// phases follow from it); kept across the layers of one CTA.
struct RoleCounters
{
    int issued = 0;  // TMA producer lane
    int mma = 0;     // MMA lane
    int epi = 0;     // epilogue threads
};

// One layer's tiles on this CTA: warp 0 lane 0 loads halo tiles, warp 1 issues
// the MMAs (after the weights, wbar phase wParity), warps 2..5 run the
// epilogue. The weights are already being loaded, bias / head are in shared memory.
__device__ __forceinline__ void conv_layer(const CUtensorMap* map0, const CUtensorMap* map1, const ConvArgs& a,
                                           const ConvRing& R, SyncState& sy, uint32_t tmem, uint32_t wParity,
                                           const float* sBias, const float* sHead, RoleCounters& rc)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cin = a.c0 + a.c1;
    const int MB = a.mb;
    const int tileH = kTileH * MB;
    const uint32_t planeBytes = static_cast<uint32_t>(kHaloW * (tileH + 2) * 16);
    const uint32_t loadBytes = static_cast<uint32_t>(cin / 8) * planeBytes;
    const uint32_t accCols = static_cast<uint32_t>(MB * a.cout);
    volatile int* abortp = &sy.abort;

    if (warp == 0)
    {
        if (lane == 0)
        {
            for (int tile = blockIdx.x; tile < a.numTiles; tile += gridDim.x, ++rc.issued)
            {
                const int s = rc.issued % R.stages;
                const uint32_t ph = (rc.issued / R.stages) & 1;
                if (rc.issued >= R.stages && !wait_or_abort(&sy.empty[s], ph ^ 1, abortp, a.status)) break;
                int b, tx, ty;
                decode_tile(tile, a.tilesX, a.tilesY, b, tx, ty);
                unsigned char* dst = R.sStage + s * R.stageBytes;
                frtc::mbar_expect_tx(&sy.full[s], loadBytes);
                frtc::tma_load_3d(dst, map0, 8 * (tx * kTileW - 1), ty * tileH - 1, b * (a.c0 / 8), &sy.full[s]);
                if (a.c1)
                    frtc::tma_load_3d(dst + (a.c0 / 8) * planeBytes, map1, 8 * (tx * kTileW - 1), ty * tileH - 1,
                                      b * (a.c1 / 8), &sy.full[s]);
            }
        }
    }
    else if (warp == 1)
    {
        const uint32_t idesc = frtc::idesc_bf16_f32(128, a.cout, 0, 0);
        const uint32_t wBase = frtc::smem_u32(R.sW);
        const uint32_t bLbo = static_cast<uint32_t>(a.cout) * 16u;
        // Descriptor constants hoisted out of the tile loop: per MMA only the
        // start addresses change (a few integer ops, so issue keeps up with
        // the tensor pipe).
        const uint64_t bHi = frtc::smem_desc_hi(bLbo, 128);
        const uint64_t aHi = frtc::smem_desc_hi(planeBytes, kRowBytes);
        const uint32_t bTapStride = static_cast<uint32_t>(cin / 8) * bLbo;
        const int kc = cin / 16;
        bool ok = warp_wait_or_abort(&sy.wbar, wParity, abortp, a.status);
        for (int tile = blockIdx.x; ok && tile < a.numTiles; tile += gridDim.x, ++rc.mma)
        {
            const int it = rc.mma;
            const int s = it % R.stages;
            if (!warp_wait_or_abort(&sy.full[s], (it / R.stages) & 1, abortp, a.status)) break;
            const int buf = it & 1;
            if (it >= 2 && !warp_wait_or_abort(&sy.tempty[buf], ((it >> 1) & 1) ^ 1, abortp, a.status)) break;
            frtc::tc_fence_after();
            const uint32_t stageAddr = frtc::smem_u32(R.sStage + s * R.stageBytes);
            if (frtc::elect_one())
            {
                for (int mb = 0; mb < MB; ++mb)
                {
                    const uint32_t d = tmem + static_cast<uint32_t>(buf) * accCols + static_cast<uint32_t>(mb * a.cout);
                    const uint32_t aBase = stageAddr + static_cast<uint32_t>(mb * kTileH) * kRowBytes;
#pragma unroll
                    for (int t = 0; t < 9; ++t)
                    {
                        const uint32_t aTap = aBase + static_cast<uint32_t>(((t / 3) * kHaloW + t % 3) * 16);
                        const uint32_t bTap = wBase + static_cast<uint32_t>(t) * bTapStride;
                        for (int j = 0; j < kc; ++j)
                        {
                            const uint64_t ad = aHi | ((aTap + static_cast<uint32_t>(2 * j) * planeBytes) >> 4);
                            const uint64_t bd = bHi | ((bTap + static_cast<uint32_t>(2 * j) * bLbo) >> 4);
                            frtc::mma_bf16(d, ad, bd, idesc, (t | j) != 0);
                        }
                    }
                }
                frtc::mma_commit(&sy.empty[s]);
                frtc::mma_commit(&sy.tfull[buf]);
            }
            __syncwarp();
        }
    }
    else
    {
        const int q = warp & 3;  // TMEM lane quarter of this warp
        const int row = q * 32 + lane;
        const int lx = row & 7, ly = row >> 3;
        const int co8 = a.co0 / 8;
        const int c1n = (a.cout - a.co0) / 8;
        const uint32_t HW = static_cast<uint32_t>(a.H) * static_cast<uint32_t>(a.W);
        for (int tile = blockIdx.x; tile < a.numTiles; tile += gridDim.x, ++rc.epi)
        {
            const int it = rc.epi;
            const int buf = it & 1;
            int ok = 1;
            if (lane == 0) ok = wait_or_abort(&sy.tfull[buf], (it >> 1) & 1, abortp, a.status);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            frtc::tc_fence_after();
            int b, tx, ty;
            decode_tile(tile, a.tilesX, a.tilesY, b, tx, ty);
            const int x = tx * kTileW + lx;
            for (int mb = 0; mb < MB; ++mb)
            {
                const int y = ty * tileH + mb * kTileH + ly;
                const bool valid = x < a.W && y < a.H;
                const uint32_t pix = static_cast<uint32_t>(y) * static_cast<uint32_t>(a.W) + static_cast<uint32_t>(x);
                const uint32_t tb = tmem + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf) * accCols +
                                    static_cast<uint32_t>(mb * a.cout);
                float z[4] = {0.f, 0.f, 0.f, 0.f};
                for (int g = 0; g < a.cout / 16; ++g)
                {
                    float v[16];
                    frtc::tmem_ld16(tb + g * 16, v);
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                    {
                        const int cc = 2 * g + h;
                        float o[8];
                        if (!a.backward)
                        {
#pragma unroll
                            for (int e = 0; e < 8; ++e) o[e] = fmaxf(v[8 * h + e] + sBias[cc * 8 + e], 0.f);
                        }
                        else
                        {
#pragma unroll
                            for (int e = 0; e < 8; ++e) o[e] = v[8 * h + e];
                            if (a.mask && valid)
                            {
                                const uint32_t moff = ((static_cast<uint32_t>(b) * (a.cout / 8) + cc) * HW + pix) * 8;
                                const uint4 m = *reinterpret_cast<const uint4*>(a.mask + moff);
                                const uint32_t mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                                for (int e = 0; e < 8; ++e)
                                {
                                    const float mv = (e & 1) ? bf16_hi(mw[e >> 1]) : bf16_lo(mw[e >> 1]);
                                    if (!(mv > 0.f)) o[e] = 0.f;
                                }
                            }
                        }
                        uint4 pk;
                        pk.x = pack_bf16x2(o[0], o[1]);
                        pk.y = pack_bf16x2(o[2], o[3]);
                        pk.z = pack_bf16x2(o[4], o[5]);
                        pk.w = pack_bf16x2(o[6], o[7]);
                        if (a.head)
                        {
                            const uint32_t pw[4] = {pk.x, pk.y, pk.z, pk.w};
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                            {
                                const float hv = (e & 1) ? bf16_hi(pw[e >> 1]) : bf16_lo(pw[e >> 1]);
#pragma unroll
                                for (int k = 0; k < 4; ++k) z[k] += sHead[k * 16 + cc * 8 + e] * hv;
                            }
                        }
                        if (valid)
                        {
                            if (cc < co8)
                                *reinterpret_cast<uint4*>(
                                    a.out0 + ((static_cast<uint32_t>(b) * co8 + cc) * HW + pix) * 8) = pk;
                            else if (a.out1)
                                *reinterpret_cast<uint4*>(
                                    a.out1 + ((static_cast<uint32_t>(b) * c1n + (cc - co8)) * HW + pix) * 8) = pk;
                        }
                    }
                }
                if (a.head && valid)
                {
                    // the block's four sub-pixels of the full-resolution AO
                    const uint32_t W2 = 2u * static_cast<uint32_t>(a.W);
                    float* o = a.ao + static_cast<uint32_t>(b) * 4u * HW + (2u * static_cast<uint32_t>(y)) * W2 +
                               2u * static_cast<uint32_t>(x);
                    float v[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) v[k] = 1.f / (1.f + expf(-(z[k] + sHead[64 + k])));
                    if (a.bg16)
                    {
                        // background pixels: the plain SSAO's per-noise-cell value
                        const uint32_t X0 = 2u * static_cast<uint32_t>(x), Y0 = 2u * static_cast<uint32_t>(y);
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                        {
                            const uint32_t px = X0 + (k & 1), py = Y0 + (k >> 1);
                            if (a.bgDepth[py * W2 + px] == FLT_MAX) v[k] = a.bg16[(py & 3u) * 4u + (px & 3u)];
                        }
                    }
                    o[0] = v[0];
                    o[1] = v[1];
                    o[W2] = v[2];
                    o[W2 + 1] = v[3];
                }
            }
            frtc::tc_fence_before();
            __syncwarp();
            if (lane == 0) frtc::mbar_arrive(&sy.tempty[buf]);
        }
    }
}

__global__ void __launch_bounds__(192) k_conv3x3(const __grid_constant__ CUtensorMap map0,
                                                 const __grid_constant__ CUtensorMap map1, const ConvArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ SyncState sy;
    __shared__ float sBias[128];
    __shared__ float sHead[kHeadParamsMax];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cin = a.c0 + a.c1;
    const int tileH = kTileH * a.mb;
    const uint32_t planeBytes = static_cast<uint32_t>(kHaloW * (tileH + 2) * 16);
    const uint32_t wAligned = (a.wbytes + 1023u) & ~1023u;
    const uint32_t stageBytes = ((static_cast<uint32_t>(cin / 8) * planeBytes) + 1023u) & ~1023u;
    const ConvRing R{smem, smem + wAligned, stageBytes, a.stages};
    const uint32_t allocCols = tmem_cols(2 * a.mb * a.cout);

    // Prologue, independent of the previous kernel's outputs: barriers, TMEM,
    // the weights (never written by the kernel launched just before).
    init_sync(sy);
    if (warp == 1) frtc::tmem_alloc(&sy.tmem, allocCols);
    frtc::tc_fence_before();
    __syncthreads();
    frtc::tc_fence_after();
    if (threadIdx.x == 0)
    {
        frtc::mbar_expect_tx(&sy.wbar, a.wbytes);
        frtc::bulk_load(R.sW, a.wpacked, a.wbytes, &sy.wbar);
    }
    // From here on the previous kernel's outputs are read (no-op without a programmatic launch).
    griddep_wait();
    for (int i = threadIdx.x; i < a.cout; i += blockDim.x) sBias[i] = a.bias ? a.bias[i] : 0.f;
    if (a.head && threadIdx.x < kHeadParamsMax) sHead[threadIdx.x] = a.head[threadIdx.x];
    __syncthreads();
    const uint32_t tmem = sy.tmem;
    RoleCounters rc;
    conv_layer(&map0, &map1, a, R, sy, tmem, 0, sBias, sHead, rc);
    if (warp == 0 && lane == 0)
    {
        // Every issued copy must land before the CTA exits.
        for (int i = rc.issued - R.stages; i < rc.issued; ++i)
            if (i >= 0) frtc::mbar_wait(&sy.full[i % R.stages], (i / R.stages) & 1, kWaitNs);
        frtc::mbar_wait(&sy.wbar, 0, kWaitNs);
    }
    else if (warp == 1)
    {
        // All MMAs of the elected lane complete before TMEM is released.
        if (frtc::elect_one())
        {
            frtc::mma_commit(&sy.done);
            frtc::mbar_wait(&sy.done, 0, kWaitNs);
            griddep_launch();
        }
        __syncwarp();
    }
    frtc::tc_fence_before();
    __syncthreads();
    if (warp == 1)
    {
        frtc::tc_fence_after();
        frtc::tmem_dealloc(tmem, allocCols);
    }
}

// Grid-wide barrier of the fused forward (all CTAs co-resident: cooperative
// launch). A CTA whose pipeline gave up raises the failure flag before it
// arrives; a barrier that waits longer than waitNs raises it too. Returns false
// when the flag is set (every CTA then leaves the stage loop).
__device__ bool grid_barrier(unsigned* sync, int* status, volatile int* abortp, uint64_t waitNs)
{
    __shared__ int failed;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        if (*abortp) atomicExch(sync + 2, 1u);
        // this CTA's stores are ordered before the other CTAs' later TMA reads
        frtc::fence_proxy_async_global();
        __threadfence();
        volatile unsigned* gen = sync + 1;
        const unsigned g = *gen;
        __threadfence();  // the generation is read before this CTA arrives
        if (atomicAdd(sync, 1u) == gridDim.x - 1)
        {
            atomicExch(sync, 0u);
            __threadfence();
            atomicAdd(sync + 1, 1u);
        }
        else
        {
            const uint64_t t0 = frtc::global_timer_ns();
            while (*gen == g)
            {
                __nanosleep(256);
                if (frtc::global_timer_ns() - t0 > waitNs)
                {
                    atomicOr(status, 4);
                    atomicExch(sync + 2, 1u);
                    break;
                }
            }
        }
        __threadfence();
        frtc::fence_proxy_async_global();
        failed = *reinterpret_cast<volatile unsigned*>(sync + 2) != 0u;
    }
    __syncthreads();
    return !failed;
}

// The whole U-Net forward in one launch: one CTA per SM runs every stage of
// U.stage in order, with a grid barrier after each.
__global__ void __launch_bounds__(192, 1) k_unet_fwd(const __grid_constant__ UnetArgs U)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ SyncState sy;
    __shared__ float sBias[128];
    __shared__ float sHead[kHeadParamsMax];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    init_sync(sy);
    if (warp == 1) frtc::tmem_alloc(&sy.tmem, U.tmemCols);
    frtc::tc_fence_before();
    __syncthreads();
    frtc::tc_fence_after();
    const uint32_t tmem = sy.tmem;
    const ConvRing R{smem, smem + U.wRegion, U.stageBytes, U.ringStages};
    RoleCounters rc;
    int convs = 0;
    const int nthreads = gridDim.x * blockDim.x;
    for (int st = 0; st < U.nStages; ++st)
    {
        const UnetStage& S = U.stage[st];
        if (S.kind == kStageConv)
        {
            const UnetConv& C = U.conv[S.conv];
            // the previous layer's MMAs have all completed (its epilogue ran): the
            // weight region is free
            if (threadIdx.x == 0)
            {
                frtc::mbar_expect_tx(&sy.wbar, C.a.wbytes);
                frtc::bulk_load(R.sW, C.a.wpacked, C.a.wbytes, &sy.wbar);
            }
            for (int i = threadIdx.x; i < C.a.cout; i += blockDim.x) sBias[i] = C.a.bias ? C.a.bias[i] : 0.f;
            if (C.a.head && threadIdx.x < kHeadParamsMax) sHead[threadIdx.x] = C.a.head[threadIdx.x];
            __syncthreads();
            conv_layer(&C.map0, &C.map1, C.a, R, sy, tmem, static_cast<uint32_t>(convs & 1), sBias, sHead, rc);
            ++convs;
        }
        else
        {
            for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < S.n; i += nthreads)
            {
                if (S.kind == kStagePool)
                    pool_vec(S.in, S.out, i, S.H, S.W);
                else
                    up_vec(S.in, S.out, i, S.H, S.W);
            }
        }
        // the test hook: a CTA that never arrives (its stage is complete, nothing in flight)
        if (st == 0 && static_cast<int>(blockIdx.x) == U.absentCta) break;
        if (!grid_barrier(U.sync, U.status, &sy.abort, U.waitNs)) break;
    }
    if (warp == 0 && lane == 0)
    {
        // every issued copy has landed before the CTA exits
        for (int i = rc.issued - R.stages; i < rc.issued; ++i)
            if (i >= 0) frtc::mbar_wait(&sy.full[i % R.stages], (i / R.stages) & 1, kWaitNs);
        if (convs > 0) frtc::mbar_wait(&sy.wbar, static_cast<uint32_t>((convs - 1) & 1), kWaitNs);
    }
    else if (warp == 1)
    {
        if (frtc::elect_one())
        {
            frtc::mma_commit(&sy.done);
            frtc::mbar_wait(&sy.done, 0, kWaitNs);
        }
        __syncwarp();
    }
    frtc::tc_fence_before();
    __syncthreads();
    if (warp == 1)
    {
        frtc::tc_fence_after();
        frtc::tmem_dealloc(tmem, U.tmemCols);
    }
}

// One tile's MMAs: 8 K steps of 16 pixels (two tile rows), each UNITS x 3 kx, unrolled
// with constant address steps; the last row block may have M = 64 (idescLast).
template <int UNITS>
__device__ __forceinline__ void wgrad_tile_mmas(uint32_t set, uint32_t cout, uint32_t xLo, uint32_t aHi, uint32_t unitStep,
                                                uint32_t yLo, uint32_t bHi, uint32_t idesc, uint32_t idescLast,
                                                uint32_t more)
{
#pragma unroll
    for (int j = 0; j < kTileH / 2; ++j)
#pragma unroll
        for (int u = 0; u < UNITS; ++u)
#pragma unroll
            for (int kx = 0; kx < 3; ++kx)  // the next kx: 16 bytes further
                frtc::mma_bf16_lohi(set + static_cast<uint32_t>(u * 3 + kx) * cout,
                                    xLo + u * unitStep + static_cast<uint32_t>(j * 2 * kRowBytes / 16 + kx), aHi,
                                    yLo + static_cast<uint32_t>(j * 16), bHi, u == UNITS - 1 ? idescLast : idesc,
                                    j == 0 ? more : 1u);
}

// Every layer's weight gradient in one launch (WgradArgs). Rows of the A operand are
// input channels, columns output channels, K the tile's pixels. With few input
// channels the three ky are rows too (X is loaded three times, one row further each
// time, so rows (ky, ci) are adjacent planes) and kx is a start address 16 bytes
// further: 24 MMAs cover the nine taps of a tile where one M = 128 MMA per tap took
// 72, each mostly fetching rows of zeros. K steps are outermost, so consecutive MMAs
// add to different accumulators. A tile's sums go to the accumulator of its chain
// (tile mod nChains), in tile order: which pixels meet in one FP32 sum does not
// depend on how the chains are dealt to CTAs. Bound by the MMAs (47 cycles each for
// 128 rows, 33 for 64: the operand fetch) and, on the small levels, where a chain is
// one tile, by storing the accumulators (about 500 cycles per 16 columns). One X copy
// with the ky rows interleaved in shared memory needs the bias as a fourth
// accumulator, 32 MMAs instead of 24, and measured 105 us against 84. At 16 x 256 x 256
// this kernel takes 67 us.
__global__ void __launch_bounds__(192) k_wgrad(const __grid_constant__ WgradArgs U)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ SyncState sy;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int L = 0;
    while (L + 1 < U.nLayers && static_cast<int>(blockIdx.x) >= U.layer[L + 1].cta0) ++L;
    const WgradLayer& a = U.layer[L];
    const int k0 = blockIdx.x - a.cta0;
    // the loops' parameters in registers: read again from the parameter bank after
    // every barrier wait, and with a division for the ring slot, they cost 350 cycles a tile
    const int cin = a.c0 + a.c1, cout = a.cout, nch = a.nChains, ctas = a.ctas, numTiles = a.numTiles;
    const int stages = a.stages, sets = a.sets, bufs = a.bufs;
    const bool kyRows = a.kyRows != 0;
    const int copies = kyRows ? 3 : 1;                               // X copies, one per ky
    const int xRows = kTileH + (kyRows ? 0 : 2);                     // rows of a copy
    const uint32_t plane = static_cast<uint32_t>(xRows * kRowBytes);
    const uint32_t xBytes = static_cast<uint32_t>(cin / 8) * plane;  // one copy
    const int units = wgrad_units(cin, kyRows);                      // row blocks, or ky
    const bool half = wgrad_half_last(cin, kyRows);                  // the last row block has M = 64
    const uint32_t unitStep = kyRows ? 16u * plane : static_cast<uint32_t>(kRowBytes);
    const uint32_t constBytes = wgrad_const_bytes(kyRows);
    const uint32_t stageBytes = wgrad_stage_bytes(cin, cout, kyRows);
    const int setCols = units * 3 * cout;
    const uint32_t allocCols = tmem_cols(bufs * sets * setCols);

    // The plane after X's is constant in every stage: 1.0 in channel 0 (its accumulator
    // row is the bias gradient), else zero.
    for (int s = 0; s < stages; ++s)
    {
        uint32_t* p = reinterpret_cast<uint32_t*>(smem + s * stageBytes + copies * xBytes);
        for (int i = threadIdx.x; i < static_cast<int>(plane) / 4; i += blockDim.x) p[i] = (i & 3) == 0 ? 0x3F80u : 0u;
    }
    frtc::fence_proxy_async_smem();
    init_sync(sy);
    if (warp == 1) frtc::tmem_alloc(&sy.tmem, allocCols);
    frtc::tc_fence_before();
    __syncthreads();
    frtc::tc_fence_after();
    const uint32_t tmem = sy.tmem;
    volatile int* abortp = &sy.abort;
    griddep_wait();
    // this CTA's chains k0, k0 + ctas, ... in groups of `sets`; a group's tiles go
    // round by round (one tile of each chain), which every role walks alike
    const int mine = (nch - 1 - k0) / ctas + 1;
    const int rounds = (numTiles + nch - 1) / nch;

    if (warp == 0)
    {
        if (lane == 0)
        {
            const uint32_t loadBytes = copies * xBytes + static_cast<uint32_t>(cout / 8) * kWgradYPlane;
            int issued = 0, s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int c0 = 0; ok && c0 < mine; c0 += sets)
                for (int r = 0; ok && r < rounds; ++r)
                    for (int c = c0; c < min(c0 + sets, mine); ++c)
                    {
                        const int tile = k0 + c * ctas + r * nch;
                        if (tile >= numTiles) break;
                        ok = issued < stages || wait_or_abort(&sy.empty[s], ph ^ 1, abortp, U.status);
                        if (!ok) break;
                        int b, tx, ty;
                        decode_tile(tile, a.tilesX, a.tilesY, b, tx, ty);
                        unsigned char* dst = smem + s * stageBytes;
                        frtc::mbar_expect_tx(&sy.full[s], loadBytes);
                        for (int ky = 0; ky < copies; ++ky, dst += xBytes)
                        {
                            frtc::tma_load_3d(dst, &a.mapX0, 8 * (tx * kTileW - 1), ty * kTileH - 1 + ky,
                                              b * (a.c0 / 8), &sy.full[s]);
                            if (a.c1)
                                frtc::tma_load_3d(dst + (a.c0 / 8) * plane, &a.mapX1, 8 * (tx * kTileW - 1),
                                                  ty * kTileH - 1 + ky, b * (a.c1 / 8), &sy.full[s]);
                        }
                        frtc::tma_load_3d(dst + constBytes, &a.mapDY, 8 * tx * kTileW, ty * kTileH, b * (cout / 8),
                                          &sy.full[s]);
                        ++issued;
                        if (++s == stages) s = 0, ph ^= 1;
                    }
            // every issued copy lands before the CTA exits
            for (int i = issued - stages; i < issued; ++i)
                if (i >= 0) frtc::mbar_wait(&sy.full[i % stages], (i / stages) & 1, kWaitNs);
        }
    }
    else if (warp == 1)
    {
        const uint32_t idesc = frtc::idesc_bf16_f32(128, cout, 1, 1);
        const uint32_t idescLast = half ? frtc::idesc_bf16_f32(64, cout, 1, 1) : idesc;
        // both operands MN-major: K core matrices (8 pixels of a row) one row apart,
        // groups of 8 rows / columns (channels) one plane apart
        const uint64_t aDesc = frtc::smem_desc_hi(kRowBytes, plane);
        constexpr uint64_t bDesc = frtc::smem_desc_hi(128u, kWgradYPlane);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int c0 = 0, g = 0; ok && c0 < mine; c0 += sets, ++g)
        {
            const int buf = bufs == 2 ? g & 1 : 0;
            const int use = bufs == 2 ? g >> 1 : g;  // earlier groups in this buffer
            if (use > 0 && !warp_wait_or_abort(&sy.tempty[buf], (use - 1) & 1, abortp, U.status)) break;
            frtc::tc_fence_after();
            for (int r = 0; ok && r < rounds; ++r)
                for (int c = c0; c < min(c0 + sets, mine); ++c)
                {
                    if (k0 + c * ctas + r * nch >= numTiles) break;
                    ok = warp_wait_or_abort(&sy.full[s], ph, abortp, U.status);
                    if (!ok) break;
                    frtc::tc_fence_after();
                    const uint32_t xb = frtc::smem_u32(smem + s * stageBytes);
                    const uint32_t yb = xb + copies * xBytes + constBytes;
                    const uint32_t set = tmem + static_cast<uint32_t>((buf * sets + c - c0) * setCols);
                    if (frtc::elect_one())
                    {
                        const uint32_t xLo = static_cast<uint32_t>(aDesc) | (xb >> 4);
                        const uint32_t yLo = static_cast<uint32_t>(bDesc) | (yb >> 4);
                        const uint32_t aHi = static_cast<uint32_t>(aDesc >> 32), bHi = static_cast<uint32_t>(bDesc >> 32);
                        if (units == 1)
                            wgrad_tile_mmas<1>(set, cout, xLo, aHi, 0u, yLo, bHi, idesc, idescLast, r > 0);
                        else if (units == 2)
                            wgrad_tile_mmas<2>(set, cout, xLo, aHi, unitStep / 16, yLo, bHi, idesc, idescLast, r > 0);
                        else
                            wgrad_tile_mmas<3>(set, cout, xLo, aHi, unitStep / 16, yLo, bHi, idesc, idescLast, r > 0);
                        frtc::mma_commit(&sy.empty[s]);
                    }
                    __syncwarp();
                    if (++s == stages) s = 0, ph ^= 1;
                }
            if (frtc::elect_one()) frtc::mma_commit(&sy.tfull[buf]);
            __syncwarp();
        }
        if (frtc::elect_one())
        {
            frtc::mma_commit(&sy.done);
            frtc::mbar_wait(&sy.done, 0, kWaitNs);
        }
        __syncwarp();
    }
    else
    {
        const int q = warp & 3;
        const int rows = 3 * cin + 1;  // (ky, ci), then the bias
        for (int c0 = 0, g = 0; c0 < mine; c0 += sets, ++g)
        {
            const int buf = bufs == 2 ? g & 1 : 0;
            const int use = bufs == 2 ? g >> 1 : g;
            int ok = 1;
            if (lane == 0) ok = wait_or_abort(&sy.tfull[buf], use & 1, abortp, U.status);
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;  // the status word is set: the gradients are not used
            frtc::tc_fence_after();
            for (int c = c0; c < min(c0 + sets, mine); ++c)
            {
                float* part = a.partial + static_cast<size_t>(k0 + c * ctas) * wgrad_partial_floats(cin, cout);
                const uint32_t set = tmem + (static_cast<uint32_t>(q * 32) << 16) +
                                     static_cast<uint32_t>((buf * sets + c - c0) * setCols);
                for (int u = 0; u < units; ++u)
                {
                    // this thread's accumulator row: (ky, ci) or, just after the channels, the bias
                    // (M = 64: 16 rows at the start of each warp's 32 lanes)
                    const bool h = half && u == units - 1;
                    const int m = (kyRows ? u * 128 : 0) + (h ? q * 16 : q * 32) + lane;
                    const int nRows = kyRows ? 3 * cin : cin;
                    const bool bias = m == nRows && (kyRows || u == 0);
                    const int row = bias ? 3 * cin : kyRows ? m : u * cin + m;
                    const bool live = (bias || m < nRows) && (!h || lane < 16);
                    for (int kx = 0; kx < 3; ++kx)
                        for (int n0 = 0; n0 < cout; n0 += 16)
                        {
                            float v[16];
                            frtc::tmem_ld16(set + static_cast<uint32_t>((u * 3 + kx) * cout + n0), v);
                            if (live)
                            {
#pragma unroll
                                for (int i = 0; i < 16; ++i)
                                    part[(static_cast<size_t>(kx) * cout + n0 + i) * rows + row] = v[i];
                            }
                            __syncwarp();
                        }
                }
            }
            frtc::tc_fence_before();
            __syncwarp();
            if (lane == 0) frtc::mbar_arrive(&sy.tempty[buf]);
        }
    }
    frtc::tc_fence_before();
    __syncthreads();
    if (warp == 1)
    {
        frtc::tc_fence_after();
        frtc::tmem_dealloc(tmem, allocCols);
    }
}

}  // namespace

// Opt-in limit for the dynamic shared memory of both kernels: the 227 KiB
// per-block maximum minus room for their static shared memory.
constexpr int kMaxDynSmem = 220 * 1024;

uint32_t conv_smem_bytes(int cin, int cout, int stages, int mb)
{
    const uint32_t wbytes = 9u * cin * cout * 2u;
    const uint32_t w = (wbytes + 1023u) & ~1023u;
    const uint32_t plane = static_cast<uint32_t>(kHaloW * (kTileH * mb + 2) * 16);
    const uint32_t stage = (static_cast<uint32_t>(cin / 8) * plane + 1023u) & ~1023u;
    return w + stage * stages;
}

void launch_conv3x3(const CUtensorMap& map0, const CUtensorMap& map1, const ConvArgs& a, int grid, uint32_t smem,
                    cudaStream_t st, bool programmatic)
{
    static bool attr = false;
    if (!attr)
    {
        cudaFuncSetAttribute(k_conv3x3, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
        attr = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(192);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = programmatic ? 1 : 0;
    cudaLaunchKernelEx(&cfg, k_conv3x3, map0, map1, a);
}

void unet_attributes()
{
    static bool attr = false;
    if (!attr)
    {
        cudaFuncSetAttribute(k_unet_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
        attr = true;
    }
}

int unet_fwd_ctas_per_sm(uint32_t smem)
{
    unet_attributes();
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_unet_fwd, 192, smem) != cudaSuccess) return 0;
    return nb;
}

cudaError_t launch_unet_fwd(const UnetArgs& u, int grid, uint32_t smem, cudaStream_t st)
{
    unet_attributes();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(192);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_unet_fwd, u);
}

void launch_wgrad(const WgradArgs& a, int grid, cudaStream_t st)
{
    static bool attr = false;
    if (!attr)
    {
        cudaFuncSetAttribute(k_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynSmem);
        attr = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(192);
    cfg.dynamicSmemBytes = kWgradSmem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_wgrad, a);
}

}  // namespace fra
