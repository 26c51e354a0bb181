// tcgen05 BF16 convolution kernels of the learned ambient-occlusion U-Net.
//
// Activation layout ("chunk-planar", CP): bf16 [B][C/8][H][W][8]. Every pixel
// of an 8-channel chunk is one 16-byte vector, so a TMA box of
// (10 pixels x 8 channels, 18 rows, chunks) lands in shared memory as
// [chunk][y][x][8] -- exactly the no-swizzle core-matrix layout the tensor
// core reads, with zero fill outside the image supplying the convolution's
// zero padding.
//
// Output tiles are 8 x 16 pixels (M = 128 rows of the implicit GEMM: row
// r = 8 * y + x). For tap (dy, dx) the A operand is the halo tile shifted by
// (dy, dx): rows 16 B apart along x, 8-row groups one halo row (160 B) apart,
// K chunks one 8-channel plane (2880 B) apart.
#pragma once

#include <cuda.h>
#include <cstdint>

namespace fra
{

constexpr int kTileW = 8;
constexpr int kTileH = 16;
constexpr int kHaloW = kTileW + 2;
constexpr int kRowBytes = kHaloW * 16;  // 160
constexpr int kMaxStages = 4;

struct ConvArgs
{
    int B, H, W;
    int tilesX, tilesY, numTiles;
    int c0, c1;          // input channels from map0 / map1 (multiples of 8); cin = c0 + c1
    int cout;            // output channels: multiple of 16, at most 128
    int stages;          // shared-memory pipeline depth (2..kMaxStages)
    int mb;              // M-blocks per tile: the tile is 8 x (16 * mb) pixels
    const uint16_t* wpacked;  // bf16 weights in the shared-memory layout (see pack_conv_weights)
    uint32_t wbytes;
    const float* bias;   // [cout] (forward) or null
    int backward;        // 0: out = relu(acc + bias); 1: out = acc * (mask > 0) (mask optional)
    uint16_t* out0;      // CP tensor receiving channels [0, co0)
    int co0;
    uint16_t* out1;      // CP tensor receiving channels [co0, cout), or null when co0 == cout
    const uint16_t* mask;  // CP tensor with cout channels (backward), or null
    const float* head;   // fused 1x1 head (forward, cout == 16): w[4][16], b[4]; or null
    float* ao;           // [B][2H][2W] sigmoid outputs of the head: sub-pixel (sy, sx) of block (y, x)
                         // is output k = 2 sy + sx
    const float* bgDepth;  // (B = 1) full-resolution depth: where it is FLT_MAX the head writes
    const float* bg16;     // bg16[(y & 3) * 4 + (x & 3)] instead (plain SSAO's background), or null
    int* status;         // bit 1: a pipeline wait timed out
};

// ---- weight gradients of every layer in one launch -------------------------------
// dW[co][ci][ky][kx] = sum_p dY[co][p] X[ci][p + (ky - 1, kx - 1)], K running over the
// pixels of 8 x 16 tiles. The tiles of a layer form nChains chains (tile mod nChains),
// each summed in one FP32 accumulator in tile order; a CTA runs several chains.
constexpr int kWgradMaxLayers = 10;
constexpr int kWgradYPlane = kTileW * kTileH * 16;  // 2048: 8 channels of a tile's dY
constexpr uint32_t kWgradSmem = 184u * 1024u;       // one CTA per SM, 2..4 stages

struct WgradLayer
{
    CUtensorMap mapX0, mapX1, mapDY;
    int tilesX, tilesY, numTiles;
    int c0, c1;          // X channels from mapX0 / mapX1; cin = c0 + c1 <= 96
    int cout;            // dY channels: 16, 32 or 64
    int kyRows;          // 1: rows (ky, ci), X loaded once per ky; 0: rows ci, ky by start address
    int nChains;
    int sets, bufs;      // accumulators of chains held at a time, and 2 when the next ones
                         // are filled while these are read out
    int stages;          // shared-memory pipeline depth
    int cta0, ctas;      // CTA cta0 + k runs the chains k, k + ctas, ...
    float* partial;      // [nChains][3 kx][cout][3 ky * cin + 1 (bias, kx = 1)]
};

struct WgradArgs
{
    WgradLayer layer[kWgradMaxLayers];
    int nLayers;
    int* status;
};

// Rows (ky, ci) unless they need three blocks of 128 (a row more for the bias): then
// rows ci and one MMA per tap is no more work.
constexpr bool wgrad_ky_rows(int cin) { return 3 * cin + 1 <= 256; }
// MMAs of a K step are 3 kx times this: row blocks, or the three ky.
__host__ __device__ constexpr int wgrad_units(int cin, bool kyRows) { return kyRows ? (3 * cin + 1 + 127) / 128 : 3; }
// Whether the last row block needs at most 64 rows.
__host__ __device__ constexpr bool wgrad_half_last(int cin, bool kyRows)
{
    return kyRows && 3 * cin + 1 - (wgrad_units(cin, true) - 1) * 128 <= 64;
}
__host__ __device__ constexpr uint32_t wgrad_plane_bytes(bool kyRows)
{
    return static_cast<uint32_t>((kTileH + (kyRows ? 0 : 2)) * kRowBytes);
}
// The constant plane behind X, up to the 128-byte boundary that a TMA copy starts on.
__host__ __device__ constexpr uint32_t wgrad_const_bytes(bool kyRows)
{
    return (wgrad_plane_bytes(kyRows) + 127u) & ~127u;
}
// Bytes of one pipeline stage: the X copies, the constant plane, dY.
__host__ __device__ constexpr uint32_t wgrad_stage_bytes(int cin, int cout, bool kyRows)
{
    return static_cast<uint32_t>((kyRows ? 3 : 1) * (cin / 8)) * wgrad_plane_bytes(kyRows) +
           wgrad_const_bytes(kyRows) + static_cast<uint32_t>(cout / 8) * kWgradYPlane;
}
// The A operand's 128-row blocks (16 planes each) are read whole, past the valid
// rows: the last stage needs this much shared memory behind its start.
constexpr uint32_t wgrad_a_window(int cin, bool kyRows)
{
    return (kyRows ? wgrad_units(cin, true) * 16u * wgrad_plane_bytes(true)
                   : 16u * wgrad_plane_bytes(false) + 2u * kRowBytes) + 64u;
}
// Floats of one chain's sums.
__host__ __device__ constexpr size_t wgrad_partial_floats(int cin, int cout)
{
    return static_cast<size_t>(3) * cout * (3 * cin + 1);
}

// ---- fused forward: the whole network in one cooperative launch ------------------
// Stages run in order with a grid-wide barrier after each: a convolution (its
// tiles spread over the persistent CTAs, weights re-loaded per layer, ring and
// TMEM buffers carried over), or an elementwise pooling / upsampling.
constexpr int kUnetMaxConvs = 10;
constexpr int kUnetMaxStages = 16;
enum UnetStageKind : int
{
    kStageConv = 0,
    kStagePool = 1,  // n output vectors of pool_vec(in, out, i, H, W)
    kStageUp = 2     // n output vectors of up_vec(in, out, i, H = h, W = w)
};

struct UnetConv
{
    CUtensorMap map0, map1;
    ConvArgs a;
};

struct UnetStage
{
    int kind, conv;  // conv: index into UnetArgs::conv
    const uint4* in;
    uint4* out;
    int n, H, W;
};

struct UnetArgs
{
    UnetConv conv[kUnetMaxConvs];
    UnetStage stage[kUnetMaxStages];
    int nStages;
    int ringStages;        // halo ring slots (every layer's tile fits one slot)
    uint32_t wRegion;      // shared bytes before the ring: the largest layer's weights
    uint32_t stageBytes;   // bytes of one ring slot
    uint32_t tmemCols;     // TMEM columns (power of two): the largest layer's two buffers
    unsigned* sync;        // [3] grid barrier count, generation, failure flag (zeroed before the launch)
    int* status;           // bit 4: a grid barrier timed out
    uint64_t waitNs;       // longest wait of a CTA at a grid barrier before it gives up
    int absentCta;         // tests of the bounded barrier: this CTA never arrives at the
                           // first barrier (it leaves the stage loop instead); -1 = none
};

// Launches the fused forward on `grid` co-resident CTAs (cooperative launch).
cudaError_t launch_unet_fwd(const UnetArgs& u, int grid, uint32_t smem, cudaStream_t st);
// CTAs of k_unet_fwd that fit on one SM with `smem` dynamic shared bytes.
int unet_fwd_ctas_per_sm(uint32_t smem);

// Shared-memory bytes of one launch.
uint32_t conv_smem_bytes(int cin, int cout, int stages, int mb);

// programmatic: launch as a programmatic dependent of the stream's previous
// kernel (the prologue overlaps its tail; outputs are read after griddepcontrol.wait).
void launch_conv3x3(const CUtensorMap& map0, const CUtensorMap& map1, const ConvArgs& a, int grid,
                    uint32_t smem, cudaStream_t st, bool programmatic);
void launch_wgrad(const WgradArgs& a, int grid, cudaStream_t st);

}  // namespace fra
