// Learned seam blend: tcgen05 (5th-generation tensor core) implicit-GEMM 3x3
// convolutions, forward and backward, the U-Net-lite built from them, its
// loss and Adam, all on the GPU.  No reference counterpart (the reference
// blends overlaps with SeamBlend.cpp:549-587 only); the network's shape is in
// include/image360_b200_blendnet.h.
//
// Convolution as GEMM: D[pixel][cout] += A[pixel][(tap, cin)] * B[cout][(tap,
// cin)], M = 128 pixels of 8 columns x 16 rows, K in steps of 16.  A tile's
// input halo sits in shared memory as TMA writes it, a pixel's channels a
// swizzled row; the swizzle is a function of the address, so the A operand of
// any tap is the same buffer from another start address - no im2col copy - and
// with the 16 rows of a block J apart one operand serves three taps of three
// blocks, N = 3 cout.  fp32 accumulators live in TMEM in two sets, so the
// epilogue of one tile overlaps the MMAs of the next, and the halos in a ring
// of stages, so the next load overlaps both (see k_conv3x3).
//
// Weight gradient: D[(dy, cin)][(dx, cout)] += X[q + dy][cin] * G[q - dx][cout]
// summed over pixels q (K), all nine taps in one MMA per 16 pixels; each CTA
// owns a share of the pixels and writes fp32 partial sums that a small kernel
// reduces (see k_conv3x3_wgrad).
#include "common.cuh"
#include "render_plan.hpp"
#include "tc_common.cuh"
#include "../../include/image360_b200_blendnet.h"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <random>
#include <vector>

namespace i360b
{
namespace
{
using bf16 = __nv_bfloat16;

constexpr int kTileX = 128;                // weight-gradient widths are multiples of this
constexpr long long kWaitSpins = 1ll << 26;  // bounded mbarrier waits
constexpr int kSlots = 4;
constexpr float kInScale = 1.0f / 32768.0f;

enum
{
    LD_PLAIN = 0,
    LD_CONCAT = 1,
    LD_SPLIT = 2  // 96 channels of one tensor
};
enum
{
    EP_RELU = I360B_CONV_BIAS_RELU,
    EP_LOGITS = I360B_CONV_LOGITS,
    EP_MASK = I360B_CONV_MASK,
    EP_RAW = I360B_CONV_RAW,
    EP_COMPOSITE = 4,
    EP_RELU_POOL = 5,  // EP_RELU, and its 2x2 averages
    EP_RAW_UP = 6      // the first 32 channels raw, 2x2 sums of the others masked
};

struct ConvArgs
{
    const bf16* x;  // [n][h][w][cin], or the skip [n][h][w][cs] for LD_CONCAT
    const bf16* u;  // LD_CONCAT: [n][h/2][w/2][cin - cs]
    int cs;
    int n, h, w;
    const bf16* wt;     // [npad][9 * cin], k = tap * cin + c
    const float* bias;  // [npad]
    void* out;
    const bf16* act;  // EP_MASK: [n][h][w][npad]; EP_RAW_UP: [n][h/2][w/2][npad - 32]
    const i360b_blend_job* jobs;  // EP_COMPOSITE: one per image
    int* error;
    bf16* half;          // EP_RELU_POOL: [n][h/2][w/2][npad]; EP_RAW_UP: [n][h/2][w/2][npad - 32]
    int rowSplit;  // the output map has the rows as (row % J, row / J): h is a multiple of J
};

// Tile geometry of the 3x3 convolution: TW x 16 J output pixels per tile, split
// into M blocks of 8 columns x 16 rows that lie J apart.  The input halo of (TW+2) x (TH+2)
// pixels is kept as rows of a pixel's channels (row pitch kP = TW+2 pixels) in
// the swizzle of that width: all 16, 32 or 64 of them, or for 96 the first 32
// and the other 64 in two such tiles.
template <int CIN, int NPAD, int TW, int J, int STAGES, int LD, int EP, int EW, int BUFS>
struct ConvShape
{
    // Roles by warp: [0, EW) epilogue, EW producer, EW + 1 MMA.
    static constexpr int kProducerWarp = EW, kMmaWarp = EW + 1, kThreads = 32 * (EW + 2);
    static constexpr int TH = 16 * J;
    static constexpr int kCA = CIN == 96 ? 32 : CIN, kCB = CIN - kCA;  // channels of the two tiles
    // With an upsampled second tile the two blocks of a row band take the even
    // and the odd columns: a tap then reads 8 successive half-resolution
    // pixels, and the first tile is kept as its odd and even columns.
    static constexpr bool kParity = LD == LD_CONCAT;
    static constexpr int kPA = kParity ? TW / 2 + 1 : TW + 2, kPB = kParity ? TW / 2 + 2 : TW + 2;  // row pitches, pixels
    static constexpr uint32_t kBoxA = kPA * (TH + 2) * kCA * 2, kPlane = (kBoxA + 1023) / 1024 * 1024;
    static constexpr uint32_t kBoxB = kPB * (kParity ? TH / 2 + 2 : TH + 2) * kCB * 2;
    static constexpr uint32_t kTileA = (kParity ? 2 : 1) * kPlane, kTileB = (kBoxB + 1023) / 1024 * 1024;
    static constexpr uint32_t kStage = kTileA + kTileB;
    static constexpr uint32_t kW = (9u * CIN * NPAD * 2 + 1023) / 1024 * 1024;
    static constexpr int kBX = TW / 8, kMB = kBX * J;  // block b: column b / J, row b % J
    static constexpr uint32_t kSlotCols = kMB * NPAD;
    static constexpr uint32_t kTmem = tc::tmem_cols(2 * kSlotCols);
    // The epilogue's unit is kBatch blocks by kGroup channels: two rows (or the
    // two parities of a row), which hide each other's latencies, where the
    // accumulators then fit registers.
    // Every four warps take the next J * 4 / EW of the rows (for EP_RAW_UP,
    // which needs both, every second or only group of 32 channels instead).
    static constexpr int kGroup = EP == EP_RAW_UP ? 32 : NPAD, kGroupStep = EP == EP_RAW_UP ? EW / 4 : 1;
    static constexpr int kRows = EP == EP_RAW_UP ? J : J * 4 / EW, kPer = kRows * kBX;  // blocks of a warp, by columns
    static constexpr int kBatch = EP == EP_COMPOSITE ? kPer : kGroup <= 32 && (kParity || kRows >= 2) ? 2 : 1;
    // Outputs leave by TMA from BUFS buffers per epilogue warp, each a unit as
    // swizzled tiles of 32 pixels and channels.
    static constexpr bool kStored = EP != EP_LOGITS && EP != EP_COMPOSITE;
    static constexpr uint32_t kOutBuf = kStored ? kBatch * 32 * kGroup * 2 : 0, kOut = EW * BUFS * kOutBuf;
    static constexpr uint32_t kBars = ((2 * STAGES + 4) * 8 + 16 + 15) / 16 * 16;
    static constexpr uint32_t kBias = NPAD * 4;
    static constexpr uint32_t kSmem = 1024 + kW + STAGES * kStage + kOut + kBars + kBias;
    static_assert(CIN == 16 || CIN == 32 || CIN == 64 || CIN == 96, "channels as swizzled rows");
    static_assert(NPAD == 16 || NPAD % 32 == 0, "MMA and output shape");
    static_assert((LD == LD_PLAIN) == (CIN != 96), "loader");
    static_assert(TW % 8 == 0 && TW + 2 <= 256 && TH + 2 <= 256 && TH % 16 == 0, "tile shape");
    static_assert((J < 3 ? J : 3) * NPAD <= 256, "MMA columns");
    static_assert(2 * kSlotCols <= 512, "TMEM capacity");
    static_assert(kSmem <= 227u * 1024u, "shared memory");
    static_assert(EW % 4 == 0 && kRows >= 1 && kPer % kBatch == 0, "epilogue warps split the rows");
    static_assert(!kParity || (TW == 16 && J == 2 && EW == 8 && kStored), "parities of a row in one unit");
    static_assert((EP != EP_RELU_POOL && EP != EP_RAW_UP) || kBatch == 2, "2x2 sums take two rows");
};

// The tiles that a persistent CTA takes, `stride` apart, as column, row and
// image, stepped with carries.
struct TileWalk
{
    int tilesX, tilesY, nx, ny, ni, tx, ty, img;
    __device__ __forceinline__ TileWalk(int tilesX_, int tilesY_, int first, int stride)
        : tilesX(tilesX_), tilesY(tilesY_), nx(stride % tilesX_), ny(stride / tilesX_ % tilesY_),
          ni(stride / tilesX_ / tilesY_), tx(first % tilesX_), ty(first / tilesX_ % tilesY_),
          img(first / tilesX_ / tilesY_)
    {
    }
    __device__ __forceinline__ void next()
    {
        tx += nx;
        ty += ny + (tx >= tilesX);
        if (tx >= tilesX) tx -= tilesX;
        img += ni + (ty >= tilesY);
        if (ty >= tilesY) ty -= tilesY;
    }
};

// Position of the 16-byte channel chunk c of pixel px in a row of C channels
// (C * 2 bytes a pixel) under the swizzle of that width; its own inverse in c.
template <int C>
__device__ __forceinline__ int swizzled_chunk(int px, int c)
{
    return C == 64 ? c ^ (px & 7) : C == 32 ? c ^ ((px >> 1) & 3) : c ^ ((px >> 2) & 1);
}

__device__ __forceinline__ uint4 pack8_bf16(const float* v)
{
    uint4 r;
    __nv_bfloat162 p0 = __floats2bfloat162_rn(v[0], v[1]);
    __nv_bfloat162 p1 = __floats2bfloat162_rn(v[2], v[3]);
    __nv_bfloat162 p2 = __floats2bfloat162_rn(v[4], v[5]);
    __nv_bfloat162 p3 = __floats2bfloat162_rn(v[6], v[7]);
    r.x = *reinterpret_cast<uint32_t*>(&p0);
    r.y = *reinterpret_cast<uint32_t*>(&p1);
    r.z = *reinterpret_cast<uint32_t*>(&p2);
    r.w = *reinterpret_cast<uint32_t*>(&p3);
    return r;
}

// All ones in each half of a bf16 pair that is > 0.
__device__ __forceinline__ uint32_t positive2(uint32_t v)
{
    return __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&v), __nv_bfloat162(__nv_bfloat16_raw{0}, __nv_bfloat16_raw{0}));
}

__device__ __forceinline__ void unpack8_bf16(uint4 q, float* v)
{
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
        __nv_bfloat162 p = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
        float2 f = __bfloat1622float2(p);
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

// Softmax-weighted composite of a pixel's covered layers (the network head).
// The pixel's layer values (0 where a slot is absent), as (r | g << 16, b).
__device__ __forceinline__ void load_slots_raw(const i360b_blend_job& J, int y, int x, uint2 (&v)[kSlots])
{
    const long long at = (long long)y * J.rowStride + (long long)x * J.pixStride;
#pragma unroll
    for (int i = 0; i < kSlots; ++i)
    {
        v[i] = make_uint2(0, 0);
        if (J.slot[i])
        {
            const unsigned short* p = J.slot[i] + at;
            v[i] = make_uint2(__ldg(p) | (uint32_t)__ldg(p + 1) << 16, __ldg(p + 2));
        }
    }
}

// The pixel's layer values (0 where a slot is absent).
__device__ __forceinline__ void load_slots(const i360b_blend_job& J, int y, int x, float (*v)[3])
{
#pragma unroll
    for (int i = 0; i < kSlots; ++i)
    {
        v[i][0] = v[i][1] = v[i][2] = 0.0f;
        if (J.slot[i])
        {
            const unsigned short* p = J.slot[i] + (long long)y * J.rowStride + (long long)x * J.pixStride;
            v[i][0] = __ldg(p);
            v[i][1] = __ldg(p + 1);
            v[i][2] = __ldg(p + 2);
        }
    }
}

// Softmax over the covered layers (value not (0,0,0)) of the logits, and the
// weighted sum of the layers; v from load_slots.
__device__ __forceinline__ void blend_slots(const float* l, const float (*v)[3], float* outDN, float* wts, bool* cov,
                                            int& nCov)
{
    float m = -INFINITY;
    nCov = 0;
#pragma unroll
    for (int i = 0; i < kSlots; ++i)
    {
        cov[i] = v[i][0] != 0.0f || v[i][1] != 0.0f || v[i][2] != 0.0f;
        if (cov[i])
        {
            m = fmaxf(m, l[i]);
            ++nCov;
        }
    }
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < kSlots; ++i)
    {
        wts[i] = cov[i] ? __expf(l[i] - m) : 0.0f;
        sum += wts[i];
    }
    const float inv = nCov ? 1.0f / sum : 0.0f;
    outDN[0] = outDN[1] = outDN[2] = 0.0f;
#pragma unroll
    for (int i = 0; i < kSlots; ++i)
    {
        wts[i] *= inv;
        outDN[0] += wts[i] * v[i][0];
        outDN[1] += wts[i] * v[i][1];
        outDN[2] += wts[i] * v[i][2];
    }
}

__device__ __forceinline__ void composite_pixel(const i360b_blend_job& J, int y, int x, const float* l, float* outDN,
                                                float* wts, float (*v)[3], bool* cov, int& nCov)
{
    load_slots(J, y, x, v);
    blend_slots(l, v, outDN, wts, cov, nCov);
}

// ---------------------------------------------------------------------------
// 3x3 convolution (forward, or backward-data with flipped transposed weights),
// persistent and warp-specialised; CTA b handles tiles b, b + gridDim.x, ...
//
// One MMA serves three taps.  The 16 rows of M block j lie J apart, rows
// j, j + J, ...; so the operand of its tap dy, rows j + dy, j + dy + J, ... of
// the halo, is "set" j + dy of J + 2, and set s is the operand of blocks s - 2,
// s - 1 and s at dy = 2, 1, 0.  Their accumulators are consecutive columns and
// the weights of the three dy consecutive rows of B: one MMA of N = 3 NPAD per
// set, dx and 16 channels (fewer at the first and last two sets), 3 (J + 2)
// CIN / 16 of them instead of 9 J CIN / 16.  An MMA costs the fetch of its 4 KB
// of A and its issue however few its columns, which bounded one MMA per tap of
// 16..64 columns.  Sets ascend, so each accumulator still sums
// in the order tap, channel that fixes the results' bits; the epilogue leaves
// zeros in accumulators that it has read, as an MMA can not start one of its
// blocks and continue two.
//
// The A operand of set s and dx for column block bx is the halo tile from
// pixel (8 bx + dx, s): 8 pixels of a row are 8 swizzled rows, the 16 rows J kP
// pixels apart (SBO), a K step 32 bytes into the row.  The swizzle is a
// function of the address, so a window may start at any pixel.  An upsampled
// half of the input is read where it lies, at half resolution: of the two
// blocks of a row one takes the even, one the odd columns, so that tap's 8
// pixels are successive there, and two rows' taps the same row.
//
// Roles:
//   warp EW        lane 0 loads a tile's halo by TMA into a STAGES-deep ring, zero
//                  fill outside the image: one 4-D box (channels x (TW+2) x
//                  (16J+2)), two for 96 channels of one tensor, or the skip's
//                  odd and even columns as 5-D boxes and the half-resolution
//                  tensor's 4-D box;
//   warp EW+1      issues the MMAs, converged, by one elected thread, into one of
//                  two sets of TMEM accumulators; commits free the ring stage
//                  and publish the accumulators;
//   warps 0..EW-1  epilogue (EW = 4, 8 or 16): TMEM lanes 32q..32q+31, q = w % 4
//                  (4 rows of each M block) -> bias/ReLU, mask or raw,
//                  then by TMA from shared memory, or blend head -> global.
// Every wait is bounded; a timeout sets the error flag and the CTA winds
// down after its loads have landed.
//
// 64 windows of 256 x 256, a 32 -> 32 layer: 89 us (537 MB, 81 us at the
// measured copy rate), and with the 2x2 averages 109; with one MMA per tap,
// 8-channel TMA boxes and outputs stored a lane's 16 bytes at a time 176 us
// and 55 for a kernel that averaged.  The 96-channel layer 0.22 ms (MMA issue
// and operand fetch; 0.49 with the upsample expanded by warps), its backward
// with the upsample's sums 0.21 (0.47 and 0.17 apart).
// ---------------------------------------------------------------------------
template <int CIN, int NPAD, int TW, int J, int STAGES, int LD, int EP, int EW, int BUFS>
__global__ void __launch_bounds__(ConvShape<CIN, NPAD, TW, J, STAGES, LD, EP, EW, BUFS>::kThreads, 1)
    k_conv3x3(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
              const __grid_constant__ CUtensorMap mapOut, ConvArgs a)
{
    using S = ConvShape<CIN, NPAD, TW, J, STAGES, LD, EP, EW, BUFS>;
    constexpr int TH = S::TH;
    extern __shared__ unsigned char smemRaw[];
    unsigned char* smem =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
    unsigned char* wsm = smem;
    unsigned char* ring = smem + S::kW;
    unsigned char* outBufs = ring + STAGES * S::kStage;
    uint64_t* full = reinterpret_cast<uint64_t*>(outBufs + S::kOut);
    uint64_t* empty = full + STAGES;
    uint64_t* accFull = empty + STAGES;
    uint64_t* accEmpty = accFull + 2;
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(accEmpty + 2);
    float* sBias = reinterpret_cast<float*>(outBufs + S::kOut + S::kBars);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int tilesX = (a.w + TW - 1) / TW, tilesY = (a.h + TH - 1) / TH;
    const long long nTiles = (long long)a.n * tilesX * tilesY;
    if ((long long)blockIdx.x >= nTiles) return;
    const int myTiles = (int)((nTiles - 1 - blockIdx.x) / gridDim.x) + 1;

    if (warp == 0) tc::tmem_alloc(tmemSlot, S::kTmem);
    if (tid == 0)
    {
        for (int s = 0; s < STAGES; ++s)
        {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int k = 0; k < 2; ++k)
        {
            tc::mbar_init(&accFull[k], 1);
            tc::mbar_init(&accEmpty[k], EW);
        }
        tc::fence_mbar_init();
    }
    {
        // [dx][channel / 8][2 - dy][n] of 8 channels, from [n][dy][dx][channel]
        constexpr int kC8 = CIN / 8, kK8 = 9 * kC8;
        for (int q = tid; q < NPAD * kK8; q += blockDim.x)
        {
            const int n = q / kK8, k8 = q % kK8, tap = k8 / kC8, c8 = k8 % kC8;
            tc::cp_async16(wsm + (((tap % 3) * kC8 + c8) * 3 + 2 - tap / 3) * (NPAD * 16) + n * 16,
                           a.wt + (size_t)n * 9 * CIN + k8 * 8, 16);
        }
        tc::cp_async_commit();
        for (int c = tid; c < NPAD; c += blockDim.x) sBias[c] = a.bias ? a.bias[c] : 0.0f;
        tc::cp_async_wait<0>();
        tc::fence_proxy_async();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmemSlot;
    bool ok = true;
    if (warp < 4)
    {
        for (uint32_t c = 0; c < 2 * S::kSlotCols; c += 16) tc::tmem_zero16(tmem + ((uint32_t)(warp * 32) << 16) + c);
        tc::tmem_wait_st();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();

    if (warp == S::kProducerWarp)
    {
        if (lane == 0)
        {
            int issued = 0;
            TileWalk t(tilesX, tilesY, blockIdx.x, gridDim.x);
            for (int i = 0; i < myTiles; ++i, t.next())
            {
                const int s = i % STAGES;
                if (!tc::mbar_wait(&empty[s], ((i / STAGES) & 1) ^ 1, kWaitSpins))
                {
                    ok = false;
                    break;
                }
                const int x0 = t.tx * TW, y0 = t.ty * TH;
                unsigned char* st = ring + s * S::kStage;
                tc::mbar_arrive_expect_tx(&full[s], (S::kParity ? 2 : 1) * S::kBoxA + S::kBoxB);
                if (S::kParity)
                {
                    // columns x0 - 1, x0 + 1, ... and x0, x0 + 2, ... (x0 even)
                    tc::tma_load_5d(st, &mapA, 0, 1, (x0 >> 1) - 1, y0 - 1, t.img, &full[s]);
                    tc::tma_load_5d(st + S::kPlane, &mapA, 0, 0, x0 >> 1, y0 - 1, t.img, &full[s]);
                    tc::tma_load_4d(st + S::kTileA, &mapB, 0, (x0 >> 1) - 1, (y0 >> 1) - 1, t.img, &full[s]);
                }
                else
                {
                    tc::tma_load_4d(st, &mapA, 0, x0 - 1, y0 - 1, t.img, &full[s]);
                    if (LD == LD_SPLIT) tc::tma_load_4d(st + S::kTileA, &mapB, S::kCA, x0 - 1, y0 - 1, t.img, &full[s]);
                }
                issued = i + 1;
            }
            // The last loads must land before the CTA may exit.
            for (int j = max(0, issued - STAGES); j < issued; ++j)
                if (!tc::mbar_wait(&full[j % STAGES], (j / STAGES) & 1, kWaitSpins)) ok = false;
        }
    }
    else if (warp == S::kMmaWarp)
    {
        // The whole warp runs the loop and one thread of it issues: operands
        // then stay in uniform registers.  From one thread's branch each MMA
        // took 70 cycles to issue, whatever its size.
        {
            const bool leader = tc::elect_one();
            const uint32_t tmemU = __shfl_sync(0xffffffffu, tmem, 0);
            const uint64_t bBase = tc::smem_desc(tc::smem_u32(wsm), 3 * NPAD * 16, 128);
            for (int i = 0; i < myTiles; ++i)
            {
                const int s = i % STAGES, acc = i & 1;
                const bool ready = tc::mbar_wait(&full[s], (i / STAGES) & 1, kWaitSpins) &&
                                   tc::mbar_wait(&accEmpty[acc], ((i >> 1) & 1) ^ 1, kWaitSpins);
                if (!__all_sync(0xffffffffu, ready))
                {
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                // Descriptors differ only in their start-address field: add
                // the (compile-time) offset in 16-byte units to a base.
                const uint32_t st = tc::smem_u32(ring + s * S::kStage);
                const uint64_t aBase = tc::smem_desc_k<S::kCA>(st, J * S::kPA * S::kCA * 2);
                const uint64_t a2Base = tc::smem_desc_k<64>(st + S::kTileA, (S::kParity ? J / 2 : J) * S::kPB * 64 * 2);
#pragma unroll
                for (int bx = 0; bx < S::kBX; ++bx)
#pragma unroll
                    for (int set = 0; set < J + 2; ++set)
                    {
                        const int j0 = set > 2 ? set - 2 : 0, j1 = set < J ? set : J - 1;  // blocks of the set
                        const uint32_t d = tmemU + acc * S::kSlotCols + (bx * J + j0) * NPAD;
                        const uint32_t idesc = tc::idesc_bf16_f32(128, (j1 - j0 + 1) * NPAD);
#pragma unroll
                        for (int k0 = 0; k0 < 3 * CIN; k0 += 16)
                        {
                            const int dx = k0 / CIN, c = k0 % CIN;
                            // first pixel of the operand in either tile
                            const int px = S::kParity ? set * S::kPA + (bx + dx) / 2 : set * S::kPA + bx * 8 + dx;
                            const int px2 = S::kParity ? (set + 1) / 2 * S::kPB + (bx + dx + 1) / 2 : px;
                            const uint32_t plane = S::kParity ? (bx + dx) % 2 * S::kPlane : 0;
                            const uint64_t aDesc = c < S::kCA ? aBase + ((plane + px * S::kCA * 2 + c * 2) >> 4)
                                                              : a2Base + ((px2 * 128 + (c - S::kCA) * 2) >> 4);
                            const uint32_t bRow = (k0 / 8) * 3 * NPAD + (2 - (set - j0)) * NPAD;
                            if (leader) tc::mma_bf16(d, aDesc, bBase + bRow, idesc, 1u);
                        }
                    }
                if (leader)
                {
                    tc::mma_commit(&empty[s]);
                    tc::mma_commit(&accFull[acc]);
                }
                __syncwarp();
            }
        }
    }
    else if (warp < EW)
    {
        // Warp w reads TMEM lane quadrant w % 4, of rows `firstRow` and groups
        // `firstGroup` on.
        constexpr int kRows = S::kRows;
        const int quad = warp & 3, firstRow = EP == EP_RAW_UP ? 0 : (warp >> 2) * kRows,
                  firstGroup = EP == EP_RAW_UP ? warp >> 2 : 0;
        unsigned char* buf = outBufs + warp * (BUFS * S::kOutBuf);
        int next = 0;  // output buffer
        constexpr int kBatch = S::kBatch, kGroup = S::kGroup;
        // Pixel of this lane in the n-th block of tile t.
        struct Px
        {
            int y, x;
        };
        auto pixel = [&](const TileWalk& t, int n) {
            return Px{t.ty * TH + firstRow + n % kRows + J * (4 * quad + (lane >> 3)),
                      t.tx * TW + (S::kParity ? n / kRows + 2 * (lane & 7) : n / kRows * 8 + (lane & 7))};
        };
        // Global inputs of a unit are loaded while the one before it is
        // finished.
        uint2 vv[EP == EP_COMPOSITE ? kBatch : 1][kSlots];
        bool inJob[kBatch];
        uint4 mk[EP == EP_MASK ? kBatch * kGroup / 8 : EP == EP_RAW_UP ? 2 : 1];
        auto load_inputs = [&](const TileWalk& t, int n, int group) {
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
            {
                const Px p = pixel(t, n + k);
                const bool valid = p.y < a.h && p.x < a.w;
                const size_t pix = ((size_t)t.img * a.h + p.y) * a.w + p.x;
                if (EP == EP_COMPOSITE)
                {
                    const i360b_blend_job& Jb = a.jobs[t.img];
                    inJob[k] = valid && p.x < Jb.width && p.y < Jb.height;
                    if (inJob[k]) load_slots_raw(Jb, p.y, p.x, vv[EP == EP_COMPOSITE ? k : 0]);
                }
                if (EP == EP_MASK && valid)
                {
                    const uint4* ap = reinterpret_cast<const uint4*>(a.act + pix * NPAD);
#pragma unroll
                    for (int q = 0; q < kGroup / 8; ++q) mk[EP == EP_MASK ? k * (kGroup / 8) + q : 0] = ap[q];
                }
                if (EP == EP_RAW_UP && k == 0 && group > 0 && valid)
                {
                    const size_t hp = ((size_t)t.img * (a.h >> 1) + (p.y >> 1)) * (a.w >> 1) + (p.x >> 1);
                    const uint4* ap = reinterpret_cast<const uint4*>(a.act + hp * (NPAD - 32) + (group - 1) * 32 +
                                                                     (lane & 1) * 16);
                    mk[0] = ap[0];
                    mk[EP == EP_RAW_UP ? 1 : 0] = ap[1];
                }
            }
        };
        TileWalk t(tilesX, tilesY, blockIdx.x, gridDim.x);
        load_inputs(t, 0, firstGroup);
        for (int i = 0; i < myTiles && ok; ++i)
        {
            const int acc = i & 1, img = t.img;
            const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + acc * S::kSlotCols;
            TileWalk following = t;
            following.next();
            const bool done = tc::mbar_wait(&accFull[acc], (i >> 1) & 1, kWaitSpins);
            if (!__all_sync(0xffffffffu, done))
            {
                ok = false;
                break;
            }
            tc::fence_after_sync();
#pragma unroll 1
            for (int n = 0; n < S::kPer; n += kBatch)
#pragma unroll 1
                for (int group = firstGroup; group < NPAD / kGroup; group += S::kGroupStep)
                {
                    auto at = [&](int k) {  // accumulators of the unit's k-th block
                        return base + ((n + k) / kRows * J + firstRow + (n + k) % kRows) * NPAD + group * kGroup;
                    };
                    uint32_t r[kBatch][kGroup];
#pragma unroll
                    for (int k = 0; k < kBatch; ++k)
#pragma unroll
                        for (int cb = 0; cb < kGroup / 16; ++cb)
                            tc::tmem_ld16_nowait(at(k) + cb * 16, r[k] + cb * 16);
                    tc::tmem_wait_ld();
#pragma unroll
                    for (int k = 0; k < kBatch; ++k)
#pragma unroll
                        for (int cb = 0; cb < kGroup / 16; ++cb) tc::tmem_reg_fence16(r[k] + cb * 16);
#pragma unroll
                    for (int k = 0; k < kBatch; ++k)
#pragma unroll
                        for (int cb = 0; cb < kGroup / 16; ++cb) tc::tmem_zero16(at(k) + cb * 16);
                    const bool lastGroup = group + S::kGroupStep >= NPAD / kGroup, last = lastGroup && n + kBatch >= S::kPer;
                    if (last)
                    {
                        tc::tmem_wait_st();
                        tc::fence_before_sync();
                        __syncwarp();
                        if (lane == 0) tc::mbar_arrive(&accEmpty[acc]);
                    }
                    const Px p = pixel(t, n);
                    const bool valid = p.y < a.h && p.x < a.w;  // of the batch's first row
                    uint4 pk[kBatch][S::kStored ? kGroup / 8 : 1];
                    if (S::kStored)
                    {
#pragma unroll
                        for (int k = 0; k < kBatch; ++k)
#pragma unroll
                            for (int c8 = 0; c8 < kGroup / 8; ++c8)
                            {
                                uint32_t w[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                {
                                    const uint32_t* v = r[k] + c8 * 8 + 2 * j;
                                    f32x2 f = pack2(__uint_as_float(v[0]), __uint_as_float(v[1]));
                                    if (EP == EP_RELU || EP == EP_RELU_POOL)
                                        f = add2(f, *reinterpret_cast<const f32x2*>(sBias + c8 * 8 + 2 * j));
                                    __nv_bfloat162 h = __floats2bfloat162_rn(lo2(f), hi2(f));
                                    if (EP == EP_RELU || EP == EP_RELU_POOL)
                                        h = __hmax2(h, __nv_bfloat162(__nv_bfloat16_raw{0}, __nv_bfloat16_raw{0}));
                                    w[j] = *reinterpret_cast<uint32_t*>(&h);
                                }
                                if (EP == EP_MASK)
                                {
                                    const uint4 m = mk[EP == EP_MASK ? k * (kGroup / 8) + c8 : 0];
                                    w[0] &= positive2(m.x);
                                    w[1] &= positive2(m.y);
                                    w[2] &= positive2(m.z);
                                    w[3] &= positive2(m.w);
                                }
                                pk[k][S::kStored ? c8 : 0] = make_uint4(w[0], w[1], w[2], w[3]);
                            }
                    }
                    if (EP == EP_LOGITS || EP == EP_COMPOSITE)
                    {
#pragma unroll
                        for (int k = 0; k < kBatch; ++k)
                        {
                            const Px q = pixel(t, n + k);
                            float l[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) l[j] = __uint_as_float(r[k][j]) + sBias[j];
                            if (EP == EP_LOGITS)
                            {
                                if (q.y < a.h && q.x < a.w)
                                    reinterpret_cast<float4*>(a.out)[((size_t)img * a.h + q.y) * a.w + q.x] =
                                        make_float4(l[0], l[1], l[2], l[3]);
                            }
                            else if (inJob[k])
                            {
                                const i360b_blend_job& Jb = a.jobs[img];
                                float o[3], wts[4];
                                bool cov[4];
                                int nCov;
                                float v[kSlots][3];
#pragma unroll
                                for (int m = 0; m < kSlots; ++m)
                                {
                                    const uint2 raw = vv[EP == EP_COMPOSITE ? k : 0][m];
                                    v[m][0] = raw.x & 0xffff;
                                    v[m][1] = raw.x >> 16;
                                    v[m][2] = raw.y;
                                }
                                blend_slots(l, v, o, wts, cov, nCov);
                                unsigned short* op = Jb.out + (long long)q.y * Jb.outRowStride + (long long)q.x * 3;
#pragma unroll
                                for (int c = 0; c < 3; ++c)
                                    op[c] = (unsigned short)__float2uint_rn(fminf(fmaxf(o[c], 0.0f), 65535.0f));
                            }
                        }
                    }
                    if (EP == EP_RELU_POOL || (EP == EP_RAW_UP && group > 0))
                    {
                        // 2x2 sums of the rounded outputs, left to right, upper
                        // row first; of 32 channels the left lane of a pair
                        // takes the first half, the right lane the second.
                        const bool right = lane & 1;
                        float sum[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c) sum[c] = 0.0f;
#pragma unroll
                        for (int k = 0; k < kBatch; ++k)
#pragma unroll
                            for (int q = 0; q < 2; ++q)
                            {
                                const uint4 lo = pk[k][S::kStored ? q : 0], hi = pk[k][S::kStored ? 2 + q : 0];
                                uint4 own = right ? hi : lo, other = right ? lo : hi;
                                other.x = __shfl_xor_sync(0xffffffffu, other.x, 1);
                                other.y = __shfl_xor_sync(0xffffffffu, other.y, 1);
                                other.z = __shfl_xor_sync(0xffffffffu, other.z, 1);
                                other.w = __shfl_xor_sync(0xffffffffu, other.w, 1);
                                float first[8], second[8];
                                unpack8_bf16(right ? other : own, first);
                                unpack8_bf16(right ? own : other, second);
#pragma unroll
                                for (int c = 0; c < 8; ++c) sum[q * 8 + c] = (sum[q * 8 + c] + first[c]) + second[c];
                            }
                        uint4 o[2];
                        if (EP == EP_RELU_POOL)
                        {
#pragma unroll
                            for (int c = 0; c < 16; ++c) sum[c] *= 0.25f;
                        }
                        o[0] = pack8_bf16(sum);
                        o[1] = pack8_bf16(sum + 8);
                        if (EP == EP_RAW_UP)
                        {
#pragma unroll
                            for (int q = 0; q < 2; ++q)
                            {
                                const uint4 m = mk[EP == EP_RAW_UP ? q : 0];
                                o[q].x &= positive2(m.x);
                                o[q].y &= positive2(m.y);
                                o[q].z &= positive2(m.z);
                                o[q].w &= positive2(m.w);
                            }
                        }
                        if (valid)
                        {
                            constexpr int kC = EP == EP_RAW_UP ? NPAD - 32 : NPAD;
                            const size_t hp = ((size_t)img * (a.h >> 1) + (p.y >> 1)) * (a.w >> 1) + (p.x >> 1);
                            uint4* op = reinterpret_cast<uint4*>(a.half + hp * kC +
                                                                 (EP == EP_RAW_UP ? (group - 1) * 32 : 0) + right * 16);
                            op[0] = o[0];
                            op[1] = o[1];
                        }
                    }
                    // inputs of the unit after this one
                    if (!lastGroup) load_inputs(t, n, group + S::kGroupStep);
                    else if (!last) load_inputs(t, n + kBatch, firstGroup);
                    else if (i + 1 < myTiles) load_inputs(following, 0, firstGroup);
                    if (S::kStored && (EP != EP_RAW_UP || group == 0))
                    {
                        unsigned char* ob = buf + next * S::kOutBuf;
                        if (BUFS > 1) next = next + 1 == BUFS ? 0 : next + 1;
                        if (lane == 0) tc::bulk_wait_read<BUFS - 1>();
                        __syncwarp();
#pragma unroll
                        for (int k = 0; k < kBatch; ++k)
#pragma unroll
                            for (int c8 = 0; c8 < kGroup / 8; ++c8)
                            {
                                // parities: one tile of 16 x 4 pixels
                                const int px = S::kParity ? 2 * lane + k : lane;
                                *reinterpret_cast<uint4*>(
                                    ob + (S::kParity ? 0 : (k * (kGroup / 32) + (c8 >> 2)) * 2048) + px * 64 +
                                    swizzled_chunk<32>(px, c8 & 3) * 16) = pk[k][S::kStored ? c8 : 0];
                            }
                        tc::fence_proxy_async();  // generic smem writes -> TMA
                        __syncwarp();
                        if (lane == 0)
                        {
#pragma unroll
                            for (int k = 0; k < (S::kParity ? 1 : kBatch); ++k)
                            {
                                const Px q = pixel(t, n + k);  // lane 0: the block's first
                                if (q.y >= a.h || q.x >= a.w) continue;
#pragma unroll
                                for (int u = 0; u < kGroup / 32; ++u)
                                {
                                    const unsigned char* tile = ob + (k * (kGroup / 32) + u) * 2048;
                                    constexpr int kRow = S::kParity ? 1024 : 512;  // bytes of a pixel row
                                    if (a.rowSplit)  // 4 rows J apart as rows / J of the map
                                        tc::tma_store_5d(&mapOut, tile, u * 32, q.x, q.y % J, q.y / J, img);
                                    else
                                        for (int v = 0; v < 4 && q.y + J * v < a.h; ++v)
                                            tc::tma_store_5d(&mapOut, tile + v * kRow, u * 32, q.x, q.y + J * v, 0, img);
                                }
                            }
                            tc::bulk_commit();
                        }
                    }
                }
            t = following;
        }
        if (S::kStored && lane == 0) tc::bulk_wait_all();
    }
    if (!ok) atomicOr(a.error, 1);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0)
    {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, S::kTmem);
    }
}

// ---------------------------------------------------------------------------
// Weight gradient, all nine taps from one MMA per 16 pixels:
//   D[(dy, cin)][(dx, cout)] += A[(dy, cin)][q] * B[q][(dx, cout)],
//   A = X[y + dy - 1][q][cin],  B = G[y][q - (dx - 1)][cout],
// summed over image rows y and pixels q (K, 16 per MMA), accumulators in TMEM
// over the CTA's whole share.  Both operands are MN-major: a pixel's CX = 16
// or 32 input channels, or its output channels, are rows of 32, 64 or 128
// bytes in the swizzle of that width, as TMA writes them.  An MMA's 16 pixels
// are those of one column parity, kept as planes.  X lies in shared memory as
// [parity][row][pixel][CX], so the operand of output row y is 128 / CX
// successive rows from y on: the three dy, then rows whose accumulators are
// not looked at.  G is kept as the four planes of columns + 2, + 1, + 0 and
// - 1: the dx of even pixels are the last three, of odd ones the first three,
// a plane apart.  Of an upsampled input both parities are the same
// half-resolution pixels, and rows y - 1 .. y + 4 three boxes of two.
// One MMA per tap would have N = cout = 16..64 columns, and fetching the 4 KB
// of A takes several times such a multiplication; here N = 3 cout.  A layer of
// more than 32 input channels is a job per 32.
//
// How far a sum is cut into slices (a CTA's share of the tiles) is not free:
// the tensor core truncates as it adds to an accumulator, so a sum comes out
// too small by an amount that grows with the number of MMAs - 1.5e-4 of it
// for 1772 of them over positive data.  The slices are therefore the ones of
// one 128-row block of (tap, cin) per SM, 74, 49, 29 or 21 by layer, that
// results have always come from: gradients of a batch of 64 windows agree
// with those to 8e-7, and one slice per SM is 1.3e-4 away.
//
// That leaves two thirds of the SMs idle, so one launch takes the jobs of all
// layers, longest first, a CTA per (job, slice).  CTA `b` of a job
// handles tiles b, b + slices, ... of 32 x 4 pixels.
//   warp 4     lane 0 loads a tile's X and G by TMA (zero fill outside the
//              image) into a ring of stages;
//   warp 5     issues the MMAs; a commit frees the stage;
//   warps 0-3  sum G for the bias gradient (where asked for); at the end write
//              the accumulators as this slice's partial sums.
// Every wait is bounded; a timeout sets the error flag and the CTA winds down
// after its loads have landed.
//
// 64 windows of 256 x 256, all eight layers with their bias gradients: 0.73
// ms for 3.3 GB of X and G (0.50 at the measured copy rate); the longest jobs,
// the 96-channel layer's 63 CTAs, set the end.  With a launch per layer 1.9 ms;
// with the pixels of an MMA successive (three full copies of G and an upsample
// by the warps) 0.77; one 128-row chunk of (tap, cin) per CTA gathered by
// cp.async, N = cout and a kernel of its own for the bias 10.9 + 0.29 ms.
// ---------------------------------------------------------------------------
enum WgradKind
{
    WG_16_32,
    WG_32_32,
    WG_32_64,
    WG_32_16,
    WG_UP32_32,  // X at half resolution, upsampled (nearest)
};

struct WgradJob
{
    CUtensorMap mapX, mapG;
    int kind, firstBlock, slices;
    int n, h, w;
    int cin, c0;     // channels of the layer, and the first of X's among them
    int xc0;         // the first of X's channels in its tensor
    int bias;        // write the sums of g
    float* partial;  // per slice [3 cin][3 COUT], then [COUT] sums of g
};

constexpr int kWgJobs = 12;  // the network's eight layers

struct WgradBatch
{
    WgradJob job[kWgJobs];
    int jobs;
    int* error;
};

constexpr int kWgRows = 4, kWgTW = 32;  // pixels of a tile

template <int CX, int COUT, bool UP>
struct WgradShape
{
    static constexpr int kXRows = kWgRows + 2, kHalfW = kWgTW / 2;
    static constexpr uint32_t kXRow = kHalfW * CX * 2, kGRow = kHalfW * COUT * 2;
    static constexpr uint32_t kXPlane = kXRows * kXRow, kGPlane = kWgRows * kGRow;
    static constexpr uint32_t kX = ((UP ? 1 : 2) * kXPlane + 1023) / 1024 * 1024, kG = 4 * kGPlane;
    static constexpr uint32_t kStage = kX + kG;
    // The last row's operand is 128 / CX rows from row 3 of the last plane on.
    static_assert(kXPlane + (kWgRows - 1 + 128 / CX) * kXRow <= kStage, "operands within the stage");
    static constexpr int kStages = 214 * 1024 / kStage > 8 ? 8 : 214 * 1024 / kStage;
    static constexpr uint32_t kSmem = 1024 + kStages * kStage + 256;
    static constexpr int kN = 3 * COUT;
    static constexpr uint32_t kTmem = tc::tmem_cols(kN);
    static_assert(CX == 16 || CX == 32, "X rows of a swizzle's width, three of them in an MMA");
    static_assert(COUT == 16 || COUT == 32 || COUT == 64, "G rows of a swizzle's width");
    static_assert(!UP || CX == 32, "upsampled input: 32 channels");
    static_assert(kStages >= 2 && kSmem <= 227u * 1024u, "shared memory");
};

template <int CX, int COUT, bool UP>
__device__ __forceinline__ void wgrad_slice(const WgradJob& a, int slice, double (&sBias)[128][9], int* error)
{
    using S = WgradShape<CX, COUT, UP>;
    extern __shared__ unsigned char smemRaw[];
    unsigned char* smem =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smemRaw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::kStages * S::kStage);
    uint64_t* empty = full + S::kStages;
    uint64_t* done = empty + S::kStages;
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(done + 1);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int tilesX = a.w / kWgTW, tilesY = (a.h + kWgRows - 1) / kWgRows;
    const long long nTiles = (long long)a.n * tilesX * tilesY;  // >= a.slices
    const int myTiles = (int)((nTiles - 1 - slice) / a.slices) + 1;
    const bool bias = !UP && a.bias;

    if (warp == 0) tc::tmem_alloc(tmemSlot, S::kTmem);
    if (tid == 0)
    {
        for (int s = 0; s < S::kStages; ++s)
        {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], bias ? 1 + 4 : 1);
        }
        tc::mbar_init(done, 1);
        tc::fence_mbar_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tmemSlot;
    bool ok = true;

    if (warp == 4)
    {
        if (lane == 0)
        {
            int issued = 0;
            TileWalk t(tilesX, tilesY, slice, a.slices);
            int s = -1;
            uint32_t phase = 0;  // of the empty barrier: one before the first use
            for (int i = 0; i < myTiles; ++i)
            {
                if (++s == S::kStages) s = 0;
                if (s == 0) phase ^= 1;
                if (!tc::mbar_wait(&empty[s], phase, kWaitSpins))
                {
                    ok = false;
                    break;
                }
                const int x0 = t.tx * kWgTW, y0 = t.ty * kWgRows;
                unsigned char* st = smem + s * S::kStage;
                const int xh = x0 >> 1;
                tc::mbar_arrive_expect_tx(&full[s], 2 * S::kXPlane / (UP ? 2 : 1) + S::kG);
                if (UP)
                    for (int k = 0; k < 3; ++k)
                        tc::tma_load_4d(st + 2 * k * S::kXRow, &a.mapX, a.xc0, xh, (y0 >> 1) - 1 + k, t.img, &full[s]);
                else
                    for (int k = 0; k < 2; ++k)
                        tc::tma_load_5d(st + k * S::kXPlane, &a.mapX, a.xc0, k, xh, y0 - 1, t.img, &full[s]);
                for (int k = 0; k < 4; ++k)  // columns x0 + 2 - k, x0 + 4 - k, ...
                    tc::tma_load_5d(st + S::kX + k * S::kGPlane, &a.mapG, 0, k & 1, xh + (2 - k - (k & 1)) / 2, y0,
                                    t.img, &full[s]);
                t.next();
                issued = i + 1;
            }
            // The last loads must land before the CTA may exit.
            for (int j = max(0, issued - S::kStages); j < issued; ++j)
            {
                const int s = j % S::kStages;
                if (!tc::mbar_wait(&full[s], (j / S::kStages) & 1, kWaitSpins)) ok = false;
            }
        }
    }
    else if (warp == 5)
    {
        // (the whole warp, so that operands stay in uniform registers)
        {
            const bool leader = tc::elect_one();
            const uint32_t tmemU = __shfl_sync(0xffffffffu, tmem, 0);
            constexpr uint32_t idesc = tc::idesc_bf16_f32(128, S::kN) | (1u << 15) | (1u << 16);  // A, B MN-major
            for (int i = 0; i < myTiles; ++i)
            {
                const int s = i % S::kStages;
                const bool ready = tc::mbar_wait(&full[s], (i / S::kStages) & 1, kWaitSpins);
                if (!__all_sync(0xffffffffu, ready))
                {
                    ok = false;
                    break;
                }
                tc::fence_after_sync();
                const uint32_t xa = tc::smem_u32(smem + s * S::kStage);
                const uint64_t aBase = tc::smem_desc_mn<CX>(xa, S::kXRow),
                               bBase = tc::smem_desc_mn<COUT>(xa + S::kX, S::kGPlane);
#pragma unroll
                for (int r = 0; r < kWgRows; ++r)
#pragma unroll
                    for (int p = 0; p < 2; ++p)  // column parity
                        if (leader)
                            tc::mma_bf16(tmemU, aBase + (((UP ? 0 : p) * S::kXPlane + r * S::kXRow) >> 4),
                                         bBase + (((1 - p) * S::kGPlane + r * S::kGRow) >> 4), idesc,
                                         (i > 0 || r > 0 || p > 0) ? 1u : 0u);
                if (leader) tc::mma_commit(&empty[s]);
                __syncwarp();
            }
            if (leader) tc::mma_commit(done);
        }
    }
    else if (bias)
    {
        // This thread's chunk position and pixels of the planes + 1 and + 0,
        // 128 rows of COUT / 8 chunks; the pixels it sees keep the chunk's
        // place in the swizzle, so its channels are fixed.  The sums cancel,
        // so chains of FP32 additions stay as short as 8 tiles.
        constexpr int kO8 = COUT / 8;
        const int pos = tid % kO8, px0 = tid / kO8;
        float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        double total[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        const uint32_t zero = (uint32_t)a.bias >> 1;  // (a.bias is 1 here)
        for (int i = 0; i < myTiles; ++i)
        {
            const int s = i % S::kStages;
            // The warp goes on, or gives up, as one.
            const bool ready = tc::mbar_wait(&full[s], (i / S::kStages) & 1, kWaitSpins);
            if (!__all_sync(0xffffffffu, ready))
            {
                ok = false;
                break;
            }
            const unsigned char* g = smem + s * S::kStage + S::kX + S::kGPlane;
            uint32_t seen = 0;
#pragma unroll
            for (int k = 0; k < kWgRows * kWgTW * kO8 / 128; ++k)
            {
                const int p = px0 + k * (128 / kO8);
                const uint4 q = *reinterpret_cast<const uint4*>(g + p * COUT * 2 + pos * 16);
                seen |= q.x | q.y | q.z | q.w;
                float v[8];
                unpack8_bf16(q, v);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[j] += v[j];
            }
            // The next TMA may overwrite the stage as soon as the arrival is
            // seen, which loads still in flight are not behind: the tensor
            // core's fetches can hold them up for longer than a TMA takes.
            // So the arrival depends on what every lane's loads returned.
            seen = __reduce_or_sync(0xffffffffu, seen);
            if (lane == 0) tc::mbar_arrive_after(&empty[s], seen, zero);
            if ((i & 7) == 7 || i + 1 == myTiles)
#pragma unroll
                for (int j = 0; j < 8; ++j)
                {
                    total[j] += acc[j];
                    acc[j] = 0.0f;
                }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) sBias[tid][j] = total[j];
    }
    __syncthreads();
    float* out = a.partial + (size_t)slice * (9 * a.cin * COUT + COUT);
    if (warp < 4)
    {
        bool got = tc::mbar_wait(done, 0, kWaitSpins);
        got = __all_sync(0xffffffffu, got);
        if (!got) ok = false;
        else
        {
            tc::fence_after_sync();
            const int m = warp * 32 + lane, dy = m / CX;
            float* row = out + ((size_t)dy * a.cin + a.c0 + m % CX) * S::kN;
#pragma unroll 1
            for (int cb = 0; cb < S::kN / 16; ++cb)
            {
                float v[16];
                tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + cb * 16, v);
                if (dy < 3)
                {
                    float4* o = reinterpret_cast<float4*>(row + cb * 16);
                    o[0] = make_float4(v[0], v[1], v[2], v[3]);
                    o[1] = make_float4(v[4], v[5], v[6], v[7]);
                    o[2] = make_float4(v[8], v[9], v[10], v[11]);
                    o[3] = make_float4(v[12], v[13], v[14], v[15]);
                }
            }
            tc::fence_before_sync();
        }
        if (bias && tid < COUT)
        {
            double b = 0.0;
            for (int t = 0; t < 128; ++t)
                if (swizzled_chunk<COUT>(t / (COUT / 8), t % (COUT / 8)) == tid >> 3) b += sBias[t][tid & 7];
            out[9 * a.cin * COUT + tid] = (float)b;
        }
    }
    if (!ok) atomicOr(error, 1);
    __syncthreads();
    if (warp == 0)
    {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, S::kTmem);
    }
}

__global__ void __launch_bounds__(192, 1) k_conv3x3_wgrad(const __grid_constant__ WgradBatch b)
{
    int j = 0;
    while (j + 1 < b.jobs && (int)blockIdx.x >= b.job[j + 1].firstBlock) ++j;
    const WgradJob& a = b.job[j];
    const int slice = blockIdx.x - a.firstBlock;
    __shared__ double sBias[128][9];
    switch (a.kind)
    {
        case WG_16_32: wgrad_slice<16, 32, false>(a, slice, sBias, b.error); break;
        case WG_32_32: wgrad_slice<32, 32, false>(a, slice, sBias, b.error); break;
        case WG_32_64: wgrad_slice<32, 64, false>(a, slice, sBias, b.error); break;
        case WG_32_16: wgrad_slice<32, 16, false>(a, slice, sBias, b.error); break;
        default: wgrad_slice<32, 32, true>(a, slice, sBias, b.error); break;
    }
}
constexpr uint32_t kWgSmem = std::max({WgradShape<16, 32, false>::kSmem, WgradShape<32, 32, false>::kSmem,
                                       WgradShape<32, 64, false>::kSmem, WgradShape<32, 16, false>::kSmem,
                                       WgradShape<32, 32, true>::kSmem});

// Channels [c0, c0 + cn) of the concatenation of x (cs channels) and the
// nearest 2x upsample of u (cin - cs) as a tensor, for splits that no kernel
// above takes directly.
__global__ void k_concat(const bf16* __restrict__ x, const bf16* __restrict__ u, int cs, int cin, int c0, int cn, int n,
                         int h, int w, bf16* __restrict__ out)
{
    const int c8n = cn / 8, sc8 = cs / 8;
    const long long total = (long long)n * h * w * c8n;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x)
    {
        const int c8 = c0 / 8 + (int)(i % c8n);
        const long long p = i / c8n;
        const int xx = (int)(p % w);
        const long long r = p / w;
        const int yy = (int)(r % h), img = (int)(r / h);
        const bf16* src = c8 < sc8 ? x + p * cs + c8 * 8
                                   : u + (((size_t)img * (h >> 1) + (yy >> 1)) * (w >> 1) + (xx >> 1)) * (cin - cs) +
                                         (c8 - sc8) * 8;
        reinterpret_cast<uint4*>(out)[i] = *reinterpret_cast<const uint4*>(src);
    }
}

// dW[co][dy][dx][c] = sum over slices of partial[slice][(dy, c)][(dx, co)], and
// db[co] (unless null) the sums of g, in slice order, for the layers of a
// batch; consecutive threads take consecutive partial sums.
struct WgradReduce
{
    struct Layer
    {
        const float* partial;
        int slices, cin, coutPad, cout, firstBlock;
        float *dw, *db;
    } layer[kWgJobs];
    int layers;
};

__global__ void k_wgrad_reduce(const __grid_constant__ WgradReduce r)
{
    int l = 0;
    while (l + 1 < r.layers && (int)blockIdx.x >= r.layer[l + 1].firstBlock) ++l;
    const WgradReduce::Layer& a = r.layer[l];
    const int N = 3 * a.coutPad, weights = 3 * a.cin * N, count = weights + a.coutPad;
    const int idx = (blockIdx.x - a.firstBlock) * blockDim.x + threadIdx.x;
    if (idx >= count) return;
    if (idx >= weights && !a.db) return;
    float s = 0.0f;
#pragma unroll 8
    for (int g = 0; g < a.slices; ++g) s += __ldg(a.partial + (size_t)g * count + idx);
    if (idx < weights)
    {
        const int m = idx / N, col = idx - m * N;
        const int dy = m / a.cin, c = m - dy * a.cin, dx = col / a.coutPad, co = col - dx * a.coutPad;
        if (co < a.cout) a.dw[((size_t)co * 9 + dy * 3 + dx) * a.cin + c] = s;
    }
    else if (idx - weights < a.cout)
    {
        double b = 0.0;  // (a sum that cancels)
        for (int g = 0; g < a.slices; ++g) b += a.partial[(size_t)g * count + idx];
        a.db[idx - weights] = (float)b;
    }
}

// ---------------------------------------------------------------------------
// Glue: input packing, pooling, loss, gradient routing, Adam.
// ---------------------------------------------------------------------------
// The mask channel of a covered pixel: 0.25 + 0.75 min(1, d / kFeather) with
// d the distance from (x, y) to the nearest of the slot's boundary segments
// (1 when it has none).
constexpr float kFeather = 2048.0f;

__device__ __forceinline__ float feathered_mask(const float* e, float x, float y)
{
    float d2 = INFINITY;
#pragma unroll
    for (int s = 0; s < 4; ++s)
    {
        const float ax = e[4 * s], ay = e[4 * s + 1];
        if (ax != ax) continue;  // absent segment
        const float dx = e[4 * s + 2] - ax, dy = e[4 * s + 3] - ay;
        const float l2 = dx * dx + dy * dy;
        float t = l2 > 0.0f ? ((x - ax) * dx + (y - ay) * dy) / l2 : 0.0f;
        t = fminf(fmaxf(t, 0.0f), 1.0f);
        const float qx = ax + t * dx - x, qy = ay + t * dy - y;
        d2 = fminf(d2, qx * qx + qy * qy);
    }
    return 0.25f + 0.75f * fminf(1.0f, sqrtf(d2) / kFeather);
}

// The network's input: each slot's scaled values and feathered mask.  Bound by
// load latency: 64 windows of 256 x 256 70 us (235 MB, 36 us at the measured
// copy rate); 91 us with each slot's loads behind the test of the one before.
__global__ void k_pack_input(const i360b_blend_job* __restrict__ jobs, int n, int h, int w, bf16* __restrict__ x0)
{
    const long long total = (long long)n * h * w;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x)
    {
        const int img = (int)(idx / ((long long)h * w));
        const int rem = (int)(idx % ((long long)h * w));
        const int y = rem / w, x = rem % w;
        const i360b_blend_job& J = jobs[img];
        float ch[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) ch[i] = 0.0f;
        if (x < J.width && y < J.height)
        {
            uint2 v[kSlots];
            load_slots_raw(J, y, x, v);  // all loads before the first value is needed
#pragma unroll
            for (int i = 0; i < kSlots; ++i)
            {
                if ((v[i].x | v[i].y) == 0) continue;
                ch[4 * i] = (unsigned short)v[i].x * kInScale;
                ch[4 * i + 1] = (unsigned short)(v[i].x >> 16) * kInScale;
                ch[4 * i + 2] = (unsigned short)v[i].y * kInScale;
                ch[4 * i + 3] = feathered_mask(J.edges[i], (float)x, (float)y);
            }
        }
        uint4* o = reinterpret_cast<uint4*>(x0 + idx * 16);
        o[0] = pack8_bf16(ch);
        o[1] = pack8_bf16(ch + 8);
    }
}

// Gradient of the skip activation: g2 = (du[..., 0:C] + dpool / 4 upsampled)
// * (a2 > 0), at full resolution (C = 8 * c8n channels).
__global__ void k_skip_grad(const bf16* __restrict__ du, int duC, const bf16* __restrict__ dpool,
                            const bf16* __restrict__ act, int n, int h, int w, int c8n, bf16* __restrict__ g)
{
    const long long total = (long long)n * h * w * c8n;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x)
    {
        const int c8 = (int)(idx % c8n);
        long long r = idx / c8n;
        const int x = (int)(r % w);
        r /= w;
        const int y = (int)(r % h), img = (int)(r / h);
        float a[8], b[8], m[8];
        unpack8_bf16(*reinterpret_cast<const uint4*>(du + (size_t)(idx / c8n) * duC + c8 * 8), a);
        const size_t ph = ((size_t)img * (h >> 1) + (y >> 1)) * (w >> 1) + (x >> 1);
        unpack8_bf16(reinterpret_cast<const uint4*>(dpool + ph * c8n * 8)[c8], b);
        unpack8_bf16(reinterpret_cast<const uint4*>(act)[idx], m);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = m[j] > 0.0f ? a[j] + 0.25f * b[j] : 0.0f;
        reinterpret_cast<uint4*>(g)[idx] = pack8_bf16(a);
    }
}

// Loss of the blend head and its gradient with respect to the 4 logits
// (written as 16-channel bf16, channels 4..15 zero, the layout the last
// layer's backward consumes).
__global__ void k_loss(const i360b_blend_job* __restrict__ jobs, int n, int h, int w, const float4* __restrict__ logits,
                       float invCount, bf16* __restrict__ g8, double* __restrict__ lossAcc)
{
    __shared__ float red[32];
    const long long total = (long long)n * h * w;
    float lsum = 0.0f;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x)
    {
        const int img = (int)(idx / ((long long)h * w));
        const int rem = (int)(idx % ((long long)h * w));
        const int y = rem / w, x = rem % w;
        const i360b_blend_job& J = jobs[img];
        float dl[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) dl[j] = 0.0f;
        if (x < J.width && y < J.height)
        {
            const float4 lv = logits[idx];
            const float l[4] = {lv.x, lv.y, lv.z, lv.w};
            float o[3], wts[4], v[4][3];
            bool cov[4];
            int nCov;
            composite_pixel(J, y, x, l, o, wts, v, cov, nCov);
            const unsigned short* tp = J.target + (long long)y * J.targetRowStride + (long long)x * 3;
            float d[3];
#pragma unroll
            for (int c = 0; c < 3; ++c)
            {
                const float e = (o[c] - (float)tp[c]) * kInScale;
                lsum += e * e;
                d[c] = 2.0f * e * invCount;
            }
#pragma unroll
            for (int i = 0; i < kSlots; ++i)
            {
                if (!cov[i]) continue;
                float s = 0.0f;
#pragma unroll
                for (int c = 0; c < 3; ++c) s += d[c] * (v[i][c] - o[c]) * kInScale;
                dl[i] = wts[i] * s;
            }
        }
        uint4* q = reinterpret_cast<uint4*>(g8 + idx * 16);
        q[0] = pack8_bf16(dl);
        q[1] = pack8_bf16(dl + 8);
    }
    for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = lsum;
    __syncthreads();
    if (threadIdx.x < 32)
    {
        float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0f;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (threadIdx.x == 0) atomicAdd(lossAcc, (double)v * invCount);
    }
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int count, float lr, float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float gi = g[i];
    const float mi = 0.9f * m[i] + 0.1f * gi;
    const float vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + 1e-8f);
}

// Network layer table.
struct LayerDef
{
    int cin, cout;
};
constexpr LayerDef kNet[8] = {{16, 32}, {32, 32}, {32, 64}, {64, 64}, {64, 64}, {96, 32}, {32, 32}, {32, 4}};
constexpr int kNumLayers = 8;

__host__ __device__ constexpr int pad16(int c) { return (c + 15) / 16 * 16; }

struct PackArgs
{
    const float* params;
    int cin[kNumLayers], cout[kNumLayers];
    long long wOff[kNumLayers], bOff[kNumLayers];
    bf16* fwd[kNumLayers];    // [pad16(cout)][9 * cin]
    bf16* dgrad[kNumLayers];  // [cin][9 * pad16(cout)] flipped, transposed
    float* bias[kNumLayers];  // [pad16(cout)]
};

// Packs the fp32 master parameters into the bf16 operands of the forward and
// backward-data convolutions (blockIdx.y = layer).
__global__ void k_pack_weights(PackArgs a)
{
    const int l = blockIdx.y;
    const int cin = a.cin[l], cout = a.cout[l], np = pad16(cout);
    const int K = 9 * cin, Kd = 9 * np;
    const float* W = a.params + a.wOff[l];
    const int nf = np * K, nd = cin * Kd;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nf + nd + np; i += gridDim.x * blockDim.x)
    {
        if (i < nf)
        {
            const int n = i / K, k = i % K;
            a.fwd[l][i] = __float2bfloat16_rn(n < cout ? W[(size_t)n * K + k] : 0.0f);
        }
        else if (i < nf + nd)
        {
            const int j = i - nf, ci = j / Kd, kd = j % Kd, tap = kd / np, co = kd % np;
            a.dgrad[l][j] = __float2bfloat16_rn(co < cout ? W[(size_t)co * K + (8 - tap) * cin + ci] : 0.0f);
        }
        else
        {
            const int c = i - nf - nd;
            a.bias[l][c] = c < cout ? a.params[a.bOff[l] + c] : 0.0f;
        }
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
int grid_for(long long work, int perSm)
{
    const long long cap = (long long)sm_count() * perSm;
    return (int)std::max<long long>(1, std::min<long long>(work, cap));
}

int elementwise_grid(long long n, int block = 256)
{
    return (int)std::max<long long>(1, std::min<long long>((n + block - 1) / block, (long long)sm_count() * 16));
}

// Tensor map of bf16 values (zero fill outside) under a shared-memory swizzle;
// dims[0] is the contiguous one, stride[i] that of dims[i + 1] in values.  The
// encoder comes from the driver through the runtime (no link against the
// driver library).
template <int RANK>
int make_map(CUtensorMap* m, const bf16* base, const long long (&dims)[RANK], const long long (&stride)[RANK - 1],
             const int (&box)[RANK], CUtensorMapSwizzle swizzle)
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static std::once_flag once;
    static cudaError_t err = cudaSuccess;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        err = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", reinterpret_cast<void**>(&encode), 12000,
                                               cudaEnableDefault, &q);
        if (err == cudaSuccess && q != cudaDriverEntryPointSuccess) err = cudaErrorSymbolNotFound;
    });
    if (err != cudaSuccess || !encode) return cuda_fail(err, "cuTensorMapEncodeTiled entry point");
    if ((reinterpret_cast<uintptr_t>(base) & 15) || dims[0] % 8)
        return fail(I360B_INVALID_PARAM, "conv3x3 tensors must be 16-byte aligned with channels a multiple of 8");
    cuuint64_t d[RANK], st[RANK - 1];
    cuuint32_t bx[RANK], es[RANK];
    for (int i = 0; i < RANK; ++i)
    {
        d[i] = (cuuint64_t)dims[i];
        bx[i] = (cuuint32_t)box[i];
        es[i] = 1;
        if (i + 1 < RANK) st[i] = (cuuint64_t)stride[i] * sizeof(bf16);
    }
    CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, RANK, const_cast<bf16*>(base), d, st, bx, es,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(I360B_CUDA_ERROR, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return I360B_SUCCESS;
}

// An NHWC tensor as (C, W, H, N) with boxes of boxC x boxW x boxH x 1.
int make_tile_map(CUtensorMap* m, const bf16* base, int c, int n, int h, int w, int boxC, int boxW, int boxH,
                  CUtensorMapSwizzle swizzle)
{
    const long long row = (long long)w * c;
    return make_map<4>(m, base, {c, w, h, n}, {c, row, h * row}, {boxC, boxW, boxH, 1}, swizzle);
}

constexpr CUtensorMapSwizzle swizzle_of(int channels)
{
    return channels == 64   ? CU_TENSOR_MAP_SWIZZLE_128B
           : channels == 32 ? CU_TENSOR_MAP_SWIZZLE_64B
                            : CU_TENSOR_MAP_SWIZZLE_32B;
}

// The columns by parity, as (C, W % 2, W / 2, H, N) with boxes of boxC x 1 x
// boxW x boxH x 1 (w even).
int make_parity_map(CUtensorMap* m, const bf16* base, int c, int n, int h, int w, int boxC, int boxW, int boxH)
{
    const long long row = (long long)w * c;
    return make_map<5>(m, base, {c, 2, w / 2, h, n}, {c, 2 * c, row, h * row}, {boxC, 1, boxW, boxH, 1},
                       swizzle_of(boxC));
}

// A convolution's output, 32 channels of boxW x 4 pixels at a time: rows
// split > 0 apart as (C, W, split, H / split, N), or (split = 0) a row at a
// time as (C, W, H, 1, N).
int make_output_map(CUtensorMap* m, const bf16* base, int c, int n, int h, int w, int split, int boxW)
{
    const long long row = (long long)w * c;
    return split > 0 ? make_map<5>(m, base, {c, w, split, h / split, n}, {c, row, split * row, h * row}, {32, boxW, 1, 4, 1},
                                   CU_TENSOR_MAP_SWIZZLE_64B)
                     : make_map<5>(m, base, {c, w, h, 1, n}, {c, row, h * row, h * row}, {32, boxW, 1, 1, 1},
                                   CU_TENSOR_MAP_SWIZZLE_64B);
}

template <int CIN, int NPAD, int TW, int J, int STAGES, int LD, int EP, int EW, int BUFS>
int run_conv(ConvArgs a, cudaStream_t s)
{
    using S = ConvShape<CIN, NPAD, TW, J, STAGES, LD, EP, EW, BUFS>;
    auto* k = k_conv3x3<CIN, NPAD, TW, J, STAGES, LD, EP, EW, BUFS>;
    static std::once_flag once;
    static cudaError_t attrErr = cudaSuccess;
    std::call_once(once, [&] {
        attrErr = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem);
    });
    if (attrErr != cudaSuccess) return cuda_fail(attrErr, "conv3x3 attributes");
    constexpr int TH = S::TH;
    const long long tiles = (long long)a.n * ((a.h + TH - 1) / TH) * ((a.w + TW - 1) / TW);
    if (tiles == 0) return I360B_SUCCESS;
    CUtensorMap ma, mb, mo;
    if (LD == LD_CONCAT)
    {
        I360B_TRY(make_parity_map(&ma, a.x, S::kCA, a.n, a.h, a.w, S::kCA, S::kPA, TH + 2));
        I360B_TRY(make_tile_map(&mb, a.u, S::kCB, a.n, a.h / 2, a.w / 2, S::kCB, S::kPB, TH / 2 + 2, swizzle_of(S::kCB)));
    }
    else
    {
        I360B_TRY(make_tile_map(&ma, a.x, CIN, a.n, a.h, a.w, S::kCA, S::kPA, TH + 2, swizzle_of(S::kCA)));
        mb = ma;
        if (LD == LD_SPLIT)
            I360B_TRY(make_tile_map(&mb, a.x, CIN, a.n, a.h, a.w, S::kCB, S::kPB, TH + 2, swizzle_of(S::kCB)));
    }
    mo = ma;
    a.rowSplit = a.h % J == 0;
    if (S::kStored)
        I360B_TRY(make_output_map(&mo, static_cast<const bf16*>(a.out), EP == EP_RAW_UP ? 32 : NPAD, a.n, a.h, a.w,
                                  a.rowSplit ? J : 0, S::kParity ? 16 : 8));
    k<<<grid_for(tiles, 1), S::kThreads, S::kSmem, s>>>(ma, mb, mo, a);
    return check_launch("conv3x3 kernel");
}

// The (cin, npad) shapes the network uses, forward and backward, with tile
// width, rows' interleave J, ring depth, epilogue warps and output buffers.
// J = 4 where the halos fit twice beside the weights (half the MMAs of one per
// tap), else 2 (two thirds); 64 windows of 256 x 256:
//   * 16 epilogue warps for the blend head, whose layer loads it must cover:
//     90 us, 129 with 8; the others are the same with 8 and 16;
//   * 8 for EP_RAW_UP: 206 us, 224 with 4;
//   * the 64-channel layers with a third ring slot and 4 warps: 75 us, 62 so;
//   * the 96-channel layer with J = 4 and one slot: 0.42 ms, 0.22 so.
int dispatch_conv(int cin, int npad, int loader, int ep, const ConvArgs& a, cudaStream_t s)
{
#define I360B_CONV(CI, NP, TW, J, ST, LD, EP_, EW, BUFS)      \
    if (cin == CI && npad == NP && loader == LD && ep == EP_) \
        return run_conv<CI, NP, TW, J, ST, LD, EP_, EW, BUFS>(a, s);
    I360B_CONV(16, 32, 16, 4, 3, LD_PLAIN, EP_RELU, 8, 2)
    I360B_CONV(32, 32, 16, 4, 2, LD_PLAIN, EP_RELU, 8, 1)
    I360B_CONV(32, 32, 16, 4, 2, LD_PLAIN, EP_RELU_POOL, 8, 1)
    I360B_CONV(32, 64, 8, 4, 3, LD_PLAIN, EP_RELU, 8, 1)
    I360B_CONV(64, 64, 8, 2, 2, LD_PLAIN, EP_RELU, 8, 1)
    I360B_CONV(96, 32, 16, 2, 2, LD_CONCAT, EP_RELU, 8, 1)
    I360B_CONV(96, 32, 8, 2, 2, LD_SPLIT, EP_RELU, 8, 1)
    I360B_CONV(32, 16, 16, 4, 2, LD_PLAIN, EP_LOGITS, 8, 1)
    I360B_CONV(32, 16, 16, 4, 2, LD_PLAIN, EP_COMPOSITE, 16, 1)
    // backward data
    I360B_CONV(16, 32, 16, 4, 3, LD_PLAIN, EP_MASK, 8, 2)
    I360B_CONV(32, 32, 16, 4, 2, LD_PLAIN, EP_MASK, 8, 1)
    I360B_CONV(32, 96, 8, 2, 3, LD_PLAIN, EP_RAW, 8, 1)
    I360B_CONV(32, 96, 8, 2, 3, LD_PLAIN, EP_RAW_UP, 8, 2)
    I360B_CONV(64, 64, 8, 2, 2, LD_PLAIN, EP_MASK, 8, 1)
    I360B_CONV(64, 32, 8, 4, 2, LD_PLAIN, EP_RAW, 4, 1)
#undef I360B_CONV
    return fail(I360B_NOT_SUPPORTED, "conv3x3: no kernel for cin=%d cout=%d loader=%d epilogue=%d", cin, npad, loader,
                ep);
}

// The kernel of a layer's jobs (of those of a plain input where 96 channels
// are concatenated), -1 where there is none.
int wgrad_kind(int cin, int cout)
{
    return cout == 64                  ? (cin == 32 || cin == 64 ? WG_32_64 : -1)
           : cout == 16                ? (cin == 32 ? WG_32_16 : -1)
           : cout != 32                ? -1
           : cin == 16                 ? WG_16_32
           : cin == 32 || cin == 96    ? WG_32_32
                                       : -1;
}

// Slices of a layer's sums at most: one 128-row block of (tap, cin) per SM.
int wgrad_slices(int cin) { return std::max(1, sm_count() / ((9 * cin / 8 + 15) / 16)); }

// The weight and bias gradients of one layer.
struct WgradLayer
{
    const bf16* x;  // [n][h][w][cin], or the skip [n][h][w][cs] where cs > 0
    const bf16* u;  // [n][h/2][w/2][cin - cs]
    int cs;
    const bf16* g;  // [n][h][w][cout]
    int n, h, w, cin, cout, coutReal;
    float *dw, *db;  // db may be null
    const bf16* mixed = nullptr;  // [n][h][w][32]: the 32 channels from cs / 32 * 32 on, where cs % 32 != 0

    int slices() const
    {
        const long long tiles = (long long)n * ((h + kWgRows - 1) / kWgRows) * (w / kWgTW);
        return (int)std::max<long long>(1, std::min<long long>(tiles, wgrad_slices(cin)));
    }
    size_t partials() const { return (size_t)slices() * (9 * cin * cout + cout); }
};

// Partial sums of the network's layers in one batch, the most at a time.
size_t wgrad_scratch_bytes()
{
    constexpr int shapes[][2] = {{16, 32}, {32, 32}, {32, 64}, {64, 64}, {64, 64}, {96, 32}, {32, 32}, {32, 16}};
    size_t floats = 0;
    for (const auto& c : shapes) floats += (size_t)(9 * c[0] * c[1] + c[1]) * wgrad_slices(c[0]);
    return floats * sizeof(float);
}

// `count` layers in one launch each of the sums and of their reduction.
int run_wgrad(const WgradLayer* layers, int count, int* error, void* scratch, size_t bytes, cudaStream_t s)
{
    static std::once_flag once;
    static cudaError_t attrErr = cudaSuccess;
    std::call_once(once, [] {
        attrErr = cudaFuncSetAttribute(k_conv3x3_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWgSmem);
    });
    if (attrErr != cudaSuccess) return cuda_fail(attrErr, "wgrad attributes");
    WgradBatch b{};
    WgradReduce r{};
    b.error = error;
    float* part = static_cast<float*>(scratch);
    size_t used = 0;
    int blocks = 0, reduceBlocks = 0;
    for (int i = 0; i < count; ++i)
    {
        const WgradLayer& L = layers[i];
        const int kind = wgrad_kind(L.cin, L.cout);
        if (kind < 0 || (L.cs % 32 && !L.mixed) || (L.cs > 0 && L.cin != 96))
            return fail(I360B_NOT_SUPPORTED, "conv3x3 wgrad: no kernel for cin=%d cout=%d loader=%d", L.cin, L.cout,
                        L.cs ? LD_CONCAT : LD_PLAIN);
        used += L.partials() * sizeof(float);
        if (used > bytes) return fail(I360B_OUT_OF_MEMORY, "wgrad scratch too small");
        for (int c = 0; c < L.cin; c += 32)
        {
            if (b.jobs == kWgJobs) return fail(I360B_NOT_SUPPORTED, "conv3x3 wgrad: batch too large");
            WgradJob& j = b.job[b.jobs++];
            const int cx = std::min(L.cin, 32);
            const bool up = L.cs > 0 && c >= L.cs, mixed = L.cs > c && L.cs < c + 32;
            j.kind = up ? WG_UP32_32 : kind;
            j.firstBlock = blocks;
            j.slices = L.slices();
            j.n = L.n;
            j.h = L.h;
            j.w = L.w;
            j.cin = L.cin;
            j.c0 = c;
            j.xc0 = up ? c - L.cs : mixed ? 0 : c;
            j.bias = L.db && c == 0;
            j.partial = part;
            if (up)
                I360B_TRY(make_tile_map(&j.mapX, L.u, L.cin - L.cs, L.n, L.h / 2, L.w / 2, cx, kWgTW / 2, 2,
                                        swizzle_of(cx)));
            else if (mixed)
                I360B_TRY(make_parity_map(&j.mapX, L.mixed, cx, L.n, L.h, L.w, cx, kWgTW / 2, kWgRows + 2));
            else
                I360B_TRY(make_parity_map(&j.mapX, L.x, L.cs > 0 ? L.cs : L.cin, L.n, L.h, L.w, cx, kWgTW / 2,
                                          kWgRows + 2));
            I360B_TRY(make_parity_map(&j.mapG, L.g, L.cout, L.n, L.h, L.w, L.cout, kWgTW / 2, kWgRows));
            blocks += j.slices;
        }
        r.layer[r.layers++] = {part, L.slices(), L.cin, L.cout, L.coutReal, reduceBlocks, L.dw, L.db};
        reduceBlocks += (9 * L.cin * L.cout + L.cout + 127) / 128;
        part += L.partials();
    }
    k_conv3x3_wgrad<<<blocks, 192, kWgSmem, s>>>(b);
    I360B_TRY(check_launch("wgrad kernel"));
    k_wgrad_reduce<<<reduceBlocks, 128, 0, s>>>(r);
    return check_launch("wgrad reduce kernel");
}

// Channels [c0, c0 + cn) of the concatenation as a tensor of its own (dev_free
// it on `s`).
int concatenate(const bf16* x, const bf16* u, int cs, int cin, int c0, int cn, int n, int h, int w, void** out,
                cudaStream_t s)
{
    const long long units = (long long)n * h * w * (cn / 8);
    I360B_TRY(dev_alloc(out, (size_t)units * 16, s, "concatenated input"));
    k_concat<<<elementwise_grid(units), 256, 0, s>>>(x, u, cs, cin, c0, cn, n, h, w, static_cast<bf16*>(*out));
    const int rc = check_launch("concatenation kernel");
    if (rc != I360B_SUCCESS)
    {
        dev_free(*out, s);
        *out = nullptr;
    }
    return rc;
}

// A concatenated input of the forward convolution whose split is not the first
// tile's 32 channels: concatenated first, a few images at a time, in scratch
// of at most kConcatBytes (one image where that is more).
constexpr size_t kConcatBytes = size_t(256) << 20;

int conv_other_split(ConvArgs a, int cin, int npad, int ep, cudaStream_t s)
{
    const size_t px = (size_t)a.h * a.w;
    const int images = a.n, per = (int)std::min<size_t>(images, std::max<size_t>(1, kConcatBytes / (px * cin * sizeof(bf16))));
    const bf16 *x = a.x, *u = a.u;
    bf16* out = static_cast<bf16*>(a.out);
    for (int i = 0; i < images; i += per)
    {
        void* full = nullptr;
        a.n = std::min(per, images - i);
        I360B_TRY(concatenate(x + i * px * a.cs, u + i * (px / 4) * (cin - a.cs), a.cs, cin, 0, cin, a.n, a.h, a.w, &full, s));
        a.x = static_cast<const bf16*>(full);
        a.out = out + i * px * npad;
        const int rc = dispatch_conv(cin, npad, LD_SPLIT, ep, a, s);
        dev_free(full, s);
        if (rc != I360B_SUCCESS) return rc;
    }
    return I360B_SUCCESS;
}

int check_window(int n, int w, int h)
{
    if (n <= 0 || w <= 0 || h <= 0) return fail(I360B_INVALID_PARAM, "Invalid dimensions.");
    if (w % 256 != 0 || h % 2 != 0)
        return fail(I360B_INVALID_PARAM, "blend network windows need width %% 256 == 0 and even height (got %dx%d)", w,
                    h);
    return I360B_SUCCESS;
}
}  // namespace

// ---------------------------------------------------------------------------
// The network object
// ---------------------------------------------------------------------------
struct BlendNet
{
    int device = 0;
    long long wOff[kNumLayers], bOff[kNumLayers];
    int nParams = 0;
    float* params = nullptr;
    float* grads = nullptr;
    float* adamM = nullptr;
    float* adamV = nullptr;
    bf16* packed = nullptr;  // forward and backward-data weights of all layers
    float* biasPacked = nullptr;
    bf16* fwdW[kNumLayers];
    bf16* dgW[kNumLayers];
    float* bias[kNumLayers];
    int step = 0;
    // Per-batch buffers (grown on demand).
    size_t capPix = 0;
    bool capTraining = false;
    char* act = nullptr;
    bf16 *x0 = nullptr, *a1 = nullptr, *a2 = nullptr, *p2 = nullptr, *a3 = nullptr, *a4 = nullptr, *a5 = nullptr,
         *a6 = nullptr, *a7 = nullptr;
    float* logits = nullptr;
    bf16 *g8 = nullptr, *gA = nullptr, *gB = nullptr, *du = nullptr, *gh1 = nullptr, *gh2 = nullptr, *dp = nullptr,
         *gC = nullptr, *gh3 = nullptr;
    void* wgScratch = nullptr;  // behind the activations
    size_t wgBytes = 0;
    double* dLoss = nullptr;
    int* dError = nullptr;
    i360b_blend_job* dJobs = nullptr;
    i360b_blend_job* hJobs = nullptr;  // pinned staging
    int jobCap = 0;
    cudaEvent_t jobsUploaded = nullptr;
    // Recorded at the end of every call on the caller's stream; the next call
    // (possibly on another stream) waits for it, because all calls share the
    // activation buffers and the job table.
    cudaEvent_t lastUse = nullptr;
    std::mutex mu;

    int begin(cudaStream_t s)
    {
        I360B_CUDA(cudaStreamWaitEvent(s, lastUse, 0), "blend network ordering");
        return I360B_SUCCESS;
    }
    int end(cudaStream_t s, int rc)
    {
        cudaEventRecord(lastUse, s);
        return rc;
    }

    ~BlendNet()
    {
        cudaFree(params);
        cudaFree(grads);
        cudaFree(adamM);
        cudaFree(adamV);
        cudaFree(packed);
        cudaFree(biasPacked);
        cudaFree(act);
        cudaFree(dLoss);
        cudaFree(dError);
        cudaFree(dJobs);
        if (hJobs) cudaFreeHost(hJobs);
        if (jobsUploaded) cudaEventDestroy(jobsUploaded);
        if (lastUse) cudaEventDestroy(lastUse);
    }

    int init(unsigned long long seed)
    {
        long long off = 0;
        for (int l = 0; l < kNumLayers; ++l)
        {
            wOff[l] = off;
            off += 9LL * kNet[l].cin * kNet[l].cout;
            bOff[l] = off;
            off += kNet[l].cout;
        }
        nParams = (int)off;
        const size_t pb = (size_t)nParams * sizeof(float);
        I360B_CUDA(cudaMalloc(&params, pb), "blendnet params");
        I360B_CUDA(cudaMalloc(&grads, pb), "blendnet grads");
        I360B_CUDA(cudaMalloc(&adamM, pb), "blendnet adam");
        I360B_CUDA(cudaMalloc(&adamV, pb), "blendnet adam");
        I360B_CUDA(cudaMemset(adamM, 0, pb), "blendnet adam");
        I360B_CUDA(cudaMemset(adamV, 0, pb), "blendnet adam");
        size_t pk = 0, bk = 0;
        for (int l = 0; l < kNumLayers; ++l)
        {
            pk += (size_t)pad16(kNet[l].cout) * 9 * kNet[l].cin + (size_t)kNet[l].cin * 9 * pad16(kNet[l].cout);
            bk += pad16(kNet[l].cout);
        }
        I360B_CUDA(cudaMalloc(&packed, pk * sizeof(bf16)), "blendnet packed weights");
        I360B_CUDA(cudaMalloc(&biasPacked, bk * sizeof(float)), "blendnet packed bias");
        size_t o = 0, ob = 0;
        for (int l = 0; l < kNumLayers; ++l)
        {
            fwdW[l] = packed + o;
            o += (size_t)pad16(kNet[l].cout) * 9 * kNet[l].cin;
            dgW[l] = packed + o;
            o += (size_t)kNet[l].cin * 9 * pad16(kNet[l].cout);
            bias[l] = biasPacked + ob;
            ob += pad16(kNet[l].cout);
        }
        I360B_CUDA(cudaMalloc(&dLoss, sizeof(double)), "blendnet loss");
        I360B_CUDA(cudaMalloc(&dError, sizeof(int)), "blendnet error flag");
        I360B_CUDA(cudaMemset(dError, 0, sizeof(int)), "blendnet error flag");
        I360B_CUDA(cudaEventCreateWithFlags(&jobsUploaded, cudaEventDisableTiming), "blendnet event");
        I360B_CUDA(cudaEventCreateWithFlags(&lastUse, cudaEventDisableTiming), "blendnet event");
        I360B_CUDA(cudaEventRecord(lastUse, nullptr), "blendnet event");
        // He-normal weights, zero biases, zero last layer (the untrained head
        // is then the coverage-weighted mean of the layers).
        std::vector<float> h(nParams, 0.0f);
        std::mt19937_64 rng(seed);
        std::normal_distribution<float> nd(0.0f, 1.0f);
        for (int l = 0; l < kNumLayers - 1; ++l)
        {
            const float sd = std::sqrt(2.0f / (9.0f * kNet[l].cin));
            for (long long i = 0; i < 9LL * kNet[l].cin * kNet[l].cout; ++i) h[wOff[l] + i] = nd(rng) * sd;
        }
        return upload(h.data());
    }

    int upload(const float* host)
    {
        I360B_CUDA(cudaMemcpy(params, host, (size_t)nParams * sizeof(float), cudaMemcpyHostToDevice), "param upload");
        return pack(nullptr);
    }

    int pack(cudaStream_t s)
    {
        PackArgs a;
        a.params = params;
        for (int l = 0; l < kNumLayers; ++l)
        {
            a.cin[l] = kNet[l].cin;
            a.cout[l] = kNet[l].cout;
            a.wOff[l] = wOff[l];
            a.bOff[l] = bOff[l];
            a.fwd[l] = fwdW[l];
            a.dgrad[l] = dgW[l];
            a.bias[l] = bias[l];
        }
        k_pack_weights<<<dim3(64, kNumLayers), 256, 0, s>>>(a);
        return check_launch("weight pack kernel");
    }

    // Activation buffers for n windows of w x h; the backward buffers and the
    // weight gradients' scratch (20 MB) only when training.
    int reserve(int n, int w, int h, bool training)
    {
        const size_t pix = (size_t)n * w * h;
        if (pix <= capPix && (!training || capTraining)) return I360B_SUCCESS;
        cudaDeviceSynchronize();
        cudaFree(act);
        act = nullptr;
        capPix = 0;
        const size_t half = pix / 4;
        const size_t tr = training ? 1 : 0;
        // bf16 element counts of every buffer, then the fp32 logits.
        const size_t counts[] = {pix * 16,       pix * 32,       pix * 32,       half * 32,      half * 64,
                                 half * 64,      half * 64,      pix * 32,       pix * 32,       tr * pix * 16,
                                 tr * pix * 32,  tr * pix * 32,  tr * pix * 32,  tr * half * 64, tr * half * 64,
                                 tr * half * 32, tr * pix * 32,  tr * half * 64};
        size_t total = 0;
        for (size_t c : counts) total += (c * sizeof(bf16) + 255) / 256 * 256;
        total += pix * 4 * sizeof(float);
        wgBytes = tr * wgrad_scratch_bytes();
        total += wgBytes;
        cudaError_t e = cudaMalloc(&act, total);
        if (e != cudaSuccess)
        {
            cudaGetLastError();
            act = nullptr;
            return fail(I360B_OUT_OF_MEMORY, "blend network: %zu bytes of activations for %d windows of %dx%d", total,
                        n, w, h);
        }
        bf16** slots[] = {&x0, &a1, &a2, &p2, &a3, &a4, &a5, &a6, &a7, &g8, &gA, &gB, &du, &gh1, &gh2, &dp, &gC, &gh3};
        size_t o = 0;
        for (size_t i = 0; i < sizeof(counts) / sizeof(counts[0]); ++i)
        {
            *slots[i] = reinterpret_cast<bf16*>(act + o);
            o += (counts[i] * sizeof(bf16) + 255) / 256 * 256;
        }
        logits = reinterpret_cast<float*>(act + o);
        wgScratch = act + o + pix * 4 * sizeof(float);
        capPix = pix;
        capTraining = training;
        return I360B_SUCCESS;
    }

    int upload_jobs(const i360b_blend_job* jobs, int n, cudaStream_t s)
    {
        if (!jobs) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
        if (n > jobCap)
        {
            cudaDeviceSynchronize();
            cudaFree(dJobs);
            if (hJobs) cudaFreeHost(hJobs);
            dJobs = nullptr;
            hJobs = nullptr;
            jobCap = 0;
            I360B_CUDA(cudaMalloc(&dJobs, (size_t)n * sizeof(i360b_blend_job)), "blend jobs");
            I360B_CUDA(cudaMallocHost(&hJobs, (size_t)n * sizeof(i360b_blend_job)), "blend jobs");
            jobCap = n;
        }
        else
        {
            I360B_CUDA(cudaEventSynchronize(jobsUploaded), "blend jobs");
        }
        std::memcpy(hJobs, jobs, (size_t)n * sizeof(i360b_blend_job));
        I360B_CUDA(cudaMemcpyAsync(dJobs, hJobs, (size_t)n * sizeof(i360b_blend_job), cudaMemcpyHostToDevice, s),
                   "blend jobs");
        I360B_CUDA(cudaEventRecord(jobsUploaded, s), "blend jobs");
        return I360B_SUCCESS;
    }

    ConvArgs conv(const bf16* x, int n, int w, int h, int l, void* out, const i360b_blend_job* jobs) const
    {
        ConvArgs a{};
        a.x = x;
        a.n = n;
        a.h = h;
        a.w = w;
        a.wt = fwdW[l];
        a.bias = bias[l];
        a.out = out;
        a.jobs = jobs;
        a.error = dError;
        return a;
    }

    // Forward pass over the windows jobs[0..n); the last layer writes logits
    // (training) or the blended output (composite).  With `ev` non-null,
    // records ev[i] before kernel i and ev[kForwardKernels] after the last.
    static constexpr int kForwardKernels = 10;
    int forward(const i360b_blend_job* jobs, int n, int w, int h, bool composite, cudaStream_t s,
                cudaEvent_t* ev = nullptr)
    {
        const int hw = w / 2, hh = h / 2;
        auto mark = [&](int i) {
            if (ev) cudaEventRecord(ev[i], s);
        };
        mark(0);
        k_pack_input<<<elementwise_grid((long long)n * w * h), 256, 0, s>>>(jobs, n, h, w, x0);
        I360B_TRY(check_launch("input pack kernel"));
        mark(1);
        I360B_TRY(dispatch_conv(16, 32, LD_PLAIN, EP_RELU, conv(x0, n, w, h, 0, a1, jobs), s));
        mark(2);
        ConvArgs c2 = conv(a1, n, w, h, 1, a2, jobs);
        c2.half = p2;
        I360B_TRY(dispatch_conv(32, 32, LD_PLAIN, EP_RELU_POOL, c2, s));
        mark(3);
        mark(4);  // the pool, a part of conv2
        I360B_TRY(dispatch_conv(32, 64, LD_PLAIN, EP_RELU, conv(p2, n, hw, hh, 2, a3, jobs), s));
        mark(5);
        I360B_TRY(dispatch_conv(64, 64, LD_PLAIN, EP_RELU, conv(a3, n, hw, hh, 3, a4, jobs), s));
        mark(6);
        I360B_TRY(dispatch_conv(64, 64, LD_PLAIN, EP_RELU, conv(a4, n, hw, hh, 4, a5, jobs), s));
        mark(7);
        ConvArgs c6 = conv(a2, n, w, h, 5, a6, jobs);
        c6.u = a5;
        c6.cs = 32;
        I360B_TRY(dispatch_conv(96, 32, LD_CONCAT, EP_RELU, c6, s));
        mark(8);
        I360B_TRY(dispatch_conv(32, 32, LD_PLAIN, EP_RELU, conv(a6, n, w, h, 6, a7, jobs), s));
        mark(9);
        if (composite) I360B_TRY(dispatch_conv(32, 16, LD_PLAIN, EP_COMPOSITE, conv(a7, n, w, h, 7, nullptr, jobs), s));
        else I360B_TRY(dispatch_conv(32, 16, LD_PLAIN, EP_LOGITS, conv(a7, n, w, h, 7, logits, jobs), s));
        mark(10);
        return I360B_SUCCESS;
    }

    // Backward data through layer l (flipped, transposed weights).
    int dgrad(int l, const bf16* g, int n, int w, int h, const bf16* actMask, void* out, int ep, cudaStream_t s,
              bf16* half = nullptr)
    {
        ConvArgs a{};
        a.x = g;
        a.n = n;
        a.h = h;
        a.w = w;
        a.wt = dgW[l];
        a.out = out;
        a.act = actMask;
        a.half = half;
        a.error = dError;
        return dispatch_conv(pad16(kNet[l].cout), kNet[l].cin, LD_PLAIN, ep, a, s);
    }

    WgradLayer wgrad(int l, const bf16* x, const bf16* g, int n, int w, int h, const bf16* u = nullptr, int cs = 0) const
    {
        return {x, u, cs, g, n, h, w, kNet[l].cin, pad16(kNet[l].cout), kNet[l].cout, grads + wOff[l], grads + bOff[l]};
    }

    // Loss, then every parameter gradient into `grads`: the output gradients
    // of all layers first, g1 .. g8 from the last down, then the layers' weight
    // gradients in one batch.
    int backward(int n, int w, int h, cudaStream_t s)
    {
        const int hw = w / 2, hh = h / 2;
        const long long pix = (long long)n * w * h;
        I360B_CUDA(cudaMemsetAsync(dLoss, 0, sizeof(double), s), "loss reset");
        k_loss<<<elementwise_grid(pix), 256, 0, s>>>(dJobs, n, h, w, reinterpret_cast<const float4*>(logits),
                                                   (float)(1.0 / (3.0 * (double)pix)), g8, dLoss);
        I360B_TRY(check_launch("loss kernel"));
        // layer 8 (32 -> 4): input a7
        I360B_TRY(dgrad(7, g8, n, w, h, a7, gA, EP_MASK, s));  // gA = g7
        // layer 7 (32 -> 32): input a6
        I360B_TRY(dgrad(6, gA, n, w, h, a6, gB, EP_MASK, s));  // gB = g6
        // layer 6 (96 -> 32): input concat(a2, up(a5))
        I360B_TRY(dgrad(5, gB, n, w, h, a5, du, EP_RAW_UP, s, gh1));  // du of the skip, gh1 = g5
        // layer 5 (64 -> 64): input a4
        I360B_TRY(dgrad(4, gh1, n, hw, hh, a4, gh2, EP_MASK, s));  // gh2 = g4
        // layer 4 (64 -> 64): input a3
        I360B_TRY(dgrad(3, gh2, n, hw, hh, a3, gh3, EP_MASK, s));  // gh3 = g3
        // layer 3 (32 -> 64): input p2
        I360B_TRY(dgrad(2, gh3, n, hw, hh, nullptr, dp, EP_RAW, s));  // dp = d(pool)
        k_skip_grad<<<elementwise_grid(pix * 4), 256, 0, s>>>(du, 32, dp, a2, n, h, w, 4, gC);
        I360B_TRY(check_launch("skip gradient kernel"));  // gC = g2
        // layer 2 (32 -> 32): input a1; layer 1 (16 -> 32): input x0
        I360B_TRY(dgrad(1, gC, n, w, h, a1, du, EP_MASK, s));  // du = g1
        const WgradLayer layers[] = {
            wgrad(5, a2, gB, n, w, h, a5, 32), wgrad(1, a1, gC, n, w, h),     wgrad(6, a6, gA, n, w, h),
            wgrad(7, a7, g8, n, w, h),         wgrad(0, x0, du, n, w, h),     wgrad(4, a4, gh1, n, hw, hh),
            wgrad(3, a3, gh2, n, hw, hh),      wgrad(2, p2, gh3, n, hw, hh),
        };
        return run_wgrad(layers, kNumLayers, dError, wgScratch, wgBytes, s);
    }

    int adam(float lr, cudaStream_t s)
    {
        ++step;
        const float c1 = (float)(1.0 / (1.0 - std::pow(0.9, step)));
        const float c2 = (float)(1.0 / (1.0 - std::pow(0.999, step)));
        k_adam<<<(nParams + 255) / 256, 256, 0, s>>>(params, grads, adamM, adamV, nParams, lr, c1, c2);
        I360B_TRY(check_launch("adam kernel"));
        return pack(s);
    }

    int check_error(cudaStream_t s)
    {
        int e = 0;
        I360B_CUDA(cudaMemcpyAsync(&e, dError, sizeof(int), cudaMemcpyDeviceToHost, s), "error flag");
        I360B_CUDA(cudaStreamSynchronize(s), "blend network");
        if (e)
        {
            cudaMemsetAsync(dError, 0, sizeof(int), s);
            return fail(I360B_KERNEL_LAUNCH_FAILED, "a tensor-core convolution gave up waiting for its MMAs");
        }
        return I360B_SUCCESS;
    }
};
}  // namespace i360b

struct i360b_blendnet
{
    i360b::BlendNet net;
};

using namespace i360b;

namespace
{
int net_prologue(i360b_blendnet* net)
{
    clear_error();
    if (!initialized()) return fail(I360B_CUDA_ERROR, "Not initialized.");
    I360B_TRY(ensure_ready());
    if (!net) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    return I360B_SUCCESS;
}
}  // namespace

extern "C" int i360b_blendnet_param_count(void)
{
    int n = 0;
    for (int l = 0; l < kNumLayers; ++l) n += 9 * kNet[l].cin * kNet[l].cout + kNet[l].cout;
    return n;
}

extern "C" int i360b_blendnet_create(unsigned long long seed, i360b_blendnet** outNet)
{
    clear_error();
    if (!initialized()) return fail(I360B_CUDA_ERROR, "Not initialized.");
    I360B_TRY(ensure_ready());
    if (!outNet) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    *outNet = nullptr;
    auto* p = new (std::nothrow) i360b_blendnet;
    if (!p) return fail(I360B_OUT_OF_MEMORY, "blend network: host allocation failed");
    int rc = p->net.init(seed);
    if (rc != I360B_SUCCESS)
    {
        delete p;
        return rc;
    }
    I360B_CUDA(cudaDeviceSynchronize(), "blend network init");
    *outNet = p;
    return I360B_SUCCESS;
}

extern "C" void i360b_blendnet_destroy(i360b_blendnet* net)
{
    if (!net) return;
    cudaDeviceSynchronize();
    delete net;
}

extern "C" int i360b_blendnet_get_params(i360b_blendnet* net, float* hostParams, int count)
{
    I360B_TRY(net_prologue(net));
    if (!hostParams || count != net->net.nParams) return fail(I360B_INVALID_PARAM, "parameter count mismatch");
    I360B_CUDA(cudaDeviceSynchronize(), "blend network");
    I360B_CUDA(cudaMemcpy(hostParams, net->net.params, (size_t)count * sizeof(float), cudaMemcpyDeviceToHost),
               "param download");
    return I360B_SUCCESS;
}

extern "C" int i360b_blendnet_set_params(i360b_blendnet* net, const float* hostParams, int count)
{
    I360B_TRY(net_prologue(net));
    if (!hostParams || count != net->net.nParams) return fail(I360B_INVALID_PARAM, "parameter count mismatch");
    I360B_CUDA(cudaDeviceSynchronize(), "blend network");
    I360B_TRY(net->net.upload(hostParams));
    I360B_CUDA(cudaDeviceSynchronize(), "blend network");
    return I360B_SUCCESS;
}

extern "C" int i360b_blendnet_get_adam(i360b_blendnet* net, float* hostM, float* hostV, int count, int* step)
{
    I360B_TRY(net_prologue(net));
    if (!hostM || !hostV || !step || count != net->net.nParams)
        return fail(I360B_INVALID_PARAM, "parameter count mismatch");
    BlendNet& N = net->net;
    std::lock_guard<std::mutex> lk(N.mu);
    I360B_CUDA(cudaDeviceSynchronize(), "blend network");
    I360B_CUDA(cudaMemcpy(hostM, N.adamM, (size_t)count * sizeof(float), cudaMemcpyDeviceToHost), "adam download");
    I360B_CUDA(cudaMemcpy(hostV, N.adamV, (size_t)count * sizeof(float), cudaMemcpyDeviceToHost), "adam download");
    *step = N.step;
    return I360B_SUCCESS;
}

extern "C" int i360b_blendnet_set_adam(i360b_blendnet* net, const float* hostM, const float* hostV, int count,
                                       int step)
{
    I360B_TRY(net_prologue(net));
    if (!hostM || !hostV || count != net->net.nParams || step < 0)
        return fail(I360B_INVALID_PARAM, "parameter count mismatch or negative step");
    BlendNet& N = net->net;
    std::lock_guard<std::mutex> lk(N.mu);
    I360B_CUDA(cudaDeviceSynchronize(), "blend network");
    I360B_CUDA(cudaMemcpy(N.adamM, hostM, (size_t)count * sizeof(float), cudaMemcpyHostToDevice), "adam upload");
    I360B_CUDA(cudaMemcpy(N.adamV, hostV, (size_t)count * sizeof(float), cudaMemcpyHostToDevice), "adam upload");
    N.step = step;
    return I360B_SUCCESS;
}

extern "C" int i360b_blendnet_logits(i360b_blendnet* net, const i360b_blend_job* jobs, int n, int w, int h,
                                     float* dLogits)
{
    I360B_TRY(net_prologue(net));
    I360B_TRY(check_window(n, w, h));
    if (!dLogits) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    BlendNet& N = net->net;
    std::lock_guard<std::mutex> lk(N.mu);
    cudaStream_t s = thread_stream();
    I360B_TRY(N.begin(s));
    int rc = [&]() -> int {
        I360B_TRY(N.reserve(n, w, h, false));
        I360B_TRY(N.upload_jobs(jobs, n, s));
        I360B_TRY(N.forward(N.dJobs, n, w, h, false, s));
        I360B_CUDA(cudaMemcpyAsync(dLogits, N.logits, (size_t)n * w * h * 4 * sizeof(float), cudaMemcpyDeviceToDevice,
                                   s),
                   "logits copy");
        return N.check_error(s);
    }();
    return N.end(s, rc);
}

extern "C" int i360b_blendnet_gradients(i360b_blendnet* net, const i360b_blend_job* jobs, int n, int w, int h,
                                        float* hostGrad, double* hostLoss)
{
    I360B_TRY(net_prologue(net));
    I360B_TRY(check_window(n, w, h));
    BlendNet& N = net->net;
    std::lock_guard<std::mutex> lk(N.mu);
    cudaStream_t s = thread_stream();
    I360B_TRY(N.begin(s));
    int rc = [&]() -> int {
        I360B_TRY(N.reserve(n, w, h, true));
        I360B_TRY(N.upload_jobs(jobs, n, s));
        I360B_TRY(N.forward(N.dJobs, n, w, h, false, s));
        I360B_TRY(N.backward(n, w, h, s));
        I360B_TRY(N.check_error(s));
        if (hostGrad)
            I360B_CUDA(cudaMemcpy(hostGrad, N.grads, (size_t)N.nParams * sizeof(float), cudaMemcpyDeviceToHost),
                       "grad download");
        if (hostLoss)
            I360B_CUDA(cudaMemcpy(hostLoss, N.dLoss, sizeof(double), cudaMemcpyDeviceToHost), "loss download");
        return I360B_SUCCESS;
    }();
    return N.end(s, rc);
}

extern "C" int i360b_blendnet_train_step(i360b_blendnet* net, const i360b_blend_job* jobs, int n, int w, int h,
                                         float lr, double* hostLoss, void* stream)
{
    I360B_TRY(net_prologue(net));
    I360B_TRY(check_window(n, w, h));
    BlendNet& N = net->net;
    std::lock_guard<std::mutex> lk(N.mu);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    I360B_TRY(N.begin(s));
    int rc = [&]() -> int {
        I360B_TRY(N.reserve(n, w, h, true));
        I360B_TRY(N.upload_jobs(jobs, n, s));
        I360B_TRY(N.forward(N.dJobs, n, w, h, false, s));
        I360B_TRY(N.backward(n, w, h, s));
        I360B_TRY(N.adam(lr, s));
        if (hostLoss)
        {
            I360B_CUDA(cudaMemcpyAsync(hostLoss, N.dLoss, sizeof(double), cudaMemcpyDeviceToHost, s), "loss download");
            return N.check_error(s);
        }
        return I360B_SUCCESS;
    }();
    return N.end(s, rc);
}

extern "C" int i360b_blendnet_infer(i360b_blendnet* net, const i360b_blend_job* jobs, int n, int w, int h,
                                    void* stream)
{
    I360B_TRY(net_prologue(net));
    I360B_TRY(check_window(n, w, h));
    BlendNet& N = net->net;
    std::lock_guard<std::mutex> lk(N.mu);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    I360B_TRY(N.begin(s));
    int rc = [&]() -> int {
        I360B_TRY(N.reserve(n, w, h, false));
        I360B_TRY(N.upload_jobs(jobs, n, s));
        return N.forward(N.dJobs, n, w, h, true, s);
    }();
    return N.end(s, rc);
}

extern "C" int i360b_blendnet_profile(i360b_blendnet* net, const i360b_blend_job* jobs, int n, int w, int h,
                                      float* kernelMs, int maxKernels)
{
    I360B_TRY(net_prologue(net));
    I360B_TRY(check_window(n, w, h));
    if (!kernelMs) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    BlendNet& N = net->net;
    std::lock_guard<std::mutex> lk(N.mu);
    cudaStream_t s = thread_stream();
    I360B_TRY(N.begin(s));
    cudaEvent_t ev[BlendNet::kForwardKernels + 1] = {};
    int rc = [&]() -> int {
        for (auto& e : ev) I360B_CUDA(cudaEventCreate(&e), "profile events");
        I360B_TRY(N.reserve(n, w, h, false));
        I360B_TRY(N.upload_jobs(jobs, n, s));
        I360B_TRY(N.forward(N.dJobs, n, w, h, true, s, ev));
        I360B_CUDA(cudaEventSynchronize(ev[BlendNet::kForwardKernels]), "profile");
        for (int i = 0; i < BlendNet::kForwardKernels && i < maxKernels; ++i)
            cudaEventElapsedTime(&kernelMs[i], ev[i], ev[i + 1]);
        return N.check_error(s);
    }();
    for (auto& e : ev)
        if (e) cudaEventDestroy(e);
    return N.end(s, rc);
}

extern "C" const char* i360b_blendnet_kernel_name(int i)
{
    static const char* const names[] = {"pack_input", "conv1_16_32",  "conv2_32_32", "pool",        "conv3_32_64",
                                        "conv4_64_64", "conv5_64_64", "conv6_96_32", "conv7_32_32", "conv8_32_4_blend"};
    return i >= 0 && i < 10 ? names[i] : nullptr;
}

extern "C" int i360b_conv3x3_forward(const void* dX, const void* dU, int skipChannels, int n, int h, int w, int cin,
                                     int cout, const void* dWeights, const float* dBias, int epilogue,
                                     const void* dAct, void* dOut, void* stream)
{
    clear_error();
    if (!initialized()) return fail(I360B_CUDA_ERROR, "Not initialized.");
    I360B_TRY(ensure_ready());
    if (!dX || !dWeights || !dOut || (skipChannels > 0 && !dU)) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (n <= 0 || h <= 0 || w <= 0) return fail(I360B_INVALID_PARAM, "Invalid dimensions.");
    if ((epilogue == EP_RELU || epilogue == EP_LOGITS) && !dBias) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (epilogue == EP_MASK && !dAct) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (epilogue < EP_RELU || epilogue > EP_RAW) return fail(I360B_INVALID_PARAM, "unknown epilogue %d", epilogue);
    if (skipChannels > 0 && (h % 2 || w % 256 || skipChannels % 8 || skipChannels >= cin))
        return fail(I360B_INVALID_PARAM, "Invalid dimensions.");
    static int* dErr = nullptr;
    if (!dErr) I360B_CUDA(cudaMalloc(&dErr, sizeof(int)), "error flag");
    ConvArgs a{};
    a.x = static_cast<const bf16*>(dX);
    a.u = static_cast<const bf16*>(dU);
    a.cs = skipChannels;
    a.n = n;
    a.h = h;
    a.w = w;
    a.wt = static_cast<const bf16*>(dWeights);
    a.bias = dBias;
    a.out = dOut;
    a.act = static_cast<const bf16*>(dAct);
    a.error = dErr;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    I360B_CUDA(cudaMemsetAsync(dErr, 0, sizeof(int), s), "error flag");
    const bool otherSplit = skipChannels > 0 && skipChannels != 32 && cin == 96 && cout == 32 && epilogue == EP_RELU;
    const int rc = otherSplit ? conv_other_split(a, cin, cout, epilogue, s)
                              : dispatch_conv(cin, cout, skipChannels > 0 ? LD_CONCAT : LD_PLAIN, epilogue, a, s);
    if (rc != I360B_SUCCESS) return rc;
    int e = 0;
    I360B_CUDA(cudaMemcpyAsync(&e, dErr, sizeof(int), cudaMemcpyDeviceToHost, s), "error flag");
    I360B_CUDA(cudaStreamSynchronize(s), "conv3x3");
    if (e) return fail(I360B_KERNEL_LAUNCH_FAILED, "conv3x3 gave up waiting for its MMAs");
    return I360B_SUCCESS;
}

extern "C" int i360b_conv3x3_wgrad(const void* dX, const void* dU, int skipChannels, const void* dGrad, int n, int h,
                                   int w, int cin, int cout, float* dGradW, void* stream)
{
    clear_error();
    if (!initialized()) return fail(I360B_CUDA_ERROR, "Not initialized.");
    I360B_TRY(ensure_ready());
    if (!dX || !dGrad || !dGradW || (skipChannels > 0 && !dU)) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (n <= 0 || h <= 0 || w <= 0 || w % kTileX != 0) return fail(I360B_INVALID_PARAM, "Invalid dimensions.");
    if (skipChannels > 0 && (h % 2 || w % 256 || skipChannels % 8 || skipChannels >= cin))
        return fail(I360B_INVALID_PARAM, "Invalid dimensions.");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    static int* dErr = nullptr;
    if (!dErr) I360B_CUDA(cudaMalloc(&dErr, sizeof(int)), "error flag");
    WgradLayer L{static_cast<const bf16*>(dX), static_cast<const bf16*>(dU), std::max(skipChannels, 0),
                 static_cast<const bf16*>(dGrad), n, h, w, cin, cout, cout, dGradW, nullptr};
    if (wgrad_kind(cin, cout) < 0 || (L.cs > 0) != (cin == 96))
        return fail(I360B_NOT_SUPPORTED, "conv3x3 wgrad: no kernel for cin=%d cout=%d loader=%d", cin, cout,
                    L.cs > 0 ? LD_CONCAT : LD_PLAIN);
    const size_t bytes = L.partials() * sizeof(float);
    void *scratch = nullptr, *mixed = nullptr;
    I360B_TRY(dev_alloc(&scratch, bytes, s, "wgrad scratch"));
    int rc = I360B_SUCCESS;
    if (cudaMemsetAsync(dErr, 0, sizeof(int), s) != cudaSuccess) rc = cuda_fail(cudaGetLastError(), "error flag");
    if (rc == I360B_SUCCESS && L.cs % 32)
    {
        // the 32-channel job that takes channels of both inputs
        rc = concatenate(L.x, L.u, L.cs, cin, L.cs / 32 * 32, 32, n, h, w, &mixed, s);
        L.mixed = static_cast<const bf16*>(mixed);
    }
    if (rc == I360B_SUCCESS) rc = run_wgrad(&L, 1, dErr, scratch, bytes, s);
    if (mixed) dev_free(mixed, s);
    int e = 0;
    cudaMemcpyAsync(&e, dErr, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    dev_free(scratch, s);
    if (rc != I360B_SUCCESS) return rc;
    if (e) return fail(I360B_KERNEL_LAUNCH_FAILED, "conv3x3 wgrad gave up waiting for its MMAs");
    return I360B_SUCCESS;
}

// ---------------------------------------------------------------------------
// Learned render of a plan's output tiles
// ---------------------------------------------------------------------------
namespace i360b
{
namespace
{
constexpr int kSub = 256;  // learned-blend window side

// Copy (src non-null) or clear a w x h RGB48 rectangle; strides in elements.
struct Region
{
    const unsigned short* src;
    unsigned short* dst;
    int w, h;
    long long srcRow, dstRow;
};

__global__ void k_regions(const Region* __restrict__ regs, int n)
{
    for (int r = blockIdx.y; r < n; r += gridDim.y)
    {
        const Region R = regs[r];
        const int vals = R.w * 3;
        for (int y = blockIdx.x; y < R.h; y += gridDim.x)
        {
            unsigned short* d = R.dst + y * R.dstRow;
            if (R.src)
            {
                const unsigned short* src = R.src + y * R.srcRow;
                for (int i = threadIdx.x; i < vals; i += blockDim.x) d[i] = src[i];
            }
            else
                for (int i = threadIdx.x; i < vals; i += blockDim.x) d[i] = 0;
        }
    }
}

// Per region: sum of squared differences and largest absolute difference
// between two RGB48 rectangles (src = learned, dst = plain).
__global__ void k_judge(const Region* __restrict__ regs, int n, double* __restrict__ sse, int* __restrict__ maxErr)
{
    __shared__ double rs[8];
    __shared__ int rm[8];
    for (int r = blockIdx.x; r < n; r += gridDim.x)
    {
        const Region R = regs[r];
        const int vals = R.w * 3;
        double acc = 0.0;
        int mx = 0;
        for (int y = 0; y < R.h; ++y)
        {
            const unsigned short* a = R.src + y * R.srcRow;
            const unsigned short* b = R.dst + y * R.dstRow;
            for (int i = threadIdx.x; i < vals; i += blockDim.x)
            {
                const int d = (int)a[i] - (int)b[i];
                acc += (double)d * d;
                mx = max(mx, abs(d));
            }
        }
        for (int o = 16; o > 0; o >>= 1)
        {
            acc += __shfl_xor_sync(0xffffffffu, acc, o);
            mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        if ((threadIdx.x & 31) == 0)
        {
            rs[threadIdx.x >> 5] = acc;
            rm[threadIdx.x >> 5] = mx;
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            double t = 0.0;
            int m = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w)
            {
                t += rs[w];
                m = max(m, rm[w]);
            }
            sse[r] = t;
            maxErr[r] = m;
        }
        __syncthreads();
    }
}

int launch_regions(const std::vector<Region>& regs, Region* dRegs, cudaStream_t s)
{
    if (regs.empty()) return I360B_SUCCESS;
    I360B_CUDA(cudaMemcpyAsync(dRegs, regs.data(), regs.size() * sizeof(Region), cudaMemcpyHostToDevice, s),
               "region upload");
    k_regions<<<dim3(16, (unsigned)std::min<size_t>(regs.size(), 65535)), 256, 0, s>>>(dRegs, (int)regs.size());
    return check_launch("region copy kernel");
}

// Footprint box of an item intersects a rectangle (inclusive box ends).
bool box_hits(const ItemDev& it, int x0, int y0, int w, int h)
{
    return it.vx0 < x0 + w && it.vx1 >= x0 && it.vy0 < y0 + h && it.vy1 >= y0;
}

long long box_overlap(const ItemDev& it, int x0, int y0, int w, int h)
{
    const long long ix = std::max(0, std::min(it.vx1 + 1, x0 + w) - std::max(it.vx0, x0));
    const long long iy = std::max(0, std::min(it.vy1 + 1, y0 + h) - std::max(it.vy0, y0));
    return ix * iy;
}

void build_subtiles(Plan& P)
{
    if (!P.subTiles.empty()) return;
    for (int t = 0; t < P.nTiles; ++t)
    {
        const TileDev& T = P.tiles[t];
        for (int oy = 0; oy < T.h; oy += kSub)
            for (int ox = 0; ox < T.w; ox += kSub)
            {
                SubTile st{};
                st.tile = t;
                st.ox = ox;
                st.oy = oy;
                st.w = std::min(kSub, T.w - ox);
                st.h = std::min(kSub, T.h - oy);
                std::vector<std::pair<long long, int>> hits;
                for (int k = 0; k < T.numItems; ++k)
                {
                    const ItemDev& it = P.items[T.firstItem + k];
                    if (box_hits(it, ox, oy, st.w, st.h)) hits.push_back({box_overlap(it, ox, oy, st.w, st.h), k});
                }
                if (hits.size() > 4)
                {
                    st.overflow = 1;
                    std::stable_sort(hits.begin(), hits.end(),
                                     [](const auto& a, const auto& b) { return a.first > b.first; });
                    hits.resize(4);
                    std::sort(hits.begin(), hits.end(), [](const auto& a, const auto& b) { return a.second < b.second; });
                }
                for (int i = 0; i < 4; ++i) st.item[i] = i < (int)hits.size() ? T.firstItem + hits[i].second : -1;
                st.kind = hits.empty() ? 0 : hits.size() == 1 ? 1 : 2;
                P.subTiles.push_back(st);
            }
    }
}

// Device scratch of the learned render, per (plan, thread of use).
struct LearnedScratch
{
    i360b_blend_job* dJobs = nullptr;
    size_t jobCap = 0;
    Region* dRegs = nullptr;
    size_t regCap = 0;
    double* dSse = nullptr;
    int* dMax = nullptr;
    size_t judgeCap = 0;
    ~LearnedScratch()
    {
        cudaFree(dJobs);
        cudaFree(dRegs);
        cudaFree(dSse);
        cudaFree(dMax);
    }
    int jobs(size_t n)
    {
        if (n <= jobCap) return I360B_SUCCESS;
        cudaFree(dJobs);
        dJobs = nullptr;
        jobCap = 0;
        I360B_CUDA(cudaMalloc(&dJobs, std::max<size_t>(n, 1) * sizeof(i360b_blend_job)), "learned jobs");
        jobCap = n;
        return I360B_SUCCESS;
    }
    int regs(size_t n)
    {
        if (n <= regCap) return I360B_SUCCESS;
        cudaFree(dRegs);
        dRegs = nullptr;
        regCap = 0;
        I360B_CUDA(cudaMalloc(&dRegs, std::max<size_t>(n, 1) * sizeof(Region)), "learned regions");
        regCap = n;
        return I360B_SUCCESS;
    }
    int judge(size_t n)
    {
        if (n <= judgeCap) return I360B_SUCCESS;
        cudaFree(dSse);
        cudaFree(dMax);
        dSse = nullptr;
        dMax = nullptr;
        judgeCap = 0;
        I360B_CUDA(cudaMalloc(&dSse, std::max<size_t>(n, 1) * sizeof(double)), "judge");
        I360B_CUDA(cudaMalloc(&dMax, std::max<size_t>(n, 1) * sizeof(int)), "judge");
        judgeCap = n;
        return I360B_SUCCESS;
    }
};

std::mutex g_scratchMu;
std::vector<std::pair<const Plan*, LearnedScratch*>> g_scratch;

LearnedScratch& scratch_for(const Plan* p)
{
    std::lock_guard<std::mutex> lk(g_scratchMu);
    for (auto& e : g_scratch)
        if (e.first == p) return *e.second;
    g_scratch.push_back({p, new LearnedScratch});
    return *g_scratch.back().second;
}
}  // namespace

void release_learned_scratch(const Plan* p)
{
    std::lock_guard<std::mutex> lk(g_scratchMu);
    for (size_t i = 0; i < g_scratch.size(); ++i)
        if (g_scratch[i].first == p)
        {
            delete g_scratch[i].second;
            g_scratch.erase(g_scratch.begin() + i);
            return;
        }
}

int learned_render(Plan& P, BlendNet& N, unsigned short* const* tileOut, int maxBatch, cudaStream_t s, float* stageMs)
{
    if (!P.render) return fail(I360B_INVALID_PARAM, "learned render needs a render plan");
    build_subtiles(P);
    LearnedScratch& S = scratch_for(&P);
    auto outOf = [&](int t) { return tileOut ? tileOut[t] : P.tiles[t].out; };
    std::vector<i360b_blend_job> jobs;
    std::vector<Region> regs;
    for (const SubTile& st : P.subTiles)
    {
        const TileDev& T = P.tiles[st.tile];
        unsigned short* out = outOf(st.tile);
        if (!out) return fail(I360B_INVALID_PARAM, "Tile %d has a null learned output.", st.tile);
        const size_t off = ((size_t)st.oy * T.w + st.ox) * 3;
        if (st.kind == 2)
        {
            i360b_blend_job j{};
            for (int i = 0; i < 4; ++i) j.slot[i] = st.item[i] >= 0 ? P.items[st.item[i]].img + off : nullptr;
            for (int i = 0; i < 4; ++i)
                for (int e = 0; e < 4; ++e)
                {
                    const float* src = st.item[i] >= 0 ? &P.itemEdges[(size_t)st.item[i] * 16 + 4 * e] : nullptr;
                    float* d = &j.edges[i][4 * e];
                    if (!src)
                    {
                        d[0] = NAN;
                        d[1] = d[2] = d[3] = 0.0f;
                        continue;
                    }
                    d[0] = src[0] - st.ox;  // NaN stays NaN
                    d[1] = src[1] - st.oy;
                    d[2] = src[2] - st.ox;
                    d[3] = src[3] - st.oy;
                }
            j.pixStride = 3;
            j.rowStride = 3LL * T.w;
            j.width = st.w;
            j.height = st.h;
            j.out = out + off;
            j.outRowStride = 3LL * T.w;
            jobs.push_back(j);
        }
        else
        {
            regs.push_back(Region{st.kind == 1 ? P.items[st.item[0]].img + off : nullptr, out + off, st.w, st.h,
                                  3LL * T.w, 3LL * T.w});
        }
    }
    I360B_TRY(S.jobs(jobs.size()));
    I360B_TRY(S.regs(regs.size()));
    cudaEvent_t ev[4] = {};
    if (stageMs)
        for (auto& e : ev) I360B_CUDA(cudaEventCreate(&e), "stage events");
    auto mark = [&](int i) {
        if (stageMs) cudaEventRecord(ev[i], s);
    };
    mark(0);
    I360B_TRY(P.enqueue_warp(s));
    mark(1);
    I360B_TRY(launch_regions(regs, S.dRegs, s));
    mark(2);
    if (!jobs.empty())
    {
        I360B_CUDA(cudaMemcpyAsync(S.dJobs, jobs.data(), jobs.size() * sizeof(i360b_blend_job), cudaMemcpyHostToDevice,
                                   s),
                   "learned jobs upload");
        const int batch = std::max(1, std::min<int>(maxBatch, (int)jobs.size()));
        I360B_TRY(N.reserve(batch, kSub, kSub, false));
        for (size_t b = 0; b < jobs.size(); b += batch)
        {
            const int n = (int)std::min<size_t>(batch, jobs.size() - b);
            I360B_TRY(N.forward(S.dJobs + b, n, kSub, kSub, true, s));
        }
    }
    mark(3);
    if (stageMs)
    {
        I360B_CUDA(cudaEventSynchronize(ev[3]), "stage events");
        for (int i = 0; i < 3; ++i) cudaEventElapsedTime(&stageMs[i], ev[i], ev[i + 1]);
        for (auto& e : ev) cudaEventDestroy(e);
    }
    // Host vectors must outlive the asynchronous uploads.
    I360B_CUDA(cudaStreamSynchronize(s), "learned render");
    return I360B_SUCCESS;
}

int learned_judge(Plan& P, unsigned short* const* tileOut, double minPsnr, double peak, i360b_learned_stats* st,
                  float* psnrOut, int maxOut, cudaStream_t s)
{
    build_subtiles(P);
    LearnedScratch& S = scratch_for(&P);
    const size_t n = P.subTiles.size();
    std::vector<Region> regs(n);
    for (size_t i = 0; i < n; ++i)
    {
        const SubTile& t = P.subTiles[i];
        const TileDev& T = P.tiles[t.tile];
        const size_t off = ((size_t)t.oy * T.w + t.ox) * 3;
        if (!tileOut[t.tile]) return fail(I360B_INVALID_PARAM, "Tile %d has a null learned output.", t.tile);
        regs[i] = Region{tileOut[t.tile] + off, P.tiles[t.tile].out + off, t.w, t.h, 3LL * T.w, 3LL * T.w};
    }
    I360B_TRY(S.regs(n));
    I360B_TRY(S.judge(n));
    if (n)
    {
        I360B_CUDA(cudaMemcpyAsync(S.dRegs, regs.data(), n * sizeof(Region), cudaMemcpyHostToDevice, s), "judge");
        k_judge<<<(unsigned)std::min<size_t>(n, 65535), 256, 0, s>>>(S.dRegs, (int)n, S.dSse, S.dMax);
        I360B_TRY(check_launch("judge kernel"));
    }
    std::vector<double> sse(n);
    std::vector<int> mx(n);
    if (n)
    {
        I360B_CUDA(cudaMemcpyAsync(sse.data(), S.dSse, n * sizeof(double), cudaMemcpyDeviceToHost, s), "judge");
        I360B_CUDA(cudaMemcpyAsync(mx.data(), S.dMax, n * sizeof(int), cudaMemcpyDeviceToHost, s), "judge");
    }
    I360B_CUDA(cudaStreamSynchronize(s), "judge");
    i360b_learned_stats r{};
    r.subTiles = (int)n;
    r.minPsnr = INFINITY;
    double psum = 0.0;
    int pcount = 0;
    std::vector<Region> fallback;
    for (size_t i = 0; i < n; ++i)
    {
        const SubTile& t = P.subTiles[i];
        r.netSubTiles += t.kind == 2;
        r.copySubTiles += t.kind == 1;
        r.emptySubTiles += t.kind == 0;
        r.overflowSubTiles += t.overflow;
        const double cnt = 3.0 * t.w * t.h;
        const double mse = sse[i] / cnt;
        const double psnr = mse > 0.0 ? 10.0 * std::log10(peak * peak / mse) : INFINITY;
        if (psnrOut && (int)i < maxOut) psnrOut[i] = (float)psnr;
        r.maxAbsError = std::max(r.maxAbsError, mx[i]);
        r.minPsnr = std::min(r.minPsnr, psnr);
        if (std::isfinite(psnr))
        {
            psum += psnr;
            ++pcount;
        }
        if (psnr < minPsnr)
        {
            ++r.fallbackSubTiles;
            // plain -> learned output
            fallback.push_back(
                Region{regs[i].dst, const_cast<unsigned short*>(regs[i].src), t.w, t.h, regs[i].dstRow, regs[i].srcRow});
        }
    }
    r.judgedSubTiles = (int)n;
    r.meanPsnr = pcount ? psum / pcount : INFINITY;
    I360B_TRY(S.regs(std::max(n, fallback.size())));
    I360B_TRY(launch_regions(fallback, S.dRegs, s));
    I360B_CUDA(cudaStreamSynchronize(s), "judge fallback");
    if (st) *st = r;
    return I360B_SUCCESS;
}
}  // namespace i360b

extern "C" int i360b_render_plan_learned(i360b_render_plan* plan, i360b_blendnet* net,
                                         unsigned short* const* dTileOut, int maxBatch, void* stream, float* stageMs)
{
    I360B_TRY(net_prologue(net));
    if (!plan) return fail(I360B_INVALID_PARAM, "Null plan.");
    if (maxBatch < 1) return fail(I360B_INVALID_PARAM, "maxBatch must be >= 1.");
    BlendNet& N = net->net;
    std::lock_guard<std::mutex> lk(N.mu);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    I360B_TRY(N.begin(s));
    int rc = learned_render(plan->plan, N, dTileOut, maxBatch, s, stageMs);
    if (rc == I360B_SUCCESS) rc = N.check_error(s);
    return N.end(s, rc);
}

extern "C" int i360b_render_plan_judge(i360b_render_plan* plan, unsigned short* const* dTileOut, double minPsnrDb,
                                       double peak, i360b_learned_stats* stats, float* hostSubTilePsnr,
                                       int maxSubTiles, void* stream)
{
    clear_error();
    if (!initialized()) return fail(I360B_CUDA_ERROR, "Not initialized.");
    I360B_TRY(ensure_ready());
    if (!plan || !dTileOut) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (!(peak > 0.0)) return fail(I360B_INVALID_PARAM, "peak must be > 0.");
    return learned_judge(plan->plan, dTileOut, minPsnrDb, peak, stats, hostSubTilePsnr, maxSubTiles,
                         static_cast<cudaStream_t>(stream));
}

extern "C" int i360b_render_plan_windows(i360b_render_plan* plan, int maxWindows, int* info, int* numWindows)
{
    clear_error();
    if (!plan || !numWindows) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    Plan& P = plan->plan;
    if (!P.render) return fail(I360B_INVALID_PARAM, "not a render plan");
    build_subtiles(P);
    *numWindows = (int)P.subTiles.size();
    if (info)
        for (int i = 0; i < (int)P.subTiles.size() && i < maxWindows; ++i)
        {
            const SubTile& t = P.subTiles[i];
            int* o = info + 6 * i;
            o[0] = t.tile;
            o[1] = t.ox;
            o[2] = t.oy;
            o[3] = t.kind;
            o[4] = t.overflow;
            o[5] = (t.item[0] >= 0) + (t.item[1] >= 0) + (t.item[2] >= 0) + (t.item[3] >= 0);
        }
    return I360B_SUCCESS;
}

extern "C" int i360b_render_plan_tile_items(i360b_render_plan* plan, int tile, int maxItems,
                                            const unsigned short** dImages, int* boxes, float* edges, int* numItems)
{
    clear_error();
    if (!plan || !numItems) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    const Plan& P = plan->plan;
    if (tile < 0 || tile >= P.nTiles) return fail(I360B_INVALID_PARAM, "Tile %d out of range.", tile);
    if (!P.render) return fail(I360B_INVALID_PARAM, "not a render plan");
    const TileDev& T = P.tiles[tile];
    *numItems = T.numItems;
    for (int k = 0; k < T.numItems && k < maxItems; ++k)
    {
        const ItemDev& it = P.items[T.firstItem + k];
        if (dImages) dImages[k] = it.img;
        if (boxes)
        {
            boxes[4 * k] = it.vx0;
            boxes[4 * k + 1] = it.vy0;
            boxes[4 * k + 2] = it.vx1;
            boxes[4 * k + 3] = it.vy1;
        }
        if (edges)
            for (int q = 0; q < 16; ++q) edges[16 * k + q] = P.itemEdges[(size_t)(T.firstItem + k) * 16 + q];
    }
    return I360B_SUCCESS;
}
