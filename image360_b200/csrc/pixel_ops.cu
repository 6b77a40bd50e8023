// Per-pixel render-path kernels: fused Bayer demosaic, backward homography
// warp (+ gain), sigma-clipped median stack and gain.  Each reproduces the
// reference CPU backend's arithmetic bit for bit (FP32, no FMA contraction,
// truncation at the same points) so outputs match Kernels::Scalar::* exactly.
#include "common.cuh"
#include "warp_taps.cuh"

namespace i360b
{
// ---------------------------------------------------------------------------
// Demosaic: BlackLevelSubtract -> WhiteBalance -> bilinear 3x3 -> 3x4 matrix,
// one pass (BayerDemosaic_Scalar.cpp:9-50, BayerDemosaicKernels.h:10-75).
// A CTA stages its (TH+2) x (TW+2) CFA footprint in shared memory with the
// black level and white balance already applied, then each thread demosaics
// and colour-corrects 2x2 output pixels.
// ---------------------------------------------------------------------------
namespace
{
constexpr int kDmTW = 64, kDmTH = 16;

struct DemosaicParams
{
    float camMul[4];
    float rgbCam[12];
    uint32_t filters;
    unsigned short black;
    // Standard Bayer layout (2x2-periodic, one R, one B, G on a diagonal):
    // colour of site (y & 1, x & 1), else std2x2 = 0 and only the generic
    // path runs.
    int std2x2;
    int color2x2[4];
};

__host__ __device__ __forceinline__ int bayer_color(int row, int col, uint32_t filters)
{
    // BayerDemosaicKernels.h:10-13.
    return (int)((filters >> ((((row << 1) & 14) | (col & 1)) << 1)) & 3u);
}

// 3x3 same-colour average of DemosaicPixel (BayerDemosaicKernels.h:25-60) for
// any filter word and any position (borders average fewer neighbours).
template <int PITCH>
__device__ __forceinline__ void demosaic_generic(const float (*s)[PITCH], int lx, int ly, int x, int y, int w, int h,
                                                 uint32_t filters, float rgb[3])
{
    float acc[3] = {0.0f, 0.0f, 0.0f};
    int cnt[3] = {0, 0, 0};
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx)
        {
            int nx = x + dx, ny = y + dy;
            if (nx < 0 || ny < 0 || nx >= w || ny >= h) continue;
            int ch = bayer_color(ny, nx, filters);
            int slot = ch == 3 ? 1 : ch;
            float v = s[ly + 1 + dy][lx + 1 + dx];
            // Integer-valued sums below 2^24: exact in any order.
            if (slot == 0) { acc[0] += v; cnt[0]++; }
            else if (slot == 1) { acc[1] += v; cnt[1]++; }
            else { acc[2] += v; cnt[2]++; }
        }
    int mine = bayer_color(y, x, filters);
    int my = mine == 3 ? 1 : mine;
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
        float v = acc[c];
        if (c == my) v = s[ly + 1][lx + 1];
        else if (cnt[c] != 0) v = fdiv(v, u2f((uint32_t)cnt[c]));
        rgb[c] = v;
    }
}

// Black level and white balance of one CFA value (BayerDemosaicKernels.h
// BLS/WB steps): the uint16 truncation and the float that the interpolation
// reads in one step (clamp_floor_u16f); `mul` is the multiplier of the
// value's colour.
__device__ __forceinline__ float demosaic_level(unsigned raw, float mul, const DemosaicParams& P)
{
    raw = raw > P.black ? raw - P.black : 0u;
    return clamp_floor_u16f(fmul(u2f(raw), mul));
}

// Truncate to uint16 (DemosaicPixel), then the 3x4 colour matrix
// (ApplyColorMatrixPixel, BayerDemosaicKernels.h:64-75).
__device__ __forceinline__ void demosaic_matrix(const DemosaicParams& P, float R, float G, float B, unsigned short* px)
{
    const float r = clamp_floor_u16f(R), g = clamp_floor_u16f(G), b = clamp_floor_u16f(B);
#pragma unroll
    for (int row = 0; row < 3; ++row)
    {
        float val = fadd(fadd(fadd(fmul(P.rgbCam[row * 4 + 0], r), fmul(P.rgbCam[row * 4 + 1], g)),
                              fmul(P.rgbCam[row * 4 + 2], b)),
                         P.rgbCam[row * 4 + 3]);
        px[row] = clamp_trunc_u16(val);
    }
}

// One pixel from global memory, wherever it lies.
__device__ void demosaic_border(const unsigned short* __restrict__ cfa, int x, int y, int w, int h,
                                const DemosaicParams& P, unsigned short* __restrict__ out)
{
    float s[3][3], rgb[3];
    for (int dy = 0; dy < 3; ++dy)
        for (int dx = 0; dx < 3; ++dx)
        {
            const int gx = x + dx - 1, gy = y + dy - 1;
            s[dy][dx] = gx >= 0 && gy >= 0 && gx < w && gy < h
                            ? demosaic_level(cfa[(size_t)gy * w + gx], P.camMul[bayer_color(gy, gx, P.filters)], P)
                            : 0.0f;
        }
    demosaic_generic<3>(s, 0, 0, x, y, w, h, P.filters, rgb);
    demosaic_matrix(P, rgb[0], rgb[1], rgb[2], out + ((size_t)y * w + x) * 3);
}

// Any filter word, size and alignment, and small frames: a thread per 2x2
// quad, a tile of the levelled values in shared memory.
__global__ void __launch_bounds__(256) k_demosaic(const unsigned short* __restrict__ cfa, int w, int h,
                                                  DemosaicParams P, unsigned short* __restrict__ out)
{
    __shared__ float s[kDmTH + 2][kDmTW + 2];
    const int tx0 = blockIdx.x * kDmTW, ty0 = blockIdx.y * kDmTH;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    auto level_m = [&](unsigned raw, float mul) { return demosaic_level(raw, mul, P); };
    auto level = [&](unsigned short raw, int gy, int gx) {
        return level_m(raw, P.camMul[bayer_color(gy, gx, P.filters)]);
    };
    if ((w & 3) == 0 && (reinterpret_cast<uintptr_t>(cfa) & 7) == 0 && tx0 >= 4 && tx0 + kDmTW + 4 <= w)
    {
        // Interior column of tiles on 8-byte aligned rows: the footprint
        // (columns tx0-1 .. tx0+64) read as 8-byte words of four values,
        // columns tx0-4 .. tx0+67.
        constexpr int kWords = kDmTW / 4 + 2;
        for (int i = tid; i < (kDmTH + 2) * kWords; i += 256)
        {
            const int r = i / kWords, wi = i - r * kWords;
            const int gy = ty0 - 1 + r, gx0 = tx0 - 4 + 4 * wi;
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (gy >= 0 && gy < h)
            {
                // gx0 is even: the four values alternate between two colours
                // (a site's colour depends on its column only through x & 1)
                const float me = P.camMul[bayer_color(gy, gx0, P.filters)];
                const float mo = P.camMul[bayer_color(gy, gx0 + 1, P.filters)];
                const uint2 q = __ldg(reinterpret_cast<const uint2*>(cfa + (size_t)gy * w + gx0));
                v[0] = level_m(q.x & 0xffffu, me);
                v[1] = level_m(q.x >> 16, mo);
                v[2] = level_m(q.y & 0xffffu, me);
                v[3] = level_m(q.y >> 16, mo);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                const int c = gx0 + k - (tx0 - 1);
                if (c >= 0 && c < kDmTW + 2) s[r][c] = v[k];
            }
        }
    }
    else
    {
        for (int i = tid; i < (kDmTH + 2) * (kDmTW + 2); i += 256)
        {
            int r = i / (kDmTW + 2), c = i % (kDmTW + 2);
            int gx = tx0 - 1 + c, gy = ty0 - 1 + r;
            float v = 0.0f;
            if (gx >= 0 && gy >= 0 && gx < w && gy < h) v = level(__ldg(cfa + (size_t)gy * w + gx), gy, gx);
            s[r][c] = v;
        }
    }
    __syncthreads();
    const bool evenW = (w & 1) == 0;
    // Every pixel of the block is an interior pixel (1 <= x <= w-2, 1 <= y <= h-2).
    const bool blockInterior = tx0 >= 1 && ty0 >= 1 && tx0 + kDmTW <= w - 1 && ty0 + kDmTH <= h - 1;
    // The quad's 4x4 neighbourhood, read once.
    float nb[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) nb[r][c] = s[threadIdx.y * 2 + r][threadIdx.x * 2 + c];
#pragma unroll
    for (int oy = 0; oy < 2; ++oy)
    {
        unsigned short px[2][3];
        const int ly = threadIdx.y * 2 + oy, y = ty0 + ly;
#pragma unroll
        for (int ox = 0; ox < 2; ++ox)
        {
            const int lx = threadIdx.x * 2 + ox, x = tx0 + lx;
            float R = 0.0f, G = 0.0f, B = 0.0f;
            if (P.std2x2 && (blockInterior || (x >= 1 && y >= 1 && x < w - 1 && y < h - 1)))
            {
                // Interior of a standard Bayer layout: the same-colour
                // neighbours are the cross (4), the diagonals (4), or a
                // horizontal / vertical pair (2 each); dividing by 4 or 2 is
                // exact, so these are the reference's averages bit for bit.
                // quad-local neighbourhood: centre at nb[oy + 1][ox + 1]
                const float c = nb[oy + 1][ox + 1];
                const float n = nb[oy][ox + 1], so = nb[oy + 2][ox + 1];
                const float we = nb[oy + 1][ox], ea = nb[oy + 1][ox + 2];
                // tx0, ty0 and the quad's corner are even: y & 1 = oy, x & 1 = ox
                const int cls = P.color2x2[(oy << 1) | ox];
                if (cls != 1)
                {
                    const float cross = ((n + we) + ea) + so;
                    const float diag = ((nb[oy][ox] + nb[oy][ox + 2]) + nb[oy + 2][ox]) + nb[oy + 2][ox + 2];
                    G = fmul(cross, 0.25f);
                    const float other = fmul(diag, 0.25f);
                    R = cls == 0 ? c : other;
                    B = cls == 0 ? other : c;
                }
                else
                {
                    const int hc = P.color2x2[(oy << 1) | (ox ^ 1)];  // colour of the left/right pair
                    const float hp = fmul(we + ea, 0.5f), vp = fmul(n + so, 0.5f);
                    G = c;
                    R = hc == 0 ? hp : vp;
                    B = hc == 0 ? vp : hp;
                }
            }
            else if (x < w && y < h)
            {
                float rgb[3];
                demosaic_generic(s, lx, ly, x, y, w, h, P.filters, rgb);
                R = rgb[0];
                G = rgb[1];
                B = rgb[2];
            }
            demosaic_matrix(P, R, G, B, px[ox]);
        }
        const int x0 = tx0 + threadIdx.x * 2;
        if (y >= h || x0 >= w) continue;
        unsigned short* o = out + ((size_t)y * w + x0) * 3;
        if (evenW && x0 + 1 < w)
        {
            // x0 even and w even: 12 bytes at a 4-byte-aligned address.
            uint32_t* o32 = reinterpret_cast<uint32_t*>(o);
            o32[0] = (uint32_t)px[0][0] | ((uint32_t)px[0][1] << 16);
            o32[1] = (uint32_t)px[0][2] | ((uint32_t)px[1][0] << 16);
            o32[2] = (uint32_t)px[1][1] | ((uint32_t)px[1][2] << 16);
        }
        else
        {
            o[0] = px[0][0];
            o[1] = px[0][1];
            o[2] = px[0][2];
            if (x0 + 1 < w)
            {
                o[3] = px[1][0];
                o[4] = px[1][1];
                o[5] = px[1][2];
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Demosaic of a standard Bayer layout, for frames of whole 4-pixel words and
// multipliers in the range that needs no lower clamp (launch_demosaic).  A
// thread makes 4 columns of two strips of rows, kDmRows apart, and marches
// down both: every value is a pair (upper strip, lower strip) of the same
// colour, so all arithmetic is paired and nothing is repacked.  The columns
// beside its own come from the neighbouring lanes, so 30 of a warp's 32 lanes
// write.  Averages are of integers below 2^18, exact in any order; kept as
// 2^23 + floor, they enter the colour matrix in one rounding each (common.cuh).
// The frame's outermost pixels, which average fewer neighbours, are left to
// the blocks after the strips' (one thread each).
// Bound by instruction issue: 24 MP 55 us (192 MB, 29 us at the measured
// copy rate); a thread per 2x2 quad from a tile in shared memory, with scalar
// arithmetic, took 117 us.
// ---------------------------------------------------------------------------
constexpr int kDmRows = 12, kDmCols = 120, kDmWarps = 4;
constexpr int kDmStripPixels = 4800;  // pixels per SM from which strips are taken

struct BayerParams
{
    f32x2 mul[2][2];                     // of site (y & 1, x & 1)
    f32x2 w[3][3], bias[3][3], add[3];   // matrix, -2^23 times it, its last column
    f32x2 negBlack;                      // -(2^23 + black)
    uint32_t black2;
};

template <int G0, int X0>
__device__ __forceinline__ void demosaic_row(const BayerParams& B, const f32x2 (&up)[6], const f32x2 (&cur)[6],
                                             const f32x2 (&dn)[6], f32x2 nz, int parity, uint32_t (&oa)[6],
                                             uint32_t (&ob)[6])
{
    const int gcol = parity ? 1 - G0 : G0;     // column parity of G in this row
    const int cx = parity ? 2 - X0 : X0;       // colour of the row's other sites
    const f32x2 big = dup2(8388608.0f);
    f32x2 v[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) v[i] = add2(up[i], dn[i]);
    uint32_t bits[2][12];
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
        const f32x2 hsum = add2(cur[i], cur[i + 2]);
        // channels as 2^23 + value, but the site's own as the value
        f32x2 ch[3];
        int own;
        if ((i & 1) == gcol)
        {
            own = 1;
            ch[cx] = fma2_rz(hsum, dup2(0.5f), big);
            ch[2 - cx] = fma2_rz(v[i + 1], dup2(0.5f), big);
        }
        else
        {
            own = cx;
            ch[1] = fma2_rz(add2(v[i + 1], hsum), dup2(0.25f), big);
            ch[2 - cx] = fma2_rz(add2(v[i], v[i + 2]), dup2(0.25f), big);
        }
        ch[own] = cur[i + 1];
#pragma unroll
        for (int r = 0; r < 3; ++r)
        {
            f32x2 p[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) p[c] = fma2(B.w[r][c], ch[c], c == own ? nz : B.bias[r][c]);
            const f32x2 s = add2(add2(add2(p[0], p[1]), p[2]), B.add[r]);
            const f32x2 q = add2_rz(pack2(clamp_u16f(lo2(s)), clamp_u16f(hi2(s))), big);
            bits[0][i * 3 + r] = __float_as_uint(lo2(q));
            bits[1][i * 3 + r] = __float_as_uint(hi2(q));
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k)
    {
        oa[k] = __byte_perm(bits[0][2 * k], bits[0][2 * k + 1], 0x5410);
        ob[k] = __byte_perm(bits[1][2 * k], bits[1][2 * k + 1], 0x5410);
    }
}

template <int G0, int X0>
__global__ void __launch_bounds__(32 * kDmWarps, 5) k_demosaic_bayer(const unsigned short* __restrict__ cfa, int w, int h,
                                                                  const __grid_constant__ BayerParams B,
                                                                  const __grid_constant__ DemosaicParams P,
                                                                  unsigned short* __restrict__ out, int strips,
                                                                  int tilesX)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if ((int)blockIdx.x >= strips)
    {
        // the frame's outermost pixels
        const int i = (blockIdx.x - strips) * blockDim.x + threadIdx.x;
        int x, y;
        if (i < w) x = i, y = 0;
        else if (i < 2 * w) x = i - w, y = h - 1;
        else if (i < 2 * w + h) x = 0, y = i - 2 * w;
        else x = w - 1, y = i - 2 * w - h;
        if (y >= h || (i >= 2 * w && (y == 0 || y == h - 1))) return;
        demosaic_border(cfa, x, y, w, h, P, out);
        return;
    }
    const int item = blockIdx.x * kDmWarps + warp;
    const int x = item % tilesX * kDmCols - 4 + 4 * lane, y0 = item / tilesX * (2 * kDmRows);
    if (y0 >= h) return;
    const f32x2 nz = neg_zero2(), big = dup2(8388608.0f), nbig = dup2(-8388608.0f);
    const bool inX = x >= 0 && x < w;
    const unsigned short* src = cfa + (inX ? x : 0);
    struct Raw
    {
        uint2 a, b;
    };
    auto load = [&](int r) {
        const int ya = min(max(y0 + r, 0), h - 1), yb = min(y0 + kDmRows + r, h - 1);
        return Raw{__ldg(reinterpret_cast<const uint2*>(src + (size_t)ya * w)),
                   __ldg(reinterpret_cast<const uint2*>(src + (size_t)yb * w))};
    };
    // Black level, white balance and truncation of the thread's columns of a
    // row, and of the one on either side.
    auto level = [&](Raw q, int parity, f32x2 (&o)[6]) {
        const uint32_t a[2] = {__vmaxu2(q.a.x, B.black2), __vmaxu2(q.a.y, B.black2)};
        const uint32_t b[2] = {__vmaxu2(q.b.x, B.black2), __vmaxu2(q.b.y, B.black2)};
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const uint32_t sel = i & 1 ? 0x7632 : 0x7610;
            f32x2 v = pack2(__uint_as_float(__byte_perm(a[i >> 1], 0x4B000000u, sel)),
                            __uint_as_float(__byte_perm(b[i >> 1], 0x4B000000u, sel)));
            v = mulx2(add2(v, B.negBlack), B.mul[parity][i & 1], nz);
            v = pack2(fminf(lo2(v), 65535.0f), fminf(hi2(v), 65535.0f));
            o[i + 1] = add2(add2_rz(v, big), nbig);
        }
        o[0] = pack2(__shfl_up_sync(0xffffffffu, lo2(o[4]), 1), __shfl_up_sync(0xffffffffu, hi2(o[4]), 1));
        o[5] = pack2(__shfl_down_sync(0xffffffffu, lo2(o[1]), 1), __shfl_down_sync(0xffffffffu, hi2(o[1]), 1));
    };
    const bool writes = inX && lane >= 1 && lane <= 30;
    const bool whole = x > 0 && x + 4 < w;
    auto store = [&](int y, const uint32_t (&o)[6]) {
        if (!writes || y < 1 || y >= h - 1) return;
        unsigned short* p = out + ((size_t)y * w + x) * 3;
        if (whole)
        {
            uint2* p2 = reinterpret_cast<uint2*>(p);
            p2[0] = make_uint2(o[0], o[1]);
            p2[1] = make_uint2(o[2], o[3]);
            p2[2] = make_uint2(o[4], o[5]);
        }
        else
        {
#pragma unroll
            for (int k = 0; k < 12; ++k)
                if (x + k / 3 > 0 && x + k / 3 < w - 1) p[k] = (unsigned short)(o[k >> 1] >> (k & 1 ? 16 : 0));
        }
    };
    f32x2 row[3][6];  // rows r - 1, r, r + 1 at (r + 2) % 3, r % 3, (r + 1) % 3
    level(load(-1), 1, row[2]);
    level(load(0), 0, row[0]);
    Raw next = load(1);
#pragma unroll 1
    for (int base = 0; base < kDmRows; base += 6)
    {
#pragma unroll
        for (int k = 0; k < 6; ++k)
        {
            const int r = base + k;
            const Raw q = next;
            next = load(r + 2);
            level(q, (k + 1) & 1, row[(k + 1) % 3]);
            uint32_t oa[6], ob[6];
            demosaic_row<G0, X0>(B, row[(k + 2) % 3], row[k % 3], row[(k + 1) % 3], nz, k & 1, oa, ob);
            store(y0 + r, oa);
            store(y0 + kDmRows + r, ob);
        }
    }
}

// ---------------------------------------------------------------------------
// Warp: backward bilinear homography warp (WarpPerspective_Scalar.cpp:8-45,
// WarpPerspectiveKernels.h:16-43), with RenderExecutor's ApplyGain fused.
// A warp makes 64 consecutive pixels of a row, lane l the pixels l and l + 32
// (consecutive lanes gather neighbouring taps, and the two pixels' arithmetic
// is paired).  Bound by instruction issue and tap latency.  A 2048 x 2048 tile,
// all of it covered: 24.5 us with the frame in L2, 29.5 from HBM, where fewer
// threads hide the longer taps; a pixel per lane with scalar arithmetic and
// 2-byte taps (k_warp_small) 29.1 and 30.2.
// ---------------------------------------------------------------------------
constexpr int kWarpPairPixels = 1700;  // destination pixels per SM from which a lane makes two

struct WarpParams
{
    float H[9];
    float gain;
    int applyGain;
};

// Small tiles: a pixel per lane, so that twice the threads share the latency
// of the taps.
__global__ void __launch_bounds__(256) k_warp_small(const unsigned short* __restrict__ src, int sw, int sh,
                                                    unsigned short* __restrict__ dst, int dw, int dh, int offX,
                                                    int offY, WarpParams P)
{
    const int x = blockIdx.x * 32 + threadIdx.x, y = blockIdx.y * 8 + threadIdx.y;
    if (x >= dw || y >= dh) return;
    const float dX = (float)(x + offX), dY = (float)(y + offY);
    float sx = fadd(fadd(fmul(P.H[0], dX), fmul(P.H[1], dY)), P.H[2]);
    float sy = fadd(fadd(fmul(P.H[3], dX), fmul(P.H[4], dY)), P.H[5]);
    const float sw1 = fadd(fadd(fmul(P.H[6], dX), fmul(P.H[7], dY)), P.H[8]);
    unsigned short o[3] = {0, 0, 0};
    sx = fdiv(sx, sw1);
    sy = fdiv(sy, sw1);
    // (NaN and positions out of range are invalid, as in warp_pair23)
    if (!(fabsf(sw1) < 1e-10f) && sx >= 0.0f && sx < (float)(sw - 1) && sy >= 0.0f && sy < (float)(sh - 1))
    {
        const int x0 = (int)f2u_floor(sx), y0 = (int)f2u_floor(sy);
        const float fx = fsub(sx, u2f((uint32_t)x0)), fy = fsub(sy, u2f((uint32_t)y0));
        const float gx = fsub(1.0f, fx), gy = fsub(1.0f, fy);
        const float w00 = fmul(gx, gy), w10 = fmul(fx, gy), w01 = fmul(gx, fy), w11 = fmul(fx, fy);
        const unsigned short* r0 = src + ((size_t)y0 * sw + x0) * 3;
        const unsigned short* r1 = r0 + (size_t)sw * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
            const float v = fadd(fadd(fadd(fmul(w00, u2f(__ldg(r0 + c))), fmul(w10, u2f(__ldg(r0 + 3 + c)))),
                                      fmul(w01, u2f(__ldg(r1 + c)))),
                                 fmul(w11, u2f(__ldg(r1 + 3 + c))));
            o[c] = P.applyGain ? clamp_trunc_u16(fmul(clamp_floor_u16f(v), P.gain)) : clamp_trunc_u16(v);
        }
    }
    unsigned short* d = dst + ((size_t)y * dw + x) * 3;
    d[0] = o[0];
    d[1] = o[1];
    d[2] = o[2];
}

template <bool AFFINE>
__global__ void __launch_bounds__(256) k_warp(WarpSource src, unsigned short* __restrict__ dst, int dw, int dh,
                                              int offX, int offY, WarpParams P)
{
    const int y = blockIdx.y * 8 + threadIdx.y;
    const int xa = blockIdx.x * 64 + threadIdx.x, xb = xa + 32;
    if (y >= dh || xa >= dw) return;
    const float dY = (float)(y + offY);
    const float hy[3] = {fmul(P.H[1], dY), fmul(P.H[4], dY), fmul(P.H[7], dY)};
    f32x2 v[3];
    warp_pair23<AFFINE>(src, P.H, hy, (float)(xa + offX), (float)(xb + offX), true, xb < dw, v);
    unsigned short* d = dst + ((size_t)y * dw + xa) * 3;
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
        if (P.applyGain) v[c] = gain_pair23(v[c], P.gain);
        d[c] = (unsigned short)__float_as_uint(lo2(v[c]));
        if (xb < dw) d[96 + c] = (unsigned short)__float_as_uint(hi2(v[c]));
    }
}

// ---------------------------------------------------------------------------
// Median stack (MedianStackKernels.h:19-55, MedianStack_Scalar.cpp:8-24).
//
// Two output scalars per thread, packed as the low and high halves of one
// 32-bit word per input.  Per scalar the statistics are accumulated
// sequentially in input order in FP32 (sumSq exceeds 2^24, so the order is
// part of the result), exactly as the reference.  A value is kept when it
// lies between the sigma bounds; values are integers, so the bounds become
// integers (ceil and floor) and both halves are tested at once with
// __vmaxu2/__vminu2.  A clipped value, and every slot past the input count,
// becomes 0xFFFF: the maximum of the type, so the first keptCount sorted
// positions hold exactly the sorted kept values (ties with a kept 65535 do
// not change any value there), and the median is element keptCount/2 - the
// reference's values[count / 2].  The sort is Batcher's odd-even merge
// network (Batcher 1968) for N values on the same packed min/max, cut off at
// N wires (the wires above would hold the maximum and never move), and only
// elements 0 .. N/2 are read, so the last stages' unread halves drop out of
// the code: 26 comparators for 9 inputs and 63 for 16, where a bitonic
// network of the next power of two has 80 for either.  Bound by the integer
// pipe (min, max and logic issue at half rate): 72 % busy.  9 inputs of 3001 x
// 2003: 146 us; one scalar per thread and an unpruned network, which odd
// counts took before, 469 us.
// ---------------------------------------------------------------------------
struct MedianInputs
{
    const unsigned short* p[kMaxContributors];
};

// The stack sizes with a network of their own; a stack in between is padded
// to the next.  Every size up to 10, where a value adds 2-5 comparators (a
// tenth to a fifth of the kernel), coarser above.
#define I360B_STACK_SIZES(X) \
    X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(12) X(14) X(16) X(20) X(24) X(28) X(32)
// The fewest inputs that take network N: inputs below it need no count test.
__host__ __device__ constexpr int stack_floor(int N) { return N <= 2 ? 1 : N <= 10 ? N : N <= 16 ? N - 1 : N - 3; }

template <int N>
__device__ __forceinline__ void merge_sort_u16x2(uint32_t (&v)[N])
{
#pragma unroll
    for (int p = 1; p < N; p <<= 1)
#pragma unroll
        for (int k = p; k > 0; k >>= 1)
#pragma unroll
            for (int i = 0; i < N; ++i)
            {
                const int j0 = k % p;
                if (i >= j0 && ((i - j0) / k) % 2 == 0 && i + k < N && i / (2 * p) == (i + k) / (2 * p))
                {
                    const uint32_t lo = __vminu2(v[i], v[i + k]), hi = __vmaxu2(v[i], v[i + k]);
                    v[i] = lo;
                    v[i + k] = hi;
                }
            }
}

// Running statistics of a packed pair of scalars, added as 2^23 + value.
struct PairSums
{
    f32x2 s, q;
    __device__ __forceinline__ void clear() { s = q = dup2(0.0f); }
    __device__ __forceinline__ void add23(f32x2 t, f32x2 nz)
    {
        const f32x2 m23 = dup2(-8388608.0f);
        const f32x2 a = add2(t, m23);
        s = add2(s, a);
        q = add2(q, fma2(a, t, mulx2(a, m23, nz)));  // a t - 2^23 a = a a, rounded once
    }
};

// a / n for a whole n of 2..32 (fn = n, inv = RN(1/n)): Markstein's division
// with one correction (P. Markstein, "Computation of elementary functions on
// the IBM RISC System/6000 processor", 1990).  With q0 = RN(a inv), at most 2
// ulp off, a - n q0 is a multiple of q0's ulp below 64 of them, so the first
// fma is exact; the second rounds a / n plus an error below 2^-22 ulp, and
// a / n is either a rounding midpoint - only for n a power of two, where inv
// and all of this is exact - or at least 1/64 ulp away from one.
__device__ __forceinline__ float div_count(float a, float fn, float inv)
{
    const float q = fmul(a, inv);
    return __fmaf_rn(__fmaf_rn(-fn, q, a), inv, q);
}

// Sigma bounds of one scalar's stack (MedianStackKernels.h:22-27) as the low
// 16 bits of lo, hi: the whole numbers that pass lo <= value <= hi; every
// number when none would pass (an empty range, or a bound that is not a
// number), as the reference then keeps every value.
__device__ __forceinline__ void clip_range(float sum, float sumSq, float fn, float inv, float sigma, uint32_t& lo,
                                           uint32_t& hi)
{
    const float mean = div_count(sum, fn, inv);
    const float var = fsub(div_count(sumSq, fn, inv), fmul(mean, mean));
    const float sd = __fsqrt_rn(var < 0.0f ? 0.0f : var);
    const float fl = fsub(mean, fmul(sigma, sd)), fh = fadd(mean, fmul(sigma, sd));
    // on [0, 65535] a sum with 2^23 rounded up / down is 2^23 + ceil / floor
    const uint32_t l = __float_as_uint(__fadd_ru(fmaxf(fl, 0.0f), 8388608.0f));
    const uint32_t h = __float_as_uint(__fadd_rd(fminf(fh, 65535.0f), 8388608.0f));
    const bool some = fl <= 65535.0f && fh >= 0.0f && l <= h;
    lo = some ? l : 0u;
    hi = some ? h : 0xffffu;
}

// The sigma-clipped median of both halves of v[0..n), n <= N (v[i] for
// i >= n must be 0xFFFFFFFF), packed the same way, from the stack's sums.
// v is sorted in place; reload(v) restores it.
template <int N, typename Reload>
__device__ __forceinline__ uint32_t median_pair(uint32_t (&v)[N], int n, float inv, float sigma, const PairSums& S,
                                                Reload reload)
{
    int cntL = n, cntH = n;
    if (N > 3 && n > 3)
    {
        const float fn = (float)n;
        uint32_t loL, hiL, loH, hiH;
        clip_range(lo2(S.s), lo2(S.q), fn, inv, sigma, loL, hiL);
        clip_range(hi2(S.s), hi2(S.q), fn, inv, sigma, loH, hiH);
        uint32_t lw = __byte_perm(loL, loH, 0x5410), hw = __byte_perm(hiL, hiH, 0x5410);
#pragma unroll 1
        for (;;)
        {
            uint32_t out = 0;  // clipped values per half
#pragma unroll
            for (int i = 0; i < N; ++i)
            {
                // 1 in a half whose value lies outside its bounds
                const uint32_t z = __vminu2(__vminu2(__vmaxu2(v[i], lw), hw) ^ v[i], 0x00010001u);
                out += z;
                v[i] |= z * 0xffffu;
            }
            // the padding slots counted as clipped where the bound is below 0xFFFF
            out -= (uint32_t)(N - n) * __vminu2(~hw, 0x00010001u);
            cntL = n - (int)(out & 0xffffu);
            cntH = n - (int)(out >> 16);
            if (cntL > 0 && cntH > 0) break;
            // nothing kept: the reference keeps every value
            if (cntL == 0) lw &= 0xffff0000u, hw |= 0x0000ffffu;
            if (cntH == 0) lw &= 0x0000ffffu, hw |= 0xffff0000u;
            reload(v);
        }
    }
    merge_sort_u16x2<N>(v);
    const int mL = cntL >> 1, mH = cntH >> 1;  // <= N / 2
    uint32_t rL = v[0], rH = v[0];
#pragma unroll
    for (int i = 1; i <= N / 2 && i < N; ++i)
    {
        rL = (i == mL) ? v[i] : rL;
        rH = (i == mH) ? v[i] : rH;
    }
    return __byte_perm(rL, rH, 0x7610);
}

// Scalars 2t and 2t+1 of every input; the last scalar of an odd count by
// itself.  WORDS: every input and the output are 4-byte aligned, so a pair is
// one word; else two 2-byte accesses.
template <int N, bool WORDS>
__global__ void __launch_bounds__(256) k_median(const __grid_constant__ MedianInputs in, int n, float inv,
                                                long long total, float sigma, unsigned short* __restrict__ out)
{
    const long long e = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 2;
    if (e >= total) return;
    const bool two = e + 1 < total;
    auto load = [&](uint32_t (&v)[N]) {
        if (WORDS && two)
        {
#pragma unroll
            for (int i = 0; i < N; ++i)
                v[i] = (i < stack_floor(N) || i < n) ? __ldg(reinterpret_cast<const uint32_t*>(in.p[i] + e))
                                                     : 0xffffffffu;
        }
        else
        {
#pragma unroll
            for (int i = 0; i < N; ++i)
                v[i] = (i < stack_floor(N) || i < n)
                           ? (uint32_t)__ldg(in.p[i] + e) | (two ? (uint32_t)__ldg(in.p[i] + e + 1) << 16 : 0u)
                           : 0xffffffffu;
        }
    };
    uint32_t v[N];
    load(v);
    PairSums S;
    S.clear();
    if (N > 3)
    {
        const f32x2 nz = neg_zero2();
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i < stack_floor(N) || i < n) S.add23(pack2(u16lo23(v[i]), u16hi23(v[i])), nz);
    }
    const uint32_t m = median_pair<N>(v, n, inv, sigma, S, load);
    if (WORDS && two)
        *reinterpret_cast<uint32_t*>(out + e) = m;
    else
    {
        out[e] = (unsigned short)(m & 0xffffu);
        if (two) out[e + 1] = (unsigned short)(m >> 16);
    }
}

// ---------------------------------------------------------------------------
// Warp + median stack fused: the median of n frames each warped onto the
// same destination grid (IComputeBackend::WarpPerspective of every frame,
// then MedianStack over the warped buffers: CpuComputeBackend.cpp:112-159).
// Each destination pixel's n samples are computed with the warp's exact FP32
// arithmetic, so the warped frames are never written.  A thread makes the
// pixels l and l + 32 of its warp's 64-pixel row segment and stacks their
// channels as three packed pairs.  Bound by instruction issue.  The frames
// are walked by a rolled loop that leaves the packed samples in shared memory
// (12 n bytes per thread) and the running sums in registers, and the channels
// are then sorted one after another by one rolled loop: the unrolled form
// held 48 samples in registers and its code did not fit the instruction cache.
// 16 frames of 4000 x 3000: 1.90 ms unrolled with scalar arithmetic and 2-byte
// taps, 1.23 ms rolled with the taps as words, 1.14 ms with the paired
// arithmetic (6155 -> 4783 instructions per warp; issue 69 % busy, the rest
// waiting for taps).  Two frames in flight, 64 threads or 10 blocks per SM
// were no faster.
// ---------------------------------------------------------------------------
constexpr int kWmThreads = 128;

struct StackParams
{
    const unsigned short* src[kMaxContributors];
    float H[kMaxContributors][9];
    uint32_t affine;  // bit i: frame i's homography has the third row (0, 0, 1)
};

template <int N>
__global__ void __launch_bounds__(kWmThreads) k_warp_median(const __grid_constant__ StackParams S, int n, float inv,
                                                            int sw, int sh, unsigned short* __restrict__ dst, int dw,
                                                            int dh, int offX, int offY, float sigma)
{
    extern __shared__ uint32_t stack[];  // [frame][channel][thread]
    const int tilesX = (dw + 63) / 64;   // blocks in row order (a linear grid holds any number of rows)
    const int by = blockIdx.x / tilesX, bx = blockIdx.x - by * tilesX;
    const int y = by * (kWmThreads / 32) + threadIdx.y;
    const int tid = threadIdx.y * 32 + threadIdx.x;
    const int xa = bx * 64 + threadIdx.x, xb = xa + 32;
    if (y >= dh || xa >= dw) return;  // no barrier below: a thread reads only what it wrote
    const float dY = (float)(y + offY), dXa = (float)(xa + offX), dXb = (float)(xb + offX);
    const f32x2 nz = neg_zero2();
    PairSums sums[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) sums[c].clear();
#pragma unroll 1
    for (int i = 0; i < n; ++i)
    {
        const float* H = S.H[i];
        const WarpSource src = warp_source(S.src[i], sw, sh);
        const float hy[3] = {fmul(H[1], dY), fmul(H[4], dY), fmul(H[7], dY)};
        f32x2 v[3];
        if ((S.affine >> i) & 1u) warp_pair23<true>(src, H, hy, dXa, dXb, true, xb < dw, v);
        else warp_pair23<false>(src, H, hy, dXa, dXb, true, xb < dw, v);
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
            stack[(i * 3 + c) * kWmThreads + tid] =
                __byte_perm(__float_as_uint(lo2(v[c])), __float_as_uint(hi2(v[c])), 0x5410);
            sums[c].add23(v[c], nz);
        }
    }
    unsigned short* oa = dst + ((size_t)y * dw + xa) * 3;
#pragma unroll 1
    for (int c = 0; c < 3; ++c)
    {
        auto load = [&](uint32_t (&v)[N]) {
#pragma unroll
            for (int i = 0; i < N; ++i)
                v[i] = (i < stack_floor(N) || i < n) ? stack[(i * 3 + c) * kWmThreads + tid] : 0xffffffffu;
        };
        uint32_t v[N];
        load(v);
        const PairSums sc = c == 0 ? sums[0] : c == 1 ? sums[1] : sums[2];
        const uint32_t m = median_pair<N>(v, n, inv, sigma, sc, load);
        oa[c] = (unsigned short)(m & 0xffffu);
        if (xb < dw) oa[96 + c] = (unsigned short)(m >> 16);
    }
}

// ---------------------------------------------------------------------------
// Gain (GainColorOps.cpp:16-26), 8 values per thread with 16-byte accesses.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_gain(unsigned short* __restrict__ d, long long n, float gain)
{
    long long i8 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (i8 >= n) return;
    if (i8 + 8 <= n && ((reinterpret_cast<uintptr_t>(d + i8) & 15) == 0))
    {
        uint4 q = *reinterpret_cast<uint4*>(d + i8);
        unsigned short* s = reinterpret_cast<unsigned short*>(&q);
#pragma unroll
        for (int k = 0; k < 8; ++k) s[k] = clamp_trunc_u16(fmul(u2f(s[k]), gain));
        *reinterpret_cast<uint4*>(d + i8) = q;
    }
    else
    {
        for (long long i = i8; i < n && i < i8 + 8; ++i) d[i] = clamp_trunc_u16(fmul(u2f(d[i]), gain));
    }
}
}  // namespace

int launch_demosaic(const unsigned short* cfa, int w, int h, unsigned short black, const float* camMul,
                    const float* rgbCam, uint32_t filters, unsigned short* out, cudaStream_t s)
{
    DemosaicParams P;
    for (int i = 0; i < 4; ++i) P.camMul[i] = camMul[i];
    for (int i = 0; i < 12; ++i) P.rgbCam[i] = rgbCam[i];
    P.filters = filters;
    P.black = black;
    // Standard Bayer layout test on the filter word (rows repeat with period
    // 2; one R, one B, G/G2 on a diagonal).
    {
        auto col = [&](int r, int c) { return (int)((filters >> ((((r << 1) & 14) | (c & 1)) << 1)) & 3u); };
        bool periodic = true;
        for (int r = 2; r < 8; ++r)
            for (int c = 0; c < 2; ++c) periodic = periodic && col(r, c) == col(r & 1, c);
        int c00 = col(0, 0), c01 = col(0, 1), c10 = col(1, 0), c11 = col(1, 1);
        auto isG = [](int v) { return v == 1 || v == 3; };
        bool diagG = (isG(c00) && isG(c11) && ((c01 == 0 && c10 == 2) || (c01 == 2 && c10 == 0))) ||
                     (isG(c01) && isG(c10) && ((c00 == 0 && c11 == 2) || (c00 == 2 && c11 == 0)));
        P.std2x2 = (periodic && diagG) ? 1 : 0;
        P.color2x2[0] = isG(c00) ? 1 : c00;
        P.color2x2[1] = isG(c01) ? 1 : c01;
        P.color2x2[2] = isG(c10) ? 1 : c10;
        P.color2x2[3] = isG(c11) ? 1 : c11;
    }
    // k_demosaic_bayer: a standard layout, rows of whole 8-byte words in and
    // out, multipliers that level to no negative or NaN and a matrix whose
    // products stay finite, and a frame large enough: a strip's 24 rows are a
    // chain of 8.2 us however few strips there are.  500 x 400 takes 5.5 us in
    // tiles and 8.2 in strips, 800 x 600 6.8 and 8.4, 1000 x 700 7.8 and 8.3,
    // 900 x 800 8.7 and 8.4, 1200 x 900 10.0 and 8.5.
    const bool large = (long long)w * h >= (long long)kDmStripPixels * sm_count();
    auto in_range = [](float v, float lo) { return v >= lo && v <= 1e30f; };
    bool fast = large && P.std2x2 && w % 4 == 0 && ((reinterpret_cast<uintptr_t>(cfa) | reinterpret_cast<uintptr_t>(out)) & 7) == 0;
    for (float m : P.camMul) fast = fast && in_range(m, 0.0f);
    for (float m : P.rgbCam) fast = fast && in_range(m, -1e30f);
    if (fast)
    {
        BayerParams B;
        for (int r = 0; r < 2; ++r)
            for (int c = 0; c < 2; ++c) B.mul[r][c] = pair_of(P.camMul[bayer_color(r, c, filters)]);
        for (int r = 0; r < 3; ++r)
        {
            for (int c = 0; c < 3; ++c)
            {
                B.w[r][c] = pair_of(rgbCam[r * 4 + c]);
                B.bias[r][c] = pair_of(-8388608.0f * rgbCam[r * 4 + c]);
            }
            B.add[r] = pair_of(rgbCam[r * 4 + 3]);
        }
        B.negBlack = pair_of(-(8388608.0f + (float)black));
        B.black2 = (uint32_t)black << 16 | black;
        const int tilesX = (w + kDmCols - 1) / kDmCols, tilesY = (h + 2 * kDmRows - 1) / (2 * kDmRows);
        const int strips = (tilesX * tilesY + kDmWarps - 1) / kDmWarps;
        const int threads = 32 * kDmWarps, border = (2 * w + 2 * h + threads - 1) / threads;
        // G in column 0 or 1 of row 0, whose other sites are red or blue
        const bool g0 = P.color2x2[0] != 1;
        auto* k = g0 ? (P.color2x2[0] == 0 ? k_demosaic_bayer<1, 0> : k_demosaic_bayer<1, 2>)
                     : (P.color2x2[1] == 0 ? k_demosaic_bayer<0, 0> : k_demosaic_bayer<0, 2>);
        k<<<strips + border, threads, 0, s>>>(cfa, w, h, B, P, out, strips, tilesX);
        return check_launch("demosaic kernel");
    }
    dim3 grid((w + kDmTW - 1) / kDmTW, (h + kDmTH - 1) / kDmTH);
    k_demosaic<<<grid, dim3(32, 8), 0, s>>>(cfa, w, h, P, out);
    return check_launch("demosaic kernel");
}

int launch_warp(const unsigned short* src, int sw, int sh, unsigned short* dst, int dw, int dh, const float* H,
                int offX, int offY, float gain, cudaStream_t s)
{
    WarpParams P;
    for (int i = 0; i < 9; ++i) P.H[i] = H[i];
    P.gain = gain;
    P.applyGain = gain_is_identity(gain) ? 0 : 1;
    const dim3 block(32, 8);
    // A pixel per lane while the tile has too few for two to fill the SMs:
    // 128 x 128 1.9 us against 2.5 for pairs, 256 x 256 2.1 and 2.5, 400 x 400
    // 2.7 and 2.8, 480 x 480 3.0 and 3.1; 512 x 512 3.2 for either, 1000 x 1000
    // 7.0 and 6.2.
    if ((long long)dw * dh < (long long)kWarpPairPixels * sm_count())
    {
        k_warp_small<<<dim3((dw + 31) / 32, (dh + 7) / 8), block, 0, s>>>(src, sw, sh, dst, dw, dh, offX, offY, P);
        return check_launch("warp kernel");
    }
    const WarpSource S = warp_source(src, sw, sh);
    const dim3 grid((dw + 63) / 64, (dh + 7) / 8);
    if (homography_affine(H)) k_warp<true><<<grid, block, 0, s>>>(S, dst, dw, dh, offX, offY, P);
    else k_warp<false><<<grid, block, 0, s>>>(S, dst, dw, dh, offX, offY, P);
    return check_launch("warp kernel");
}

int launch_median(const unsigned short* const* inputs, int n, unsigned short* out, int w, int h, float sigma,
                  cudaStream_t s)
{
    MedianInputs in;
    const int cnt = n < kMaxContributors ? n : kMaxContributors;
    uintptr_t align = reinterpret_cast<uintptr_t>(out);
    for (int i = 0; i < kMaxContributors; ++i)
    {
        in.p[i] = i < cnt ? inputs[i] : nullptr;
        if (i < cnt) align |= reinterpret_cast<uintptr_t>(inputs[i]);
    }
    const long long total = (long long)w * h * 3;
    const unsigned blocks = (unsigned)(((total + 1) / 2 + 255) / 256);
    const bool words = (align & 3) == 0;
    const float inv = 1.0f / (float)cnt;
#define I360B_MEDIAN(N)                                                              \
    if (cnt <= N)                                                                    \
    {                                                                                \
        if (words) k_median<N, true><<<blocks, 256, 0, s>>>(in, cnt, inv, total, sigma, out); \
        else k_median<N, false><<<blocks, 256, 0, s>>>(in, cnt, inv, total, sigma, out); \
        return check_launch("median kernel");                                        \
    }
    I360B_STACK_SIZES(I360B_MEDIAN)
#undef I360B_MEDIAN
    return fail(I360B_INVALID_PARAM, "numInputs must be 1-32.");
}

namespace
{
template <int N>
int run_warp_median(const StackParams& S, int cnt, int sw, int sh, unsigned short* out, int dw, int dh, int offX,
                    int offY, float sigma, cudaStream_t s)
{
    const size_t smem = (size_t)cnt * 3 * kWmThreads * sizeof(uint32_t);  // at most 48 KB, at 32 frames
    const unsigned grid = (unsigned)((dw + 63) / 64) * (unsigned)((dh + kWmThreads / 32 - 1) / (kWmThreads / 32));
    k_warp_median<N><<<grid, dim3(32, kWmThreads / 32), smem, s>>>(S, cnt, 1.0f / (float)cnt, sw, sh, out, dw, dh, offX, offY, sigma);
    return check_launch("warp + median kernel");
}
}  // namespace

int launch_warp_median(const unsigned short* const* frames, int n, int sw, int sh, const float* H, unsigned short* out,
                       int dw, int dh, int offX, int offY, float sigma, cudaStream_t s)
{
    StackParams S;
    S.affine = 0;
    const int cnt = n < kMaxContributors ? n : kMaxContributors;
    for (int i = 0; i < kMaxContributors; ++i)
    {
        S.src[i] = i < cnt ? frames[i] : nullptr;
        for (int q = 0; q < 9; ++q) S.H[i][q] = i < cnt ? H[(size_t)i * 9 + q] : 0.0f;
        if (i < cnt && homography_affine(S.H[i])) S.affine |= 1u << i;
    }
#define I360B_WARP_MEDIAN(N) \
    if (cnt <= N) return run_warp_median<N>(S, cnt, sw, sh, out, dw, dh, offX, offY, sigma, s);
    I360B_STACK_SIZES(I360B_WARP_MEDIAN)
#undef I360B_WARP_MEDIAN
    return fail(I360B_INVALID_PARAM, "numInputs must be 1-32.");
}

int launch_gain(unsigned short* data, long long n, float gain, cudaStream_t s)
{
    if (gain_is_identity(gain) || n <= 0) return I360B_SUCCESS;
    long long threads = (n + 7) / 8;
    k_gain<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(data, n, gain);
    return check_launch("gain kernel");
}
}  // namespace i360b
