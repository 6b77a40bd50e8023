// The backward bilinear warp of one destination pixel, shared by the single
// warp, the fused warp + median stack (pixel_ops.cu) and the tile warp of a
// render plan (blend_kernels.cu).  Arithmetic of WarpPerspective_Scalar.cpp:8-45
// and WarpPerspectiveKernels.h:16-43: FP32, one rounding per operation, source
// order.
#pragma once

#include "common.cuh"
#include "tap_words.cuh"

namespace i360b
{
// The low / high 16 bits of a word as the float 2^23 + value: the bytes over
// 2^23's exponent, one byte permute.
__device__ __forceinline__ float u16lo23(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7410)); }
__device__ __forceinline__ float u16hi23(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7432)); }
// The same as the value itself (an exact subtraction, see u2f).
__device__ __forceinline__ float u16lo_f(uint32_t w) { return __fsub_rn(u16lo23(w), 8388608.0f); }
__device__ __forceinline__ float u16hi_f(uint32_t w) { return __fsub_rn(u16hi23(w), 8388608.0f); }

// A source frame as the warp reads it: 4-byte words from the word that holds
// its first sample on.
struct WarpSource
{
    const uint32_t* words;
    uint32_t phase;     // bytes of the first sample past words: 0 or 2
    uint32_t pitch;     // bytes per row
    int width;
    float maxX, maxY;   // positions below these have all four taps
    bool wide;          // byte offsets need more than 32 bits
};

__host__ __device__ __forceinline__ WarpSource warp_source(const unsigned short* src, int w, int h)
{
    WarpSource s;
    const uintptr_t a = reinterpret_cast<uintptr_t>(src);
    s.words = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3));
    s.phase = (uint32_t)(a & 2);
    s.pitch = (uint32_t)w * 6u;
    s.width = w;
    s.maxX = (float)(w - 1);
    s.maxY = (float)(h - 1);
    s.wide = (unsigned long long)w * (unsigned long long)h * 6ull + 8ull > 0xffffffffull;
    return s;
}

__host__ __device__ __forceinline__ bool homography_affine(const float* H)
{
    return H[6] == 0.0f && H[7] == 0.0f && H[8] == 1.0f;
}

// Both rows of taps at column x0 of row y0, given as 2^23 + x0 and 2^23 + y0.
__device__ __forceinline__ void load_taps(const WarpSource& s, float x23, float y23, uint32_t t[3], uint32_t b[3])
{
    const uint32_t xb = __float_as_uint(x23), yb = __float_as_uint(y23);
    if (!s.wide)
    {
        // (y0 w + x0) 6 modulo 2^32, the exponent bits taken out in the constant
        const uint32_t bias = 0x4B000000u * ((uint32_t)s.width + 1u) * 6u - s.phase;
        const uint32_t o = (yb * (uint32_t)s.width + xb) * 6u - bias;
        load_tap_pair(s.words, o, t);
        load_tap_pair(s.words, o + s.pitch, b);
    }
    else
    {
        const unsigned long long o =
            ((unsigned long long)(yb & 0x7FFFFFu) * s.width + (xb & 0x7FFFFFu)) * 6ull + s.phase;
        load_tap_pair(s.words, o, t);
        load_tap_pair(s.words, o + s.pitch, b);
    }
}

// The warp of two destination pixels (dX: their x) of one row, per channel
// 2^23 + the value truncated to uint16 (the truncated value is the low 16
// bits of each float); 2^23, value 0, where a pixel is (0,0,0) by the
// |w| < 1e-10 or the range rule (stated on the floats, so NaN and
// out-of-int-range positions are invalid as in the reference's int
// conversion).  H is row-major; hy = {H[1] dY, H[4] dY, H[7] dY} of the row
// (the same rounded products, summed in the reference's order).  AFFINE: the
// third row of H is (0, 0, 1), so the divisor is exactly 1 for every pixel
// and the divisions, which return their dividend, are skipped.
//
// The two pixels' arithmetic is paired (f32x2).  A tap t arrives as T =
// 2^23 + t, and fma(w, T, -2^23 w) is w t rounded once - the reference's
// product, without a subtraction per tap.  The reference clamps to [0, 65535]
// before truncating; the weights are products of values in [0, 1], so the mix
// lies in [0, 65535 (1 + 8 2^-24)], below 65536, and the clamps never change
// the truncated value.
template <bool AFFINE>
__device__ __forceinline__ void warp_pair23(const WarpSource& s, const float* H, const float* hy, float dXa, float dXb,
                                            bool inA, bool inB, f32x2 out[3])
{
    const f32x2 k23 = dup2(8388608.0f), m23 = dup2(-8388608.0f);
    out[0] = out[1] = out[2] = k23;
    f32x2 sx = add2(add2(pack2(fmul(H[0], dXa), fmul(H[0], dXb)), dup2(hy[0])), dup2(H[2]));
    f32x2 sy = add2(add2(pack2(fmul(H[3], dXa), fmul(H[3], dXb)), dup2(hy[1])), dup2(H[5]));
    bool va = inA, vb = inB;
    if (!AFFINE)
    {
        const f32x2 sw = add2(add2(pack2(fmul(H[6], dXa), fmul(H[6], dXb)), dup2(hy[2])), dup2(H[8]));
        va = va && !(fabsf(lo2(sw)) < 1e-10f);
        vb = vb && !(fabsf(hi2(sw)) < 1e-10f);
        sx = pack2(fdiv(lo2(sx), lo2(sw)), fdiv(hi2(sx), hi2(sw)));
        sy = pack2(fdiv(lo2(sy), lo2(sw)), fdiv(hi2(sy), hi2(sw)));
    }
    va = va && lo2(sx) >= 0.0f && lo2(sx) < s.maxX && lo2(sy) >= 0.0f && lo2(sy) < s.maxY;
    vb = vb && hi2(sx) >= 0.0f && hi2(sx) < s.maxX && hi2(sy) >= 0.0f && hi2(sy) < s.maxY;
    if (!(va || vb)) return;
    if (!(va && vb))
    {
        // the invalid pixel reads the valid one's taps; its result is dropped
        sx = va ? dup2(lo2(sx)) : dup2(hi2(sx));
        sy = va ? dup2(lo2(sy)) : dup2(hi2(sy));
    }
    // 0 <= sx, sy < 2^23: 2^23 + floor(s) exactly, and s - floor(s)
    const f32x2 bx = add2_rz(sx, k23), by = add2_rz(sy, k23);
    const f32x2 neg1 = dup2(-1.0f), one = dup2(1.0f);
    const f32x2 fx = fma2(add2(bx, m23), neg1, sx), fy = fma2(add2(by, m23), neg1, sy);  // products by -1 are exact
    const f32x2 gx = fma2(fx, neg1, one), gy = fma2(fy, neg1, one);
    // weights (their only uses are fma operands, so no sum can contract them) and -2^23 w
    const f32x2 nz = neg_zero2();
    const f32x2 w00 = mulx2(gx, gy, nz), w10 = mulx2(fx, gy, nz), w01 = mulx2(gx, fy, nz), w11 = mulx2(fx, fy, nz);
    const f32x2 c00 = mulx2(w00, m23, nz), c10 = mulx2(w10, m23, nz), c01 = mulx2(w01, m23, nz),
                c11 = mulx2(w11, m23, nz);
    uint32_t ta[3], ba[3], tb[3], bb[3];
    load_taps(s, lo2(bx), lo2(by), ta, ba);
    load_taps(s, hi2(bx), hi2(by), tb, bb);
    auto mix = [&](f32x2 t00, f32x2 t10, f32x2 t01, f32x2 t11) {
        return add2_rz(add2(add2(add2(fma2(w00, t00, c00), fma2(w10, t10, c10)), fma2(w01, t01, c01)),
                            fma2(w11, t11, c11)),
                       k23);
    };
    auto lo = [](uint32_t a, uint32_t b) { return pack2(u16lo23(a), u16lo23(b)); };
    auto hi = [](uint32_t a, uint32_t b) { return pack2(u16hi23(a), u16hi23(b)); };
    out[0] = mix(lo(ta[0], tb[0]), hi(ta[1], tb[1]), lo(ba[0], bb[0]), hi(ba[1], bb[1]));
    out[1] = mix(hi(ta[0], tb[0]), lo(ta[2], tb[2]), hi(ba[0], bb[0]), lo(ba[2], bb[2]));
    out[2] = mix(lo(ta[1], tb[1]), hi(ta[2], tb[2]), lo(ba[1], bb[1]), hi(ba[2], bb[2]));
    if (!va || !vb)
#pragma unroll
        for (int c = 0; c < 3; ++c)
            out[c] = pack2(va ? lo2(out[c]) : 8388608.0f, vb ? hi2(out[c]) : 8388608.0f);
}

// ApplyGain of a warped pair given as 2^23 + value (GainColorOps.cpp:16-26),
// in the same form (both clamps: the gain is any number).
__device__ __forceinline__ f32x2 gain_pair23(f32x2 v23, float gain)
{
    const f32x2 v = add2(v23, dup2(-8388608.0f));
    float a = fmul(lo2(v), gain), b = fmul(hi2(v), gain);
    a = a > 0.0f ? a : 0.0f;  // NaN -> 0
    b = b > 0.0f ? b : 0.0f;
    a = a < 65535.0f ? a : 65535.0f;
    b = b < 65535.0f ? b : 65535.0f;
    return add2_rz(pack2(a, b), dup2(8388608.0f));
}
}  // namespace i360b
