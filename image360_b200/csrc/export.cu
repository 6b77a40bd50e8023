// Export of a panorama's rendered chunk outputs, device-resident:
//   * the preview composite of PanoramaExporter::ExportPreviewJpeg
//     (PanoramaExporter.cpp:46-102): every chunk's RGB48 output placed, in
//     chunk order, into an RGB8 canvas scaled so its longest edge is
//     maxDimension - placement and source pixel by the FP32 steps of
//     ComputeExportScale / ComputeChunkPlacement (PanoramaExporter.cpp:9-24)
//     and int(d / scale) (a table over d, shared by all chunks), samples >> 8,
//     pixels without a source left at 0.  When no two placements overlap (a
//     chunk grid) one launch covers every chunk; otherwise one launch per
//     chunk in chunk order reproduces the reference loop's last-writer-wins;
//   * the framed chunk blob of StorageEngine::WritePixelBuffer
//     (StorageEngine.cpp:130-144): int32 width, int32 height, the samples;
//   * the 16-bit RGB TIFF of WriteTiff16RGB (Tiff16Writer.cpp:40-97) of a
//     whole canvas of chunk outputs, assembled band by band on the device
//     (2-D copies of every chunk row range into a zeroed band) and streamed
//     to the file through two pinned buffers, so the host writes one band
//     while the next is copied.
// The JPEG encode of the preview is left to the caller's codec (nvJPEG in the
// reference, IImageCodec::Encode).
#include "render_plan.hpp"

#include <algorithm>
#include <cstdio>
#include <vector>

using namespace i360b;

namespace
{
struct ExportTile
{
    const unsigned short* src;
    int x, y, w, h;
};

// ComputeChunkPlacement (PanoramaExporter.cpp:16-24).
__host__ __device__ __forceinline__ void placement(const ExportTile& t, float scale, int* p)
{
#ifdef __CUDA_ARCH__
    p[0] = __float2int_rz(__fmul_rn((float)t.x, scale));
    p[1] = __float2int_rz(__fmul_rn((float)t.y, scale));
    const int w = __float2int_rz(__fmul_rn((float)t.w, scale)), h = __float2int_rz(__fmul_rn((float)t.h, scale));
#else
    p[0] = (int)((float)t.x * scale);
    p[1] = (int)((float)t.y * scale);
    const int w = (int)((float)t.w * scale), h = (int)((float)t.h * scale);
#endif
    p[2] = w > 1 ? w : 1;
    p[3] = h > 1 ? h : 1;
}

// int(d / scale) for every placement offset d (PanoramaExporter.cpp:86-87).
__global__ void k_export_source_table(float scale, int n, int* tab)
{
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d < n) tab[d] = __float2int_rz(__fdiv_rn((float)d, scale));
}

// Chunks [t0, t0 + gridDim.z) write their placements (PanoramaExporter.cpp:74-101).
// A warp writes kExportWords x 32 aligned 4-byte words of one placement row,
// a word per lane at a time, so its stores are whole 128-byte lines; the
// row's first and last bytes, which may share a word with a neighbouring
// placement, are stored by the byte.  Scale 1: the source samples of a word
// are four consecutive u16, read as two or three words (the samples of a row
// lie at one phase of the word grid).  Bound by HBM.  `clear`: a pixel without
// a source (rounding at the placement's edge) is written as 0 here - the
// placements do not overlap and cover the canvas, which is then not cleared
// beforehand.  Else such pixels are left alone.
// 17700 x 9600 at scale 1 (1.53 GB): 247 us (0.94 of the copy rate); one pixel
// per thread (2-byte loads, 1-byte stores) took 735 us and the clearing 83 us.
constexpr int kExportWords = 8;

__global__ void __launch_bounds__(256) k_export_place(const ExportTile* __restrict__ tiles, int t0, float scale,
                                                      int ow, int oh, bool clear, unsigned char* __restrict__ out)
{
    const ExportTile T = tiles[t0 + blockIdx.z];
    int p[4];
    placement(T, scale, p);
    const int dy = blockIdx.y * blockDim.y + threadIdx.y;
    if (dy >= p[3]) return;
    const int oy = p[1] + dy;
    if (oy < 0 || oy >= oh) return;
    const long long x0 = p[0] < 0 ? -(long long)p[0] : 0;
    const long long x1 = (long long)p[0] + p[2] > ow ? (long long)ow - p[0] : p[2];
    if (x0 >= x1) return;
    const int sy = dy;  // int(d / 1.0f) = d while the float holds d exactly
    const bool rowIn = sy < T.h;
    if (!rowIn && !clear) return;
    // bytes [b0, b1) of the placement row, at o + b
    const long long b0 = x0 * 3, b1 = x1 * 3;
    unsigned char* o = out + ((long long)oy * ow + p[0]) * 3;
    const long long rowElems = (long long)T.w * 3;
    const unsigned short* src = T.src + (size_t)sy * rowElems;  // read only where rowIn
    const long long chunkElems = (long long)T.h * rowElems;
    const long long firstElem = (long long)sy * rowElems;  // of the row, in the chunk
    const long long first = b0 - (long long)(reinterpret_cast<uintptr_t>(o + b0) & 3);  // first word's byte 0
    const bool odd = (reinterpret_cast<uintptr_t>(src + first) & 2) != 0;  // the samples straddle the word grid
    const long long base = first + (long long)blockIdx.x * (kExportWords * 128) + threadIdx.x * 4;
    if (base >= b1) return;
    // Samples [e0, e1) of the row may be read as words: the words that hold
    // samples b .. b + 3 hold b - 1 .. b + 4 at most, inside the chunk.
    const long long e0 = firstElem > 0 ? 0 : 1, e1 = firstElem + rowElems < chunkElems ? rowElems : rowElems - 1;
    if (rowIn && base >= b0 && base >= e0 && base + (kExportWords - 1) * 128 + 4 <= b1 &&
        base + (kExportWords - 1) * 128 + 4 <= e1)
    {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(src + base - (odd ? 1 : 0));
        uint32_t* d = reinterpret_cast<uint32_t*>(o + base);
        uint32_t r[kExportWords];
        if (!odd)
        {
#pragma unroll
            for (int j = 0; j < kExportWords; ++j)
                r[j] = __byte_perm(__ldcs(w + j * 64), __ldcs(w + j * 64 + 1), 0x7531);
        }
        else
        {
#pragma unroll
            for (int j = 0; j < kExportWords; ++j)
                r[j] = __byte_perm(__byte_perm(__ldcs(w + j * 64), __ldcs(w + j * 64 + 1), 0x0753),
                                   __ldcs(w + j * 64 + 2), 0x5210);
        }
#pragma unroll
        for (int j = 0; j < kExportWords; ++j) d[j * 32] = r[j];
        return;
    }
    // the ends of a row
    for (int j = 0; j < kExportWords; ++j)
    {
        const long long b = base + j * 128;
        if (b >= b1) return;
        const bool whole = b >= b0 && b + 4 <= b1;
        uint32_t v = 0;
        unsigned have = 0;  // bytes with a source
#pragma unroll
        for (int i = 0; i < 4; ++i)
        {
            const long long e = b + i;
            if (!rowIn || e < b0 || e >= b1) continue;
            if (e >= rowElems) continue;
            v |= (uint32_t)(__ldg(src + e) >> 8) << (8 * i);
            have |= 1u << i;
        }
        if (whole && (have == 15u || clear))
            *reinterpret_cast<uint32_t*>(o + b) = v;
        else
        {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (b + i >= b0 && b + i < b1 && (clear || ((have >> i) & 1u))) o[b + i] = (unsigned char)(v >> (8 * i));
        }
    }
}

// The same at any other scale: kExportPx pixels of a row per thread, 32 apart,
// each from the source pixel that the table gives.  Bound by load latency: the
// pixels' lookups and samples are in flight together.  16000 x 9000 into 9000 x
// 5062: 148 us; one pixel per thread 231 and the clearing 24; a word per lane,
// each byte looked up by itself, slower than either on small previews.
constexpr int kExportPx = 4;

__global__ void __launch_bounds__(256) k_export_scaled(const ExportTile* __restrict__ tiles, int t0, float scale,
                                                       int ow, int oh, const int* __restrict__ srcOf, bool clear,
                                                       unsigned char* __restrict__ out)
{
    const ExportTile T = tiles[t0 + blockIdx.z];
    int p[4];
    placement(T, scale, p);
    const int dx0 = blockIdx.x * (32 * kExportPx) + threadIdx.x, dy = blockIdx.y * blockDim.y + threadIdx.y;
    if (dx0 >= p[2] || dy >= p[3]) return;
    const int oy = p[1] + dy;
    if (oy < 0 || oy >= oh) return;
    const int sy = __ldg(srcOf + dy);
    const bool rowIn = sy >= 0 && sy < T.h;
    if (!rowIn && !clear) return;
    int sx[kExportPx];
#pragma unroll
    for (int k = 0; k < kExportPx; ++k) sx[k] = dx0 + 32 * k < p[2] ? __ldg(srcOf + dx0 + 32 * k) : -1;
    unsigned short v[kExportPx][3];
    const unsigned short* row = T.src + (size_t)(rowIn ? sy : 0) * T.w * 3;
#pragma unroll
    for (int k = 0; k < kExportPx; ++k)
    {
        const bool in = rowIn && sx[k] >= 0 && sx[k] < T.w;
        if (!in) sx[k] = -1;
#pragma unroll
        for (int c = 0; c < 3; ++c) v[k][c] = in ? __ldg(row + (size_t)sx[k] * 3 + c) : 0;
    }
#pragma unroll
    for (int k = 0; k < kExportPx; ++k)
    {
        const int dx = dx0 + 32 * k, ox = p[0] + dx;
        if (dx >= p[2] || ox < 0 || ox >= ow || (sx[k] < 0 && !clear)) continue;
        unsigned char* o = out + ((size_t)oy * ow + ox) * 3;
#pragma unroll
        for (int c = 0; c < 3; ++c) o[c] = (unsigned char)(v[k][c] >> 8);
    }
}

struct Scratch
{
    void* p = nullptr;
    cudaStream_t s = nullptr;
    ~Scratch() { dev_free(p, s); }
};

// ComputeExportScale (PanoramaExporter.cpp:9-14) and the composite size
// (PanoramaExporter.cpp:50-52).
void export_size(int totalW, int totalH, int maxDimension, float* scale, int* ow, int* oh)
{
    const int longest = totalW > totalH ? totalW : totalH;
    *scale = longest <= 0 ? 1.0f : (float)maxDimension / (float)longest;
    const int w = (int)((float)totalW * *scale), h = (int)((float)totalH * *scale);
    *ow = w > 1 ? w : 1;
    *oh = h > 1 ? h : 1;
}

int export_preview(const std::vector<ExportTile>& tiles, int totalW, int totalH, int maxDimension, unsigned char* dOut,
                   long long capacity, int* outW, int* outH, cudaStream_t s)
{
    if (!outW || !outH) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (maxDimension <= 0 || totalW <= 0 || totalH <= 0)
        return fail(I360B_INVALID_PARAM, "Invalid canvas size or maximum dimension.");
    if (tiles.size() > 65535) return fail(I360B_INVALID_PARAM, "More than 65535 chunks.");
    float scale;
    int ow, oh;
    export_size(totalW, totalH, maxDimension, &scale, &ow, &oh);
    *outW = ow;
    *outH = oh;
    if ((long long)ow * oh * 3 > capacity)
        return fail(I360B_INVALID_PARAM, "The %dx%d preview needs %lld bytes (capacity %lld).", ow, oh,
                    (long long)ow * oh * 3, capacity);
    if (!dOut) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (tiles.empty())
    {
        I360B_CUDA(cudaMemsetAsync(dOut, 0, (size_t)ow * oh * 3, s), "preview export");
        return I360B_SUCCESS;
    }
    // placements clipped to the canvas; overlap decides between one launch
    // and one launch per chunk
    std::vector<int> pl(tiles.size() * 4);
    int maxW = 1, maxH = 1;
    for (size_t t = 0; t < tiles.size(); ++t)
    {
        placement(tiles[t], scale, &pl[t * 4]);
        maxW = pl[t * 4 + 2] > maxW ? pl[t * 4 + 2] : maxW;
        maxH = pl[t * 4 + 3] > maxH ? pl[t * 4 + 3] : maxH;
    }
    bool overlap = false;
    for (size_t a = 0; a < tiles.size() && !overlap; ++a)
        for (size_t b = a + 1; b < tiles.size() && !overlap; ++b)
        {
            const int* A = &pl[a * 4];
            const int* B = &pl[b * 4];
            const int x0 = std::max(std::max(A[0], B[0]), 0), x1 = std::min(std::min(A[0] + A[2], B[0] + B[2]), ow);
            const int y0 = std::max(std::max(A[1], B[1]), 0), y1 = std::min(std::min(A[1] + A[3], B[1] + B[3]), oh);
            overlap = x0 < x1 && y0 < y1;
        }
    // Placements that do not overlap and cover the canvas write every pixel
    // themselves (a chunk grid at scale 1: one pass over the output instead of
    // two); else the canvas is cleared first.
    long long placed = 0;
    for (size_t t = 0; t < tiles.size(); ++t)
    {
        const int* A = &pl[t * 4];
        const long long x0 = std::max(A[0], 0), x1 = std::min<long long>((long long)A[0] + A[2], ow);
        const long long y0 = std::max(A[1], 0), y1 = std::min<long long>((long long)A[1] + A[3], oh);
        if (x0 < x1 && y0 < y1) placed += (x1 - x0) * (y1 - y0);
    }
    const bool clear = !overlap && placed == (long long)ow * oh;
    if (!clear) I360B_CUDA(cudaMemsetAsync(dOut, 0, (size_t)ow * oh * 3, s), "preview export");
    Scratch desc, tab;
    desc.s = tab.s = s;
    const int tabN = std::max(maxW, maxH);
    I360B_TRY(dev_alloc(&desc.p, tiles.size() * sizeof(ExportTile), s, "preview export"));
    // int(d / 1.0f) = d while the float holds d exactly
    const bool identity = scale == 1.0f && tabN <= (1 << 24);
    if (!identity) I360B_TRY(dev_alloc(&tab.p, (size_t)tabN * sizeof(int), s, "preview export"));
    I360B_CUDA(cudaMemcpyAsync(desc.p, tiles.data(), tiles.size() * sizeof(ExportTile), cudaMemcpyHostToDevice, s),
               "preview export");
    if (!identity)
    {
        k_export_source_table<<<(tabN + 255) / 256, 256, 0, s>>>(scale, tabN, static_cast<int*>(tab.p));
        I360B_TRY(check_launch("preview source table kernel"));
    }
    const dim3 block(32, 8);
    const ExportTile* dT = static_cast<const ExportTile*>(desc.p);
    const int* dTab = static_cast<const int*>(tab.p);
    // a row of w pixels spans at most 3w + 3 bytes from its first word on
    auto grid = [&](int w, int h, size_t chunks) {
        const long long cols = identity ? (3ll * w + 3 + kExportWords * 128 - 1) / (kExportWords * 128)
                                        : (w + 32 * kExportPx - 1) / (32 * kExportPx);
        return dim3((unsigned)cols, (unsigned)((h + 7) / 8), (unsigned)chunks);
    };
    auto place = [&](const dim3& g, int t0) {
        if (identity) k_export_place<<<g, block, 0, s>>>(dT, t0, scale, ow, oh, clear, dOut);
        else k_export_scaled<<<g, block, 0, s>>>(dT, t0, scale, ow, oh, dTab, clear, dOut);
        return check_launch("preview placement kernel");
    };
    if (!overlap) return place(grid(maxW, maxH, tiles.size()), 0);
    for (size_t t = 0; t < tiles.size(); ++t) I360B_TRY(place(grid(pl[t * 4 + 2], pl[t * 4 + 3], 1), (int)t));
    return I360B_SUCCESS;
}

void put_u16(unsigned char* p, uint16_t v)
{
    p[0] = (unsigned char)(v & 0xff);
    p[1] = (unsigned char)(v >> 8);
}

void put_u32(unsigned char* p, uint32_t v)
{
    for (int i = 0; i < 4; ++i) p[i] = (unsigned char)(v >> (8 * i));
}

// The bytes of Tiff16Writer.cpp:58-61 (header) and :69-90 (blocks after the
// pixel data, then the IFD) for a w x h image.
void tiff_header(int w, int h, unsigned char* hdr8, std::vector<unsigned char>& trailer)
{
    const uint32_t pix = (uint32_t)((size_t)w * h * 6);
    const uint32_t bps = 8 + pix, xres = bps + 6, yres = xres + 8, ifd = yres + 8;
    hdr8[0] = 'I';
    hdr8[1] = 'I';
    put_u16(hdr8 + 2, 42);
    put_u32(hdr8 + 4, ifd);
    trailer.assign(6 + 16 + 2 + 12 * 12 + 4, 0);
    unsigned char* p = trailer.data();
    put_u16(p, 16);
    put_u16(p + 2, 16);
    put_u16(p + 4, 16);
    put_u32(p + 6, 72);
    put_u32(p + 10, 1);
    put_u32(p + 14, 72);
    put_u32(p + 18, 1);
    p += 22;
    put_u16(p, 12);
    const uint32_t e[12][4] = {{256, 4, 1, (uint32_t)w}, {257, 4, 1, (uint32_t)h}, {258, 3, 3, bps},
                               {259, 3, 1, 1},          {262, 3, 1, 2},          {273, 4, 1, 8},
                               {277, 3, 1, 3},          {278, 4, 1, (uint32_t)h}, {279, 4, 1, pix},
                               {282, 5, 1, xres},       {283, 5, 1, yres},       {296, 3, 1, 2}};
    for (int i = 0; i < 12; ++i)
    {
        unsigned char* q = p + 2 + 12 * i;
        put_u16(q, (uint16_t)e[i][0]);
        put_u16(q + 2, (uint16_t)e[i][1]);
        put_u32(q + 4, e[i][2]);
        put_u32(q + 8, e[i][3]);
    }
}

struct HostBuf
{
    void* p = nullptr;
    ~HostBuf()
    {
        if (p) cudaFreeHost(p);
    }
};

struct File
{
    FILE* f = nullptr;
    ~File()
    {
        if (f) fclose(f);
    }
};

int write_tiff(const char* path, const std::vector<ExportTile>& tiles, int W, int H, cudaStream_t s)
{
    if (!path) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (W <= 0 || H <= 0) return fail(I360B_INVALID_PARAM, "Invalid dimensions.");
    const unsigned long long pix = (unsigned long long)W * H * 6;
    if (pix + 8 + 64 > 0xffffffffull)
        return fail(I360B_INVALID_PARAM, "A %dx%d RGB48 image does not fit the 32-bit offsets of a baseline TIFF.", W, H);
    const size_t rowBytes = (size_t)W * 6;
    int band = (int)((size_t)(256u << 20) / rowBytes);
    band = band < 1 ? 1 : (band > H ? H : band);
    const size_t bandBytes = rowBytes * band;
    Scratch dBand;
    dBand.s = s;
    I360B_TRY(dev_alloc(&dBand.p, bandBytes, s, "TIFF export"));
    HostBuf hb[2];
    for (auto& b : hb) I360B_CUDA(cudaHostAlloc(&b.p, bandBytes, cudaHostAllocDefault), "TIFF export staging");
    cudaEvent_t ev[2] = {nullptr, nullptr};
    for (auto& e : ev) I360B_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "TIFF export");
    struct Events
    {
        cudaEvent_t* e;
        ~Events()
        {
            cudaEventDestroy(e[0]);
            cudaEventDestroy(e[1]);
        }
    } evGuard{ev};
    File file;
    file.f = fopen(path, "wb");
    if (!file.f) return fail(I360B_INVALID_PARAM, "Cannot open %s for writing.", path);
    unsigned char hdr[8];
    std::vector<unsigned char> trailer;
    tiff_header(W, H, hdr, trailer);
    if (fwrite(hdr, 1, 8, file.f) != 8) return fail(I360B_INVALID_PARAM, "Cannot write %s.", path);
    const int nb = (H + band - 1) / band;
    size_t pending = 0;
    for (int b = 0; b <= nb; ++b)
    {
        if (b < nb)
        {
            const int y0 = b * band, y1 = y0 + band < H ? y0 + band : H;
            I360B_CUDA(cudaMemsetAsync(dBand.p, 0, rowBytes * (y1 - y0), s), "TIFF export");
            for (const ExportTile& t : tiles)
            {
                const int r0 = t.y > y0 ? t.y : y0, r1 = t.y + t.h < y1 ? t.y + t.h : y1;
                const int c0 = t.x > 0 ? t.x : 0, c1 = t.x + t.w < W ? t.x + t.w : W;
                if (r0 >= r1 || c0 >= c1) continue;
                const unsigned short* src = t.src + ((size_t)(r0 - t.y) * t.w + (c0 - t.x)) * 3;
                unsigned char* dst = static_cast<unsigned char*>(dBand.p) + (size_t)(r0 - y0) * rowBytes + (size_t)c0 * 6;
                I360B_CUDA(cudaMemcpy2DAsync(dst, rowBytes, src, (size_t)t.w * 6, (size_t)(c1 - c0) * 6, r1 - r0,
                                             cudaMemcpyDeviceToDevice, s),
                           "TIFF export band copy");
            }
            I360B_CUDA(cudaMemcpyAsync(hb[b & 1].p, dBand.p, rowBytes * (y1 - y0), cudaMemcpyDeviceToHost, s),
                       "TIFF export download");
            I360B_CUDA(cudaEventRecord(ev[b & 1], s), "TIFF export");
        }
        if (b > 0)
        {
            const int p = (b - 1) & 1;
            I360B_CUDA(cudaEventSynchronize(ev[p]), "TIFF export");
            if (fwrite(hb[p].p, 1, pending, file.f) != pending) return fail(I360B_INVALID_PARAM, "Cannot write %s.", path);
        }
        if (b < nb)
        {
            const int y0 = b * band, y1 = y0 + band < H ? y0 + band : H;
            pending = rowBytes * (y1 - y0);
        }
    }
    if (fwrite(trailer.data(), 1, trailer.size(), file.f) != trailer.size())
        return fail(I360B_INVALID_PARAM, "Cannot write %s.", path);
    if (fclose(file.f) != 0)
    {
        file.f = nullptr;
        return fail(I360B_INVALID_PARAM, "Cannot write %s.", path);
    }
    file.f = nullptr;
    return I360B_SUCCESS;
}

int require_ready()
{
    if (!initialized()) return fail(I360B_CUDA_ERROR, "Not initialized.");
    return ensure_ready();
}

int gather_tiles(const unsigned short* const* dTiles, const int* rects, int numTiles, bool skipNull,
                 std::vector<ExportTile>& out)
{
    if (numTiles < 0) return fail(I360B_INVALID_PARAM, "Invalid chunk count.");
    if (numTiles > 0 && (!dTiles || !rects)) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    for (int t = 0; t < numTiles; ++t)
    {
        const int* r = rects + 4 * t;
        if (r[2] <= 0 || r[3] <= 0) return fail(I360B_INVALID_PARAM, "Chunk %d has invalid dimensions.", t);
        if (!dTiles[t])
        {
            if (skipNull) continue;
            return fail(I360B_INVALID_PARAM, "Chunk %d has no output buffer.", t);
        }
        out.push_back(ExportTile{dTiles[t], r[0], r[1], r[2], r[3]});
    }
    return I360B_SUCCESS;
}

void plan_tiles(const i360b_render_plan* plan, bool renderedOnly, std::vector<ExportTile>& out)
{
    const Plan& P = plan->plan;
    for (int t = 0; t < P.nTiles; ++t)
    {
        if (renderedOnly && P.tileListed[t] == 0) continue;  // no render task (PanoramaExporter.cpp:69)
        const int* r = &P.tileRects[(size_t)t * 4];
        out.push_back(ExportTile{P.tiles[t].out, r[0], r[1], r[2], r[3]});
    }
}
}  // namespace

extern "C" int i360b_launch_export_preview(const unsigned short* const* dChunks, const int* rects, int numChunks,
                                           int totalW, int totalH, int maxDimension, unsigned char* dOut,
                                           long long capacity, int* outW, int* outH, void* stream)
{
    clear_error();
    I360B_TRY(require_ready());
    std::vector<ExportTile> tiles;
    I360B_TRY(gather_tiles(dChunks, rects, numChunks, true, tiles));
    return export_preview(tiles, totalW, totalH, maxDimension, dOut, capacity, outW, outH,
                          static_cast<cudaStream_t>(stream));
}

extern "C" int i360b_render_plan_export_preview(i360b_render_plan* plan, int totalW, int totalH, int maxDimension,
                                                unsigned char* dOut, long long capacity, int* outW, int* outH,
                                                void* stream)
{
    clear_error();
    if (!plan) return fail(I360B_INVALID_PARAM, "Null plan.");
    I360B_TRY(require_ready());
    std::vector<ExportTile> tiles;
    plan_tiles(plan, true, tiles);
    return export_preview(tiles, totalW, totalH, maxDimension, dOut, capacity, outW, outH,
                          static_cast<cudaStream_t>(stream));
}

extern "C" int i360b_write_tiff16_chunks(const char* path, const unsigned short* const* dChunks, const int* rects,
                                         int numChunks, int canvasW, int canvasH, void* stream)
{
    clear_error();
    I360B_TRY(require_ready());
    std::vector<ExportTile> tiles;
    I360B_TRY(gather_tiles(dChunks, rects, numChunks, true, tiles));
    return write_tiff(path, tiles, canvasW, canvasH, static_cast<cudaStream_t>(stream));
}

extern "C" int i360b_render_plan_write_tiff16(i360b_render_plan* plan, const char* path, int canvasW, int canvasH,
                                              void* stream)
{
    clear_error();
    if (!plan) return fail(I360B_INVALID_PARAM, "Null plan.");
    I360B_TRY(require_ready());
    std::vector<ExportTile> tiles;
    plan_tiles(plan, false, tiles);
    return write_tiff(path, tiles, canvasW, canvasH, static_cast<cudaStream_t>(stream));
}

extern "C" int i360b_download_framed(const unsigned short* dData, int width, int height, void* hostOut, void* stream)
{
    clear_error();
    I360B_TRY(require_ready());
    if (!dData || !hostOut) return fail(I360B_INVALID_PARAM, "Null pointer argument.");
    if (width <= 0 || height <= 0) return fail(I360B_INVALID_PARAM, "Invalid dimensions.");
    unsigned char* o = static_cast<unsigned char*>(hostOut);
    put_u32(o, (uint32_t)width);
    put_u32(o + 4, (uint32_t)height);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    I360B_CUDA(cudaMemcpyAsync(o + 8, dData, (size_t)width * height * 6, cudaMemcpyDeviceToHost, s),
               "framed download");
    I360B_CUDA(cudaStreamSynchronize(s), "framed download");
    return I360B_SUCCESS;
}
