// Watches the reads of the warp's tap loads (image360_b200/csrc/tap_words.cuh):
// for frames of every small size at both phases of the word grid and every
// position with four taps, the values are the frame's and no byte is read past
// its end, nor before the word it starts in.  Prints the first violation; exit
// code 0: none.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#define __device__
#define __forceinline__ inline
static const unsigned char *g_first, *g_end;
static long g_outside;
template <typename T>
static T __ldg(const T* p)
{
    const unsigned char* b = reinterpret_cast<const unsigned char*>(p);
    if (b < g_first || b + sizeof(T) > g_end) ++g_outside;
    T v;
    std::memcpy(&v, b, sizeof(T));
    return v;
}
static uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, unsigned sh)
{
    return (uint32_t)(((uint64_t)hi << 32 | lo) >> (sh & 31));
}
#include "tap_words.cuh"

int main()
{
    for (int w = 2; w < 9; ++w)
        for (int h = 2; h < 6; ++h)
            for (int phase = 0; phase < 4; phase += 2)
            {
                std::vector<uint32_t> mem((size_t)w * h * 6 / 4 + 8, 0xa5a5a5a5u);
                unsigned char* base = reinterpret_cast<unsigned char*>(mem.data() + 2) + phase;
                g_first = base - phase;
                g_end = base + (size_t)w * h * 6;
                std::vector<uint16_t> px((size_t)w * h * 3);
                for (size_t i = 0; i < px.size(); ++i) px[i] = (uint16_t)(i * 40503u + 7);
                std::memcpy(base, px.data(), px.size() * 2);
                for (int y = 0; y + 1 < h; ++y)
                    for (int x = 0; x + 1 < w; ++x)
                        for (int wide = 0; wide < 2; ++wide)
                        {
                            uint32_t t[3], b[3];
                            const uint32_t o = (uint32_t)((y * w + x) * 6 + phase);
                            g_outside = 0;
                            if (wide)
                            {
                                i360b::load_tap_pair(mem.data() + 2, (unsigned long long)o, t);
                                i360b::load_tap_pair(mem.data() + 2, (unsigned long long)o + w * 6, b);
                            }
                            else
                            {
                                i360b::load_tap_pair(mem.data() + 2, o, t);
                                i360b::load_tap_pair(mem.data() + 2, o + (uint32_t)w * 6u, b);
                            }
                            const uint16_t* r0 = px.data() + (size_t)(y * w + x) * 3;
                            if (g_outside || std::memcmp(t, r0, 12) || std::memcmp(b, r0 + 3 * w, 12))
                            {
                                std::printf("%dx%d phase %d at (%d, %d): %ld reads outside, values %s\n", w, h, phase, x,
                                            y, g_outside, std::memcmp(t, r0, 12) || std::memcmp(b, r0 + 3 * w, 12) ? "differ" : "equal");
                                return 1;
                            }
                        }
            }
    std::puts("every read inside the frame's words, none past its end");
    return 0;
}
