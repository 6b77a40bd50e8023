// Bilinear taps read as words (part of warp_taps.cuh; by itself so that a host
// program can compile it and watch its reads).
#pragma once

#include <cstdint>

namespace i360b
{
// Two horizontally adjacent RGB48 pixels (six u16) from byte offset o (even)
// of a frame's words, as three words in memory order: the aligned words that
// hold them, shifted together.  Half the L1 accesses of six 2-byte loads.
// Where the six end in the middle of a word only that half is read: the frame,
// and its allocation, may end there.  A frame that starts in the middle of a
// word has its first word read whole, from the 2 bytes before the frame on,
// which are its allocation's (allocations start on words) and are shifted
// out: a test for them in every load would cost the tile warp and the stack
// 2 to 4 %.
template <typename Off>
__device__ __forceinline__ void load_tap_pair(const uint32_t* words, Off o, uint32_t w[3])
{
    const uint32_t* q = words + (o >> 2);
    const unsigned sh = (unsigned)o << 3;  // 0 or 16, modulo 32
    const uint32_t r0 = __ldg(q), r1 = __ldg(q + 1), r2 = __ldg(q + 2);
    uint32_t r3 = 0;
    if (o & 2) r3 = __ldg(reinterpret_cast<const unsigned short*>(q + 3));
    w[0] = __funnelshift_r(r0, r1, sh);
    w[1] = __funnelshift_r(r1, r2, sh);
    w[2] = __funnelshift_r(r2, r3, sh);
}
}  // namespace i360b
