// Shifts in cells to 64-bit fixed-point phase slopes (host and device).
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define ISAR_HD __host__ __device__ __forceinline__
#else
#define ISAR_HD static inline
#endif

namespace isar {

// v / N cycles for a power of two N, as a signed fraction of a cycle in units
// of 2^-64 (rounded half to even, whole cycles dropped), from v's bits in
// integer instructions.  FP64 issues about two operations per clock and SM on
// this part, so one warp-wide FP64 instruction holds the SM's FP64 pipe for
// ~16 clocks: with division, floor and scaling in double in every warp, and
// three FP64 block sums, the range alignment of a 1024 x 8192 frame took
// 33 us more (1556 -> 1523 us per frame; a batch of 32 learned frames 16.68 ->
// 16.17 ms).  A shift that is no number (the correlation with a missing pulse
// has no peak to fit) or infinite is half a cycle, what the device's
// double-to-integer conversion makes of it.
ISAR_HD int64_t cells_to_fixed(uint64_t bits, int lgN)
{
    const int ex = (int)((bits >> 52) & 0x7ff);
    if (ex == 0) return 0;                                     // zero (subnormals round to it)
    if (ex == 0x7ff) return INT64_MIN;                         // NaN, infinity
    const uint64_t man = (bits & 0xfffffffffffffull) | 0x10000000000000ull;
    const int k = ex - 1075 + 64 - lgN;                        // v / N * 2^64 = man * 2^k
    uint64_t r;
    if (k >= 64 || k < -54) {
        r = 0;
    } else if (k >= 0) {
        r = man << k;                                          // whole cycles fall off the top
    } else {
        const int d = -k;                                      // 1 .. 54: round half to even
        r = man >> d;
        const uint64_t rem = man & ((1ull << d) - 1), half = 1ull << (d - 1);
        r += (rem > half || (rem == half && (r & 1))) ? 1 : 0;
    }
    return (int64_t)((bits >> 63) ? 0ull - r : r);
}

}  // namespace isar
