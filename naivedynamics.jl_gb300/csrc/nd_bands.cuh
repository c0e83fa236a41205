// nd_bands.cuh -- where the pairs of the all-pairs Coulomb recurrence lie in its
// bands of rows (see nd_compat.cu).  Plain integer arithmetic, also for a host
// compiler.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define ND_HD __host__ __device__
#else
#define ND_HD
#endif

namespace nd {

constexpr int kBandRows = 256;         // rows of a band: eight a lane
constexpr int kBandPad = 128;          // column words before the first (columns leaving a band early)
constexpr int kBandMaxAtoms = 20480;   // the columns' array fits a block's shared memory

constexpr int kBandCopy = 4;           // steps (of 4 KB) a copy brings
// steps (tiles of four columns a lane) of band 0, padded to whole copies: band
// b has band_steps(n) - 64 b
ND_HD inline int32_t band_steps(int32_t n) {
    return ((n + 3) / 4 + 31 + kBandCopy - 1) / kBandCopy * kBandCopy;
}
ND_HD inline int64_t band_off(int32_t b, int32_t P) {  // in steps
    return (int64_t)b * P - 32LL * b * (b - 1);
}
// bytes of the columns' array (words written: 4 (band_steps(n) - 31) + kBandPad)
ND_HD inline int32_t band_col_bytes(int32_t n) {
    return (8 * (4 * band_steps(n) + kBandPad) + 127) & ~127;
}
// Row r (0 .. 7) of `lane` in band b, and the first column of its tile of step t.
ND_HD inline int32_t band_row(int32_t b, int32_t lane, int32_t r) {
    return kBandRows * b + 8 * lane + r;
}
ND_HD inline int32_t band_col(int32_t b, int32_t lane, int32_t t) {
    return kBandRows * b + 4 * (t - lane);
}
// Whether row i meets a later atom in columns j0 .. j0 + 3 (rows past the last
// atom meet none: their position and charge do not exist).
ND_HD inline bool band_tile_has_pair(int32_t i, int32_t j0, int32_t n) {
    return i < n - 1 && j0 + 3 > i && j0 < n;
}

}  // namespace nd
