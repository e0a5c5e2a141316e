// tc_shape.h -- the tile shape of a tensor-core product (tc_gemm.cu), by its size.
#pragma once
#include <stdint.h>

namespace gbgpu {

// 128 x 256 (one limb), 128 x 128 (two) or 128 x 64 tiles; 128 x 64 tiles with their
// accumulators twice (one and two limbs)
constexpr int TC_BIG = 0, TC_MID = 2;

// The narrow shape for a product of up to three waves of wide tiles: a wave costs
// a fixed part (the epilogue, which the next tile's MMAs do not overlap in the wide
// shapes with one accumulator set) and a part per 128 columns of K, in 10 ns,
// fitted to the times of both shapes over 1 to 3 waves and K = 200 .. 4000:
//   two limbs, 2520 x 1220: K = 200 66 / 54 us wide / narrow, 937 80 / 67,
//   2000 101 / 89, 4000 125 / 135; 3032 x 1476: 937 81 / 79, 2000 90 / 104;
//   one limb, 2520 x 2500: 200 68 / 61, 937 82 / 72, 2000 78 / 94.
// A single wave of wide tiles leaves SMs idle that the narrow ones use (the larger
// allowance).  With more waves the wide shape's fetches overlap its epilogue, and
// it wins at every K (5000 x 20000 x 256, two limbs: 302 against 316 us).
inline bool few_waves_mid(int L, int K, int64_t ww, int64_t wn) {
    const int64_t steps = (K + 127) / 128;
    const int64_t cost_w = ww * (L == 1 ? 55 * steps + 1100 : 95 * steps + 750);
    const int64_t cost_n = wn * (L == 1 ? 46 * steps + 170 : 81 * steps + 190);
    return 100 * cost_n < (ww == 1 ? 131 : 108) * cost_w;
}

// The shape for a product of L limbs on `sms` SMs; tuned: the autotuner's choice for
// this K, -1 for none.  With fewer narrow tiles than SMs a wide one only lengthens the
// one tile of its SM (two limbs: 512 x 512 x 128 8.4 us against 6.4, 1024 x 1024 x
// 1024 14.0 against 11.7).  The tuner times products of four waves and more, so its
// choice holds for those alone: one for the wide shape would cost 2520 x 1220 x 200,
// two limbs, 66 us instead of 54.
inline int tc_shape(int L, int64_t M, int64_t N, int K, int64_t batch, int sms, int tuned) {
    const int64_t rows = (M + 127) / 128 * batch, wide_cols = L == 1 ? 256 : 128;
    const int64_t narrow = rows * ((N + 63) / 64), wide = rows * ((N + wide_cols - 1) / wide_cols);
    if (L > 2) return TC_BIG;
    if (narrow <= sms) return TC_MID;
    const int64_t ww = (wide + sms - 1) / sms;
    if (ww <= 3) return few_waves_mid(L, K, ww, (narrow + sms - 1) / sms) ? TC_MID : TC_BIG;
    return tuned >= 0 ? tuned : TC_BIG;
}

}  // namespace gbgpu
