// split_plan.h -- K ranges per row tile of the skinny products on the tensor cores
// (skinny.cu): plain functions of the tile count, the steps of K and the SM count, so
// that they can be checked without a device.
#pragma once

#include <math.h>
#include <stdint.h>

#include <numeric>

namespace gb {

// K ranges per tile: units for four waves and more (one range when there are as
// many tiles), up to twice as many where that leaves the last wave fuller; at
// least `least` of the nst steps of K a range.
inline int balanced_splits(int64_t tiles, int64_t nst, int64_t least, int sm_count) {
    const double sms = sm_count;
    int best = 1;
    double best_fill = 0.0;
    for (int s = 1; s <= 64 && (s == 1 || nst / s >= least); s++) {
        const double units = (double)(tiles * s), fill = units / (ceil(units / sms) * sms);
        if (units >= 8.0 * sms && s > 1 && best_fill > 0.0) break;
        if (units < 4.0 * sms || fill > best_fill + 0.02) {
            best = s;
            best_fill = units < 4.0 * sms ? 0.0 : fill;
        }
        if (tiles >= 4 * (int64_t)sms) break;
    }
    return best;
}

// Ranges that double while there are fewer than four waves of units.
inline int doubled_splits(int64_t tiles, int64_t nst, int64_t least, int sm_count) {
    int s = 1;
    while (tiles * s < 4 * (int64_t)sm_count && nst / (s * 2) >= least && s < 64) s *= 2;
    return s;
}

// Steps of K that the CTA with the most work walks when each tile has (up to) `splits`
// ranges, all but the last range of a tile of the same length.  CTA b takes units b,
// b + SMs, ...  by_range: units in the order of their ranges, the short ones last; else
// the ranges of a tile in a row.
inline int64_t walked_steps(int64_t tiles, int64_t nst, int splits, bool by_range, int sm_count) {
    const int64_t per = (nst + splits - 1) / splits, ranges = (nst + per - 1) / per, units = tiles * ranges;
    const int64_t less = per - (nst - (ranges - 1) * per), most = (units + sm_count - 1) / sm_count;
    if (by_range) {   // of the CTAs with the most units the first has the fewest short ones
        const int64_t whole = (units - tiles + sm_count - 1) / sm_count;
        return most * per - (most - whole) * less;
    }
    // the CTAs below `full` have one unit more; short ones repeat every `ranges` CTAs
    const int64_t full = units - (most - 1) * sm_count;
    int64_t worst = 0;
    for (int64_t i = 0; i < 2 * ranges; i++) {
        const int64_t n = i < ranges ? most : most - 1, b = i < ranges ? i : full + i - ranges;
        if (b >= (i < ranges ? full : sm_count)) continue;
        int64_t shorts = 0;
        for (int64_t u = 0; u < n; u++) shorts += (b + u * sm_count) % ranges == ranges - 1;
        if (n * per - shorts * less > worst) worst = n * per - shorts * less;
    }
    return worst;
}

// Whether FP64 units are taken in the order of their K ranges (K-major X: CTAs at work
// read neighbouring pieces of the same k lines) or the ranges of a tile in a row.  X
// that is copied in 8-byte pieces (odd leading dimensions) loses by the former where a
// CTA meets only few row tiles, i.e. the tile and SM counts share a large factor: us,
// by ranges / in a row, 2358 x 215593, n 10 (19 tiles) 2241 / 1887; 4850 x 98864, n 3
// (38) 2105 / 1701; 1976 x 204156, n 5 (16) 1525 / 1445; factors up to 4 gain 4 per cent by
// ranges.  X read by TMA gains 2 to 7 per cent throughout.
inline bool oz_by_range(bool kmajor, bool pieces, int64_t tiles, int sm_count) {
    return kmajor && !(pieces && std::gcd(tiles, (int64_t)sm_count) >= 8);
}

// FP64 (steps of 512 k).  With few tiles more ranges can spill units into another
// wave, and every SM then waits for those: the doubled count where its longest walk is
// shorter by more than a twentieth.  Row-major X, us, balanced / doubled: 3919 x 4701,
// n 43, 355 / 282 (155 units of 2 steps on 152 SMs against 124 of 3); 4419 x 7256, n 15,
// 169 / 125; 1088 x 19414, n 42, 280 / 222; but 6482 x 3073, n 54, 244 / 281 (walks of 4).
inline int oz_splits(int64_t tiles, int64_t nchunks, bool by_range, int sm_count) {
    const int balanced = balanced_splits(tiles, nchunks, 2, sm_count);
    const int doubled = doubled_splits(tiles, nchunks, 2, sm_count);
    if (balanced == doubled) return balanced;
    const int64_t walk = walked_steps(tiles, nchunks, balanced, by_range, sm_count);
    return 1.05 * (double)walked_steps(tiles, nchunks, doubled, by_range, sm_count) < (double)walk ? doubled : balanced;
}

}  // namespace gb
