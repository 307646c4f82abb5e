// How the prefill GEMMs (qkm_wgemm.cu) cut an expert's rows into units.  Host arithmetic only.
#pragma once

#include <math.h>
#include <stdint.h>

namespace qkm {

constexpr uint32_t kWgemmRows = 128, kWgemmRowsWide = 160;   // activation rows per unit

// Pairs that a resident expert has on average when `n` rows, each with n_used of n_expert experts, are at hand and routing is even.
// picked: of a larger batch only the rows that chose one of the `resident` experts (as the exchange of expert parallelism sends them).
inline double mean_pairs(uint32_t n, uint32_t n_used, uint32_t n_expert, uint32_t resident, bool picked) {
    const double per_expert = (double)n * n_used / n_expert;
    if (!picked || resident >= n_expert) return per_expert;
    return per_expert / (1.0 - pow(1.0 - (double)resident / n_expert, (double)n_used));
}

// 160 rows where the average expert has 116 to 165 pairs: most of those would need a second expansion of their weights for a few pairs
// over 128.  Elsewhere the fourth stage is worth more.  Layer, 256 experts, top 8, IQ3_XXS and IQ4_XS, tiles of 128 -> 160:
// 3400 tokens 443 -> 454 us, 3600: 471 -> 472, 3750: 493 -> 485, 3900: 517 -> 494, 4096: 561 -> 508, 5120: 697 -> 649, 5600: 717 -> 724.
// Only the mean is known here.  With uneven routing (pairs an expert 128 +- 52, +- 94, +- 161, the largest 275 to 695) the widths
// differ little and the wide one is not behind: 4096 tokens 521 -> 515 us, 531 -> 527, 536 -> 531; 5120: 637 -> 625, 637 -> 630, 647 -> 636.
inline uint32_t wgemm_rows_per_unit(double mean) { return mean > 115.0 && mean <= 165.0 ? kWgemmRowsWide : kWgemmRows; }

}  // namespace qkm
