// How many CTAs a cluster of the decode attention has; kept free of CUDA so that it can be checked on a host
// (tests/cpp/test_attn_plan.cpp).
#pragma once

#include <cstdint>

namespace prism {

// `clusters` of a launch on `sm_count` SMs, caches of at most `max_seq` positions of which the warps of a CTA take `cta_rows` at a
// time; `resident16`: clusters of 16 CTAs that this GPU holds at once.
//  * a tile for every warp while there are SMs to give one CTA each;
//  * 16 (more than the 8 that every GPU can place) only for contexts that still give every warp two tiles, and only if all
//    clusters are resident together: how many fit depends on the SMs of each GPC, not on their number in all.  A B200 holds 7
//    of 128-wide heads; 8 in two waves, 72B at 12 000 positions, two layers: 449 to 476 us a step, with clusters of 8 418 to 428.
//    4 clusters, 7B at 6 000: 138 with 16 as before.
inline uint32_t attn_cluster_ctas(uint32_t sm_count, uint32_t clusters, uint32_t max_seq, uint32_t cta_rows, uint32_t resident16) {
    uint32_t S = 1;
    while (S < 8 && S * cta_rows < max_seq && 2 * S * clusters <= sm_count) S *= 2;
    if (S == 8 && clusters <= resident16 && max_seq >= 32 * cta_rows) S = 16;
    return S;
}

}  // namespace prism
