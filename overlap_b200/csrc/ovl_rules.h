// Rules that choose a launch from sizes alone: plain host C++, so that they can
// be evaluated without a GPU (tests/test_dispatch_rules.py).
#pragma once

#include <algorithm>

namespace ovl {

// Mode blocks a CTA runs on one gathering of its sites' links (link tables,
// packed link records), at most.
constexpr int kLinkBlocks = 8;

// The packed FP32 stencil: `tiles` CTAs along the sites, n_mb mode blocks.
// kLinkBlocks, halved while the launch would hold fewer than `least` CTAs.
inline int mode_blocks_per_cta(int tiles, int n_mb, int least) {
    int m = kLinkBlocks;
    while (m > 1 && (long long)tiles * ((n_mb + m - 1) / m) < least) m /= 2;
    return m;
}

// The FP64 and FP40 stencils, two CTAs of 8 warps per SM; 1 selects the stencil
// without the table.  The time of a launch goes with the mode blocks that the
// fullest SM runs, on CTAs of m blocks and 0.15 of a block for the gathering; an
// odd last CTA has the SM to itself and takes longer than its share, counted as
// half a CTA more.  The largest m within 6 % of the least such time: where the
// times are equal fewer, longer CTAs gather less.
// Measured (us per step of a context on its own / with three contexts in turn
// on their own streams, which fill each other's idle SMs), m = 8, 4, 2, 1; the
// rule's choice in brackets:
//   FP64  6^3 x 1024 modes    49/32 45/29 43/30 [39/32]
//         6^3 x 4096        154/111 [132/113] 136/118 132/119
//         8^3 x 256           49/26 33/20 [33/18] 31/20
//         8^3 x 1024          [87/67] 90/68 91/73 86/72
//         8^3 x 2048        165/134 [164/135] 160/141 156/140
//         10 x 13 x 9 x 512   [94/76] 96/78 99/84 97/83
//         12^3 x 128          45/30 45/30 48/32 [41/33]
//         12^3 x 512        161/120 [138/118] 137/121 133/120
//   FP40  12^3 x 256          70/45 58/46 [62/50] 58/52
//         12^3 x 512         129/88 [111/90] 115/98 115/100
// One CTA per SM as the only condition is best for contexts in turn and up to 26 %
// slower for one on its own (17 % at 12^3 x 512: m = 8); four CTAs per SM is up to 20 %
// slower in turn (9 % at 8^3 x 1024: m = 2).  Over 102 launches of 6^3 to 16^3 sites and
// 64 to 4096 modes, geometric means of the time alone against four CTAs per SM and of
// the time in turn against one: this rule 1.00 and 1.01, one CTA per SM 1.03 and 1, four
// 1 and 1.03.
inline int link_blocks(int site_ctas, int n_mb, int sm_count) {
    double cost[kLinkBlocks + 1], least = 0.0;
    for (int m = kLinkBlocks; m >= 1; m /= 2) {
        const long long ctas = (long long)site_ctas * ((n_mb + m - 1) / m), on = (ctas + sm_count - 1) / sm_count;
        cost[m] = (std::min(m, n_mb) + 0.15) * ((double)on + (on & 1 ? 0.5 : 0.0));
        if (m == kLinkBlocks || cost[m] < least) least = cost[m];
    }
    for (int m = kLinkBlocks; m > 1; m /= 2)
        if (m / 2 < n_mb && cost[m] <= 1.06 * least) return m;
    return 1;
}

}  // namespace ovl
