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
// odd last CTA of several blocks has the SM to itself and takes longer than its
// share, counted as half a CTA more.  The largest m within 6 % of the least such
// time: where the times are equal fewer, longer CTAs gather less.
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
//         16^3 x 64           49/39 49/39 50/39 [47/38]
//   FP40  12^3 x 256          70/45 58/46 [62/50] 58/52
//         12^3 x 512         129/88 [111/90] 115/98 115/100
// One CTA per SM as the only condition is best for contexts in turn and up to 26 %
// slower for one on its own (17 % at 12^3 x 512: m = 8); four CTAs per SM is up to 20 %
// slower in turn (9 % at 8^3 x 1024: m = 2).  Over 102 launches of 6^3 to 16^3 sites and
// 64 to 4096 modes, geometric means of the time alone against four CTAs per SM and of
// the time in turn against one: this rule 1.00 and 1.01, one CTA per SM 1.03 and 1, four
// 1 and 1.03; the larger of the two losses is 1.7 % in the mean (1.2 % for the best m
// of every launch), 4.0 % and 3.6 %.
inline int link_blocks(int site_ctas, int n_mb, int sm_count) {
    double cost[kLinkBlocks + 1], least = 0.0;
    for (int m = kLinkBlocks; m >= 1; m /= 2) {
        const long long ctas = (long long)site_ctas * ((n_mb + m - 1) / m), on = (ctas + sm_count - 1) / sm_count;
        cost[m] = (std::min(m, n_mb) + 0.15) * ((double)on + (m > 1 && (on & 1) ? 0.5 : 0.0));
        if (m == kLinkBlocks || cost[m] < least) least = cost[m];
    }
    for (int m = kLinkBlocks; m > 1; m /= 2)
        if (m / 2 < n_mb && cost[m] <= 1.06 * least) return m;
    return 1;
}

// ------------------------------------ the Chebyshev overlap operator on chip --
// How ovl_resident.cuh lays a lattice out: a cluster of `ranks` CTAs with `planes`
// z planes each (the last CTA may hold fewer), `groups` sets of modes per cluster; a CTA
// has groups x sites threads.
struct ResidentShape {
    int planes, groups, ranks;
};

constexpr int kResMaxRanks = 8;  // the portable cluster size

// A call: colours, FP64 or FP32, the lattice, the sets of modes (modes / modes per
// thread), the degree of the series.
struct ResidentCall {
    int nc;
    bool f64;
    int N0, N1, N2, slots, degree;
};

// The time of the operator on chip, in us: clusters at a time on the GPU's sms
// SMs, waves of them, degree + 4 terms each (the links and phi laid out first and the
// combination at the end take as long as four).  A term of two phases takes a
// barrier of the CTA or the cluster and a time per thread on the SM, and more where
// every CTA hands its outer planes on, where the rows of a plane do not fill 8 lanes
// (bank conflicts where they wrap), where no two threads share the reads of a link,
// and with more than 512 threads of three colours (96 registers, spilling).
// Fitted to 7829 timings (51 pairs of lattice and storage, 4 to 32 sites a side, 32 to
// 4096 modes, degrees 24 and 96): 5 to 8 % rms, 9 to 16 % at the 95th percentile.
inline double resident_term_us(const ResidentCall &c, const ResidentShape &sh, int cap, long long ctas_per_sm) {
    struct Times { double one, one_thread, many, many_thread; };  // us per term: one CTA, several
    const Times t = c.nc == 2 ? (c.f64 ? Times{0.40, 0.0100, 1.52, 0.0088} : Times{0.50, 0.0089, 1.87, 0.0085})
                              : (c.f64 ? Times{0.95, 0.0178, 2.47, 0.0151} : Times{1.12, 0.0088, 2.38, 0.0077});
    const double threads = (double)c.N0 * c.N1 * sh.planes * sh.groups * ctas_per_sm;
    double term = sh.ranks == 1 ? t.one + t.one_thread * threads
                                : (t.many + t.many_thread * threads) * (1.0 + 0.12 / sh.planes);
    if ((c.N0 * sh.groups) % 8 != 0) term *= 1.11;
    if (sh.groups == 1) term *= 1.09;
    if (c.nc == 3 && cap > 512) term *= 1.14;
    return term;
}
inline double resident_us(const ResidentCall &c, const ResidentShape &sh, int cap, int clusters, int sms) {
    const long long need = (c.slots + sh.groups - 1) / sh.groups, waves = (need + clusters - 1) / clusters;
    const long long ctas_per_sm = (std::min<long long>(need, clusters) * sh.ranks + sms - 1) / sms;
    return (double)waves * (c.degree + 4) * resident_term_us(c, sh, cap, ctas_per_sm);
}

// The time of the kernels that go through memory, in us: two launches a term, no
// faster than 12.3 us, that move seven fields at the rate they reach beyond L2.
inline double through_memory_us(const ResidentCall &c, double field_bytes) {
    const double rate = c.f64 ? 4.9e6 : 5.2e6;  // bytes per us
    return (c.degree + 0.6) * std::max(12.3, 3.5 + 7.0 * field_bytes / rate);
}

// The best shape for CTAs of `cap` threads, if it takes less than `best` us: then
// shape and best are set.  fits(shape) is the number of clusters that run at a time
// (0: it does not fit; never more than two CTAs per SM), asked only where the
// answer could matter.
template <class Fits>
inline bool resident_choose(const ResidentCall &c, int cap, int sms, const Fits &fits, ResidentShape &shape, double &best) {
    bool found = false;
    for (int ranks = 1; ranks <= std::min(kResMaxRanks, c.N2); ranks++) {
        const int planes = (c.N2 + ranks - 1) / ranks;
        const long long sites = (long long)c.N0 * c.N1 * planes;
        if ((c.N2 + planes - 1) / planes != ranks || sites > cap) continue;
        for (int groups = 1; groups <= std::min<long long>(cap / sites, c.slots); groups++) {
            const ResidentShape sh{planes, groups, ranks};
            // no less than this, two CTAs per SM that do not slow each other
            const int most = std::max(1, 2 * sms / ranks), need = (c.slots + groups - 1) / groups;
            if ((double)((need + most - 1) / most) * (c.degree + 4) * resident_term_us(c, sh, cap, 1) >= best) continue;
            const int clusters = fits(sh);
            if (clusters < 1) continue;
            const double us = resident_us(c, sh, cap, clusters, sms);
            if (us >= best) continue;
            best = us;
            shape = sh;
            found = true;
        }
    }
    return found;
}

}  // namespace ovl
