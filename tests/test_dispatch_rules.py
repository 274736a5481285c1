"""The rules that choose a launch from sizes (csrc/ovl_rules.h), evaluated
without a GPU: the header is compiled as plain C++."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "overlap_b200" / "csrc"
SMS = 148  # of a B200
# clusters of 1 to 8 CTAs that run at a time with one CTA per SM
# (cudaOccupancyMaxActiveClusters on that GPU)
CLUSTERS = (0, 148, 74, 45, 33, 26, 22, 15, 15)

SHIM = r"""
#include "ovl_rules.h"
extern "C" int link(int t, int n, int s) { return ovl::link_blocks(t, n, s); }
// out: planes, groups, ranks; us: the time of the choice, and through memory
extern "C" int chip(int nc, int f64, const int *N, int slots, int degree, int cap, double field_bytes, int sms,
                    const int *clusters, int *out, double *us) {
    const ovl::ResidentCall c{nc, f64 != 0, N[0], N[1], N[2], slots, degree};
    ovl::ResidentShape sh{0, 0, 0};
    us[0] = us[1] = ovl::through_memory_us(c, field_bytes);
    const bool ok = ovl::resident_choose(c, cap, sms, [&](const ovl::ResidentShape &s) { return clusters[s.ranks]; }, sh, us[0]);
    out[0] = sh.planes;
    out[1] = sh.groups;
    out[2] = sh.ranks;
    return ok;
}
extern "C" double chip_us(int nc, int f64, const int *N, int slots, int degree, int cap, int planes, int groups, int ranks,
                          int sms, const int *clusters) {
    return ovl::resident_us(ovl::ResidentCall{nc, f64 != 0, N[0], N[1], N[2], slots, degree}, {planes, groups, ranks}, cap,
                            clusters[ranks], sms);
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "rules.cpp"), "-o",
                    str(d / "rules.so")], check=True)
    return C.CDLL(str(d / "rules.so"))


# (site CTAs of 8 sites, mode blocks): what the measurements beside the rule give, for a
# context on its own as well as for several in turn
@pytest.mark.parametrize("N,modes,m", [
    ((12, 12, 12), 128, 1), ((12, 12, 12), 256, 2), ((12, 12, 12), 512, 4), ((6, 6, 6), 1024, 1), ((6, 6, 6), 4096, 4),
    ((8, 8, 8), 256, 2), ((8, 8, 8), 1024, 8), ((8, 8, 8), 2048, 4), ((8, 8, 8), 4096, 8), ((10, 13, 9), 512, 8),
    ((16, 16, 16), 64, 1), ((13, 11, 12), 96, 1)])
def test_mode_blocks_per_cta_of_the_link_table_stencils(rules, N, modes, m):
    sites = (N[0] * N[1] * N[2] + 7) // 8
    assert rules.link(sites, modes // 32, SMS) == m


def test_mode_blocks_per_cta_over_all_sizes(rules):
    """A power of two up to 8, never twice the blocks there are, and in every
    launch the fullest SM's blocks stay within the rule's margin of the least."""
    for sites in list(range(4, 600, 7)) + [1 << 20, (1 << 30) // 64]:
        for n in (1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 31, 64, 65, 500, 65535):
            m = rules.link(sites, n, SMS)
            assert m in (1, 2, 4, 8) and (m == 1 or m // 2 < n), (sites, n, m)

            def load(k):
                on = -(-sites * -(-n // k) // SMS)
                return min(k, n) * (on + (0.5 if k > 1 and on % 2 else 0.0))

            # the gathering counts for 0.15 of a block per CTA: at most 15 % between two choices
            assert load(m) <= 1.06 * 1.15 * min(load(k) for k in (1, 2, 4, 8)) + 1e-9, (sites, n, m)


def chip(rules, nc, f64, N, modes, degree):
    """(shape or None, us, us through memory) of the two-colour FP32 (pairs of modes), FP64
    and three-colour capacities."""
    padded = -(-modes // 32) * 32
    per_thread = 2 if nc == 2 and not f64 else 1
    cap = {(2, 0): 512, (2, 1): 384, (3, 0): 512, (3, 1): 256}[nc, f64]
    field = N[0] * N[1] * N[2] * padded * nc * 4 * (16 if f64 else 8)
    out, us = (C.c_int * 3)(), (C.c_double * 2)()
    ok = rules.chip(nc, f64, (C.c_int * 3)(*N), padded // per_thread, degree, cap, C.c_double(field), SMS,
                    (C.c_int * 9)(*CLUSTERS), out, us)
    return tuple(out) if ok else None, us[0], us[1], padded // per_thread, cap


# The best of all shapes and memory by measurement (planes, sets of modes, CTAs; None: memory).
# Shared memory does not limit these.
@pytest.mark.parametrize("nc,f64,N,modes,degree,shape", [
    (2, 0, (5, 5, 5), 64, 24, (5, 1, 1)), (2, 0, (8, 8, 8), 32, 24, (1, 2, 8)), (2, 0, (8, 8, 8), 256, 24, (8, 1, 1)),
    (2, 0, (8, 8, 8), 4096, 64, (8, 1, 1)), (2, 0, (7, 6, 13), 32, 24, (3, 1, 5)), (2, 0, (16, 16, 16), 1024, 96, (2, 1, 8)),
    (2, 0, (12, 11, 10), 2048, 24, None), (2, 0, (14, 14, 14), 1024, 24, None), (2, 1, (4, 4, 4), 128, 24, (4, 1, 1)),
    (2, 1, (8, 8, 8), 64, 24, (2, 2, 4)), (3, 0, (4, 4, 4), 32, 24, (4, 1, 1)), (3, 0, (8, 8, 8), 64, 24, (2, 2, 4)),
    (3, 1, (7, 7, 7), 4096, 24, None)])
def test_chebyshev_on_chip_choice(rules, nc, f64, N, modes, degree, shape):
    assert chip(rules, nc, f64, N, modes, degree)[0] == shape


def test_chebyshev_on_chip_choice_over_all_sizes(rules):
    """The shape holds the lattice, and no other takes less time by the rule."""
    for nc in (2, 3):
        for f64 in (0, 1):
            for N in ((3, 3, 3), (4, 6, 5), (5, 5, 5), (9, 5, 11), (8, 8, 8), (10, 10, 10), (12, 12, 12), (16, 16, 16),
                      (3, 3, 40), (31, 16, 3), (40, 3, 3)):
                for modes in (1, 33, 96, 256, 1000, 4096):
                    for degree in (1, 24, 96):
                        sh, us, mem, slots, cap = chip(rules, nc, f64, N, modes, degree)
                        best = mem
                        for ranks in range(1, 9):
                            planes = -(-N[2] // ranks)
                            sites = N[0] * N[1] * planes
                            if -(-N[2] // planes) != ranks:
                                continue
                            for g in range(1, min(cap // sites, slots) + 1):
                                rules.chip_us.restype = C.c_double
                                best = min(best, rules.chip_us(nc, f64, (C.c_int * 3)(*N), slots, degree, cap, planes, g, ranks,
                                                               SMS, (C.c_int * 9)(*CLUSTERS)))
                        assert us == pytest.approx(best, rel=1e-12), (nc, f64, N, modes, degree)
                        assert (sh is None) == (us == mem)
                        if sh:
                            planes, g, ranks = sh
                            assert planes * (ranks - 1) < N[2] <= planes * ranks and N[0] * N[1] * planes * g <= cap
                            assert 1 <= g <= slots and 1 <= ranks <= 8
