"""The rules that choose a launch from sizes (csrc/ovl_rules.h), evaluated
without a GPU: the header is compiled as plain C++."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "overlap_b200" / "csrc"
SMS = 148  # of a B200

SHIM = r"""
#include "ovl_rules.h"
extern "C" int link(int t, int n, int s) { return ovl::link_blocks(t, n, s); }
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
    ((8, 8, 8), 256, 2), ((8, 8, 8), 1024, 8), ((8, 8, 8), 2048, 4), ((8, 8, 8), 4096, 8), ((10, 13, 9), 512, 8)])
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
                return min(k, n) * (on + (0.5 if on % 2 else 0.0))

            # the gathering counts for 0.15 of a block per CTA: at most 15 % between two choices
            assert load(m) <= 1.06 * 1.15 * min(load(k) for k in (1, 2, 4, 8)) + 1e-9, (sites, n, m)
