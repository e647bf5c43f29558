"""How many CTAs share a system (csrc/eph_share.h), for every size the ensemble launch takes and for devices that hold
clusters of up to 16, 8, 4, 2 CTAs or none: the choice is one the device holds, its shared memory fits, and it is
refused only where no size that the device holds fits."""
import os
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "eph_share.h"
using namespace eph;
int main() {
    for (unsigned shares : {31u, 30u, 28u, 24u, 16u})
        for (int mixed = 0; mixed < 2; ++mixed)
            for (int n = 1; n <= kMaxBodies; ++n) {
                const int split = batch_split(n), few = fewest_ctas(n, split, mixed, shares);
                std::printf("%u %d %d %d %d %d", shares, mixed, n, split, few, shortest_stage(n, split, mixed, shares));
                for (int g = few; g >= 0; g = more_ctas(n, split, mixed, shares, g)) std::printf(" %d", g);
                std::printf(" ;");
                for (int g = 0; g < kShares; ++g) std::printf(" %d", system_smem(n, kSharePeers[g], split, mixed) <= kBMaxSmem);
                std::printf("\n");
            }
}
"""


@pytest.fixture(scope="module")
def rows(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("share")
    src, exe = d / "share.cpp", d / "share"
    src.write_text(PROGRAM)
    csrc = os.path.join(ROOT, "ephemeris_b200", "csrc")
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", csrc, str(src), "-o", str(exe)], check=True)
    out = []
    for line in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.splitlines():
        head, fits = line.split(";")
        h = [int(x) for x in head.split()]
        out.append((h[0], h[1], h[2], h[3], h[4], h[5], h[6:], [int(x) for x in fits.split()]))
    return out


def test_choices_are_held_by_the_device(rows):
    for shares, mixed, n, split, few, short, chain, fits in rows:
        held = [g for g in range(5) if shares >> g & 1 and fits[g]]
        for g in chain + [g for g in (few, short) if g >= 0]:
            assert g in held, (shares, mixed, n)
        assert (few < 0) == (not held) == (short < 0), (shares, mixed, n)
        assert chain == sorted(chain, reverse=True) and len(set(chain)) == len(chain)
        assert few < 0 or (chain[0] == few and short in chain)


def test_every_size_fits_a_whole_device(rows):
    for shares, mixed, n, split, few, short, chain, fits in rows:
        if shares == 31:
            assert few >= 0 and short >= 0, (mixed, n)
        if shares == 16 and n <= 100:      # no clusters at all: small systems run on one CTA
            assert few == short == 4, (mixed, n)
