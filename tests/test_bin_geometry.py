"""Room of the bins of a binned insert, against the exact share of the 32-bit hashes that each bin gets (CPU)."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "cuckoo-filter_b200")

SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "cf_binned.cuh"
using namespace cfb;
int main(int argc, char** argv) {
    const uint32_t policy = atoi(argv[1]);
    for (int a = 2; a + 1 < argc; a += 2) {
        const uint64_t nb = strtoull(argv[a], nullptr, 10), m = strtoull(argv[a + 1], nullptr, 10);
        BinGeom g{};
        if (!bin_geometry(nb, 32, 16, policy, m, &g)) return printf("%llu: no geometry\n", (unsigned long long)nb), 1;
        // hashes of buckets [0, x): bucket b is hash % range, so the first 2^32 % range have one more
        const uint64_t range = policy == ALT_ADDSUB ? nb / 2 : nb;
        auto below = [&](uint64_t x) {
            x = std::min<uint64_t>(x, range);
            return x * ((1ull << 32) / range) + std::min<uint64_t>(x, (1ull << 32) % range);
        };
        double over = 0;  // keys expected past the room of their bin
        auto bins = [&](int log2_buckets, uint64_t room) {
            for (uint64_t b = 0; b < range; b += 1ull << log2_buckets) {
                const double mean = static_cast<double>(m) * (below(b + (1ull << log2_buckets)) - below(b)) / 4294967296.0;
                if (mean + 5.0 * std::sqrt(mean) > room) over += std::max(0.0, mean - static_cast<double>(room)) + std::sqrt(mean);
            }
        };
        bins(g.sbl, g.room2);
        if (g.l2) bins(g.sbl + g.l2, g.room1);
        const double bytes = (g.ent[0] + g.ent[1]) / (2.0 * m);
        printf("%llu buckets, %llu keys: %.0f over, %.3f entries of room per key\n", (unsigned long long)nb,
               (unsigned long long)m, over, bytes);
        if (over > 0) return 1;
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(cfb, tmp_path_factory):
    sys.path.insert(0, PKG)
    import build

    d = tmp_path_factory.mktemp("geometry")
    (d / "rooms.cu").write_text(SRC)
    r = subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I" + os.path.join(PKG, "csrc"), str(d / "rooms.cu"), "-o",
                        str(d / "rooms")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return str(d / "rooms")


@pytest.mark.parametrize("policy,slots", [
    (0, [1 << 14, 1 << 20, 1 << 26, 1 << 31]),
    (1, [100, 1_000_003, 200_000_000, 1_000_000_000, 1_300_000_000, 2_100_000_000, 2_147_483_000]),
    (2, [100, 777_777, 100_000_000, 1_000_000_000, 1_300_000_000, 2_100_000_000, 2_147_483_647]),
])
@pytest.mark.parametrize("load", [0.3, 0.95])
def test_hashed_keys_fit_their_bins(program, policy, slots, load):
    """Every bin's mean plus five standard deviations is within its room, where the
    bucket is a hash modulo a count that is no power of two too."""
    args = []
    for n in slots:
        nb = -(-n // 16)
        nb += policy == 1 and nb % 2
        args += [str(nb), str(int(load * n))]
    r = subprocess.run([program, str(policy), *args], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
