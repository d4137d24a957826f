"""Helpers of the kernels that also compile for the host, run here on the CPU with
inputs that a GPU run should never see: values that are not numbers, pair counts
next to 2^31."""

import os
import subprocess

import numpy as np
import pytest

from muspinsim_gb300 import build

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "msp_cluster.cuh"
#include "msp_internal.cuh"
using namespace msp;

// nan-max: the values from stdin; sort: n levels, their ranks; item: slots, P, IP,
// their prefixes, the item
int main(int argc, char **argv) {
    const char kind = argv[1][0];
    if (kind == 'm') {
        float m = 0.f, x;
        while (std::scanf("%f", &x) == 1) m = max_or_nan(m, x);
        std::printf("%g\n", m);
    } else if (kind == 's') {
        double lam[64];
        int n = 0;
        while (n < 64 && std::scanf("%lf", &lam[n]) == 1) ++n;
        for (int i = 0; i < n; ++i) std::printf("%d ", level_rank(lam, n, i));
    } else {
        PhaseArgs a = {};
        int slot_first[8], item_first[8];
        if (std::scanf("%d %d %d", &a.num_slots, &a.P, &a.IP) != 3) return 1;
        for (int i = 0; i <= a.num_slots; ++i)
            if (std::scanf("%d %d", &slot_first[i], &item_first[i]) != 2) return 1;
        a.slot_first = slot_first;
        a.item_first = item_first;
        int item, b, e;
        while (std::scanf("%d", &item) == 1) {
            phase_item_range(a, item, &b, &e);
            std::printf("%d %d ", b, e);
        }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def helper(tmp_path_factory):
    d = tmp_path_factory.mktemp("host")
    src, exe = str(d / "h.cu"), str(d / "h")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build.nvcc_path(), *build.ARCH, "-std=c++17", "-I", build.CSRC, "-I",
                    os.path.join(os.path.dirname(build.HERE), "include"), "-o", exe, src], check=True,
                   capture_output=True, text=True)

    def run(kind, values):
        out = subprocess.run([exe, kind], input=" ".join(str(v) for v in values), check=True,
                             capture_output=True, text=True).stdout
        return out.split()

    return run


@pytest.mark.parametrize("at", [0, 1, 4])
def test_largest_keeps_a_nan(helper, at):
    values = [1.0, 5.0, 2.0, 0.0, 3.0]
    assert float(helper("m", values)[0]) == 5.0
    values[at] = "nan"
    assert np.isnan(float(helper("m", values)[0]))


@pytest.mark.parametrize("levels", [[3.0, -1.0, 2.0, 2.0, -0.0, 0.0], ["nan"] * 5,
                                    [1.0, "nan", -2.0, "-nan", "inf", "-inf", 1.0, 0.5]])
def test_ranks_are_a_permutation(helper, levels):
    ranks = [int(r) for r in helper("s", levels)]
    assert sorted(ranks) == list(range(len(levels)))
    x = np.array(levels, dtype=float)
    ok = [i for i in range(len(x)) if not np.isnan(x[i])]
    assert sorted(ok, key=lambda i: ranks[i]) == sorted(ok, key=lambda i: (x[i], np.signbit(x[i]) == 0, i))


def test_item_ranges_next_to_the_largest_pair_count(helper):
    """One row of 7,780,000 snapshots of n = 24 (2^31 - 203,648 pairs), in items of 2^30."""
    S, P, IP = 7780000, 276, 1 << 30
    got = [int(v) for v in helper("i", [1, P, IP, 0, 0, S, 2, 0, 1, 2])]
    assert got == [0, IP, IP, S * P, -1, -1]
