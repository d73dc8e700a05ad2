"""The solvers' control rules (sw-mpdec_b200/csrc/swm_rules.h), built by the host compiler
and called from here."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sw-mpdec_b200", "csrc")

SOURCE = r"""
#include "swm_rules.h"
extern "C" {
int barrier_open(unsigned c, unsigned t) { return swm::barrier_open(c, t); }
int ring_at(int pos, int steps, int n) { return swm::ring_at(pos, steps, n); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    src, so = str(d / "rules.cpp"), str(d / "rules.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-shared",
                    "-fPIC", src, "-o", so], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("blocks", [1, 2, 148, 444, 1184])
def test_barrier_opens_at_the_last_arrival_also_past_2_to_32(lib, blocks):
    # uses around the first and around the one whose target passes 2^32 (and twice that)
    wrap = 2 ** 32 // blocks
    for nth in [1, 2, 3, *range(wrap - 2, wrap + 4), 2 * wrap, 2 * wrap + 1]:
        target = nth * blocks
        for arrived in range(target - blocks, target + blocks):  # true count of arrivals
            got = lib.barrier_open(ctypes.c_uint(arrived % 2 ** 32),
                                   ctypes.c_uint(target % 2 ** 32))
            assert bool(got) == (arrived >= target), (nth, arrived - target)


def test_ring_positions_stay_in_the_ring(lib):
    for n in (3, 4):
        for pos in range(n):
            for steps in range(n + 1):
                assert lib.ring_at(pos, steps, n) == (pos + steps) % n
