"""The passes' stop decision on FP64 sums (stop_decision, sw-mpdec_b200/csrc/swm_rules.h, built
by the host compiler) against the exact rule: whatever the order of the terms, outside the
band both agree, and inside it the decision is left to exact sums."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sw-mpdec_b200", "csrc")

SOURCE = r"""
#include "swm_rules.h"
extern "C" {
int decide(double s, double thresh, double n) { return swm::stop_decision(s, thresh, n); }
double band() { return swm::kBand; }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("band")
    src, so = str(d / "band.cpp"), str(d / "band.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-shared",
                    "-fPIC", src, "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.decide.argtypes = [ctypes.c_double] * 3
    lib.band.restype = ctypes.c_double
    return lib


def limbs(v):
    """floor(v 2^100), saturated from 2^20 on (NaN too)."""
    return int(math.ldexp(v, 100)) if v < 2.0 ** 20 else (1 << 120) - 1


def sums(vals, rng):
    """FP64 sums of the terms in a few orders and groupings."""
    yield float(np.cumsum(vals)[-1])
    yield float(np.cumsum(vals[::-1])[-1])
    p = rng.permutation(vals)
    yield float(np.cumsum(p)[-1])
    k = int(rng.integers(1, 65))
    yield float(np.cumsum([np.cumsum(p[i::k])[-1] for i in range(min(k, len(p)))])[-1])


@pytest.mark.parametrize("tol", [1e-16, 1e-9, 3e-29, 1e-32, 0.0])
def test_decisions_are_the_exact_rule_s(lib, tol):
    rng = np.random.default_rng(int(1e6 * abs(math.log(tol or 1e-40))))
    band = lib.band()
    outside, inside = 0, 0
    for trial in range(400):
        n = int(rng.integers(2, 3000))
        goal = tol * n
        thresh = limbs(goal)
        vals = 10.0 ** rng.uniform(-3, 0, n)
        # exact sums from far outside the band to its middle, on both sides, or (where the
        # truncation is not small beside the threshold) a few truncations away
        at = goal * (1.0 + rng.choice([-1, 1]) * band * 2.0 ** rng.uniform(-8, 8))
        at += rng.choice([-1, 0, 1]) * rng.uniform(0, 4) * n * 2.0 ** -100
        vals = vals * (max(at, 0.0) / math.fsum(vals))
        exact = sum(limbs(float(v)) for v in vals) <= thresh
        for s in sums(vals, rng):
            d = lib.decide(s, math.ldexp(thresh, -100), float(n))
            if d < 0:
                inside += 1
            else:
                outside += 1
                assert (d == 1) == exact, (n, s, goal)
    assert inside > 100
    assert outside > 100


def test_both_edges_of_the_band(lib):
    n, thresh = 2.0 ** 20, 2.0 ** -33
    lo, hi = thresh * (1.0 - lib.band()), thresh * (1.0 + lib.band())
    slack = n * 2.0 ** -100
    for s, want in ((0.0, 1), (lo - 2 * slack, 1), (lo + slack, -1), (thresh, -1), (hi, -1),
                    (hi + 2 * slack + math.ulp(hi), 0), (1.0, 0), (math.inf, 0), (math.nan, 0)):
        assert lib.decide(s, thresh, n) == want, s
    assert lib.decide(0.0, 0.0, n) == -1  # a zero threshold: never by the FP64 sum alone


def test_unusable_sums_go_on(lib):
    for bad in (math.nan, math.inf, 2.0 ** 1000, 2.0 ** 21):
        assert lib.decide(bad, 2.0 ** -33, 100.0) == 0
        assert limbs(bad if bad == bad else 2.0 ** 21) > limbs(2.0 ** -33)
