"""Which schedule the ensemble's first step keeps (fastest_schedule,
sw-mpdec_b200/csrc/swm_rules.h), built by the host compiler and called with given times."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sw-mpdec_b200", "csrc")

SOURCE = r"""
#include "swm_rules.h"
extern "C" int keep(int n, const int* form, const float* ms, int* tried) {
  return swm::fastest_schedule(
      n, [&](int i) { return form[i]; },
      [&](int i) { tried[i] = 1; return ms[i]; });
}
"""


@pytest.fixture(scope="module")
def keep(tmp_path_factory):
    d = tmp_path_factory.mktemp("schedule")
    src, so = str(d / "schedule.cpp"), str(d / "schedule.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "-shared", "-fPIC", src, "-o", so],
                   check=True)
    lib = ctypes.CDLL(so)

    def call(schedules):
        n = len(schedules)
        tried = (ctypes.c_int * n)()
        k = lib.keep(n, (ctypes.c_int * n)(*[f for f, _ in schedules]),
                     (ctypes.c_float * n)(*[t for _, t in schedules]), tried)
        return k, list(tried)

    return call


def test_a_slow_later_schedule_hides_none_of_its_form(keep):
    # one form only (chosen by the caller): half the grid is slow, longer passes are best
    k, tried = keep([(1, 10.0), (1, 14.0), (1, 9.5), (1, 13.0), (1, 8.0), (1, 12.0)])
    assert k == 4 and all(tried)
    # both forms, the second near the first with its first schedule
    k, tried = keep([(0, 10.0), (0, 13.0), (1, 11.0), (1, 15.0), (1, 9.0)])
    assert k == 4 and all(tried)


def test_a_form_far_behind_is_tried_once(keep):
    k, tried = keep([(0, 37.0), (0, 40.0), (1, 60.0), (1, 1.0), (1, 57.0)])
    assert k == 0 and tried == [1, 1, 1, 0, 0]


def test_a_failed_trial_ends_the_search(keep):
    k, tried = keep([(0, 10.0), (0, -1.0), (1, 5.0)])
    assert k == -1 and tried == [1, 1, 0]
