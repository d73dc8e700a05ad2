"""Which RHS launches form the quotients of the mass fluxes (fluxes_over_len,
sw-mpdec_b200/csrc/swm_rules.h, built by the host compiler): those whose quotients an assembly
reads.  The explicit time schemes (1 to 4) have no assembly."""
import ctypes
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "sw-mpdec_b200", "csrc")


def test_only_the_exact_assembly_takes_quotients(tmp_path):
    src, so = str(tmp_path / "flux.cpp"), str(tmp_path / "flux.so")
    with open(src, "w") as f:
        f.write("""#include "swm_rules.h"
extern "C" int over(int t, int fast) { return swm::fluxes_over_len(t, fast != 0); }
""")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "-shared", "-fPIC", src, "-o", so],
                   check=True)
    over = ctypes.CDLL(so).over
    assert [over(t, 0) for t in range(1, 8)] == [0, 0, 0, 0, 1, 1, 1]
    assert [over(t, 1) for t in range(1, 8)] == [0] * 7
