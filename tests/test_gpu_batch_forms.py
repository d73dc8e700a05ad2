"""Ensembles: what the two step forms report."""
import pytest

import cases

pytestmark = pytest.mark.gpu

def test_sweeps_per_pass_of_the_form_in_use(gpu):
    # the per-phase form solves by strips, which sweep at most four times per pass
    c = cases.case("vortex", n=40)
    for block, phased in ((1, 1), (2, 2), (4, 4), (8, 4)):
        b = gpu.Batch([gpu.make_params(c["nx"], c["ny"], c["x0"], c["x1"], solver="stencil",
                                       jacobi_block=block)])
        b.set_planes(0, cases.cell_averages(c))
        for per_phase, sweeps in ((True, phased), (False, block)):
            b.set_launches(per_phase)
            b.step()
            assert b.stats()[0] == sweeps
        b.close()
