"""The exact Patankar assembly's division paths against the oracle, bit for bit: depths so
small that fluxes and weights leave the range of the branch-free division, beside ordinary
cells, for every assembly the step uses (three substeps at once, single substeps, the
two-substep scheme; CSR and stencil layouts)."""
import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", ["csr", "stencil"])
@pytest.mark.parametrize("timescheme", [5, 7])
@pytest.mark.parametrize("depth", [1e-150, 1e-125, 1e-30])
def test_tiny_depths(gpu, solver, timescheme, depth):
    nx, ny = 41, 36
    c = cases.case("vortex")
    c["nx"], c["ny"] = nx, ny
    P = cases.cell_averages(c)
    P[0, 10:20, 12:30] = depth
    P[1:, 10:20, 12:30] = 0.0
    kw = dict(g=c["g"], cfl=c["cfl"], timescheme=timescheme)
    o = O.Oracle(O.make_params(nx, ny, c["x0"], c["x1"], **kw))
    s = gpu.Solver(nx=nx, ny=ny, x0=c["x0"], x1=c["x1"], solver=solver, **kw)
    o.set_planes(P)
    s.set_planes(P)
    dt = o.timestep()
    assert s.timestep() == dt
    o.step(0.0, dt)
    ref = o.get_planes()
    if np.isfinite(ref).all():
        assert s.step(0.0, dt) == 0
    else:  # the reference's own step leaves the finite range: reported, the bits the same
        with pytest.raises(gpu.SwmError) as e:
            s.step(0.0, dt)
        assert e.value.code == -3
    assert np.array_equal(s.get_planes(), ref, equal_nan=True)
    assert s.stats()["jacobi_iters"] == o.last_jacobi_iters()
