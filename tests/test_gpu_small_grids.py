"""The RHS of small grids (8 x 8 tiles; several states in one launch) against the oracle and
against the ensemble's 16 x 16 tiles, at the edges of both tile sizes and of the dispatch."""
import numpy as np
import pytest

import cases
import oracle as O
from test_gpu_parity import make_pair

pytestmark = pytest.mark.gpu

# 64 tiles of 16 x 16 is the small-tile limit: 3 states of 21 tiles take 8 x 8, of 22 not
SIZES = [(3, 3), (8, 8), (9, 7), (16, 17), (33, 25), (48, 112), (112, 49), (64, 88), (112, 65)]


@pytest.mark.parametrize("nx,ny", SIZES)
@pytest.mark.parametrize("timescheme", [5, 7, 2])
def test_fp64_bitwise(gpu, nx, ny, timescheme):
    c = cases.case("lake")  # bathymetry, no well-balanced reference
    c["nx"], c["ny"] = nx, ny
    kw = dict(g=c["g"], cfl=c["cfl"], bathy_flag=3, bathy_par=c["bathy_par"], timescheme=timescheme)
    o = O.Oracle(O.make_params(nx, ny, c["x0"], c["x1"], **kw))
    s = gpu.Solver(nx=nx, ny=ny, x0=c["x0"], x1=c["x1"], **kw)
    P = cases.cell_averages(c)
    o.set_planes(P)
    s.set_planes(P)
    for _ in range(2):
        dt = o.timestep()
        assert s.timestep() == dt
        o.step(0.0, dt)
        s.step(0.0, dt)
    assert np.array_equal(s.get_planes(), o.get_planes())


@pytest.mark.parametrize("n", [32, 48])
def test_well_balanced_lake_bitwise(gpu, n):
    c, o, s = make_pair(gpu, "lake_dry", n)
    for _ in range(2):
        dt = o.timestep()
        assert s.timestep() == dt
        o.step(0.0, dt)
        s.step(0.0, dt)
    assert np.array_equal(s.get_planes(), o.get_planes())


@pytest.mark.parametrize("precision", ["split", "fp64_fma"])
@pytest.mark.parametrize("nx,ny", SIZES)
def test_same_as_the_ensembles_tiles(gpu, nx, ny, precision):
    c = cases.case("dambreak")
    c["nx"], c["ny"] = nx, ny
    kw = dict(nx=nx, ny=ny, x0=c["x0"], x1=c["x1"], g=c["g"], cfl=c["cfl"], precision=precision,
              solver="stencil", jacobi_block=4)
    P = cases.cell_averages(c)
    s = gpu.Solver(**kw)
    b = gpu.Batch([gpu.make_params(**kw)])
    s.set_planes(P)
    b.set_planes(0, P)
    for _ in range(2):
        dt = s.timestep()
        try:
            s.step(0.0, dt)
        except gpu.SwmError as e:  # a dam break on so few cells can leave the finite range
            assert e.code == -3
        dts, _ = b.step()
        assert dts[0] == dt
        if not np.isfinite(b.get_planes(0)).all():
            break
    assert np.array_equal(s.get_planes(), b.get_planes(0), equal_nan=True)
    s.close()
    b.close()
