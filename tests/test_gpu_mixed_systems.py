"""A correction's three systems solved by one launch, of which some leave the passes for exact
sums (a zero tolerance, met when no cell moves any more) and the others end by the sweep
limit: FP64 against the oracle, split and FMA against the persistent ensemble step, whose
sums are always exact."""
import numpy as np
import pytest

import cases
import oracle as O

pytestmark = pytest.mark.gpu

LIMITS = range(3, 22)


def problem(maxiter):
    c = cases.case("vortex")
    c["nx"], c["ny"] = 57, 44
    return c, dict(g=c["g"], cfl=0.01, jacobi_tol=0.0, jacobi_maxiter=maxiter)


def mixed(iters, maxiter):
    """Some correction's systems ended on both sides of the limit."""
    groups = [iters[k:k + 3] for k in range(0, 12, 3)]
    return any(min(g) < maxiter == max(g) for g in groups)


def test_fp64_against_the_oracle(gpu):
    seen = 0
    for maxiter in LIMITS:
        c, kw = problem(maxiter)
        P = cases.cell_averages(c)
        o = O.Oracle(O.make_params(c["nx"], c["ny"], c["x0"], c["x1"], **kw))
        s = gpu.Solver(nx=c["nx"], ny=c["ny"], x0=c["x0"], x1=c["x1"], solver="stencil", **kw)
        o.set_planes(P)
        s.set_planes(P)
        for _ in range(2):
            dt = o.timestep()
            assert s.timestep() == dt
            o.step(0.0, dt)
            s.step(0.0, dt)
            assert np.array_equal(s.get_planes(), o.get_planes()), maxiter
            seen += mixed(s.stats()["jacobi_iters"], maxiter)
        s.close()
    assert seen > 0


@pytest.mark.parametrize("precision", ["split", "fp64_fma"])
def test_fast_forms_against_exact_sums(gpu, precision):
    seen = 0
    for maxiter in LIMITS:
        c, kw = problem(maxiter)
        P = cases.cell_averages(c)
        p = gpu.make_params(c["nx"], c["ny"], c["x0"], c["x1"], solver="stencil",
                            precision=precision, jacobi_block=4, **kw)
        s = gpu.Solver(p)
        b = gpu.Batch([p])
        b.set_launches(False)
        s.set_planes(P)
        b.set_planes(0, P)
        for _ in range(2):
            s.step(0.0, s.timestep())
            b.step()
            assert np.array_equal(s.get_planes(), b.get_planes(0)), maxiter
            iters = s.stats()["jacobi_iters"]
            assert iters == list(b.stats()[2][:, 0]), maxiter
            seen += mixed(iters, maxiter)
        s.close()
        b.close()
    assert seen > 0
