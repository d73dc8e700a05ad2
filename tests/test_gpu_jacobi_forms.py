"""The Jacobi kernel's forms (tiles, strips, one-sweep exact passes) against the oracle,
bit for bit, where they can go wrong: the edges of tiles (56 x 40 and 48 x 32 cells) and
strips (56 columns), grids smaller than a warp's halo, odd widths, and operands that the fast
division does not take."""
import numpy as np
import pytest

import oracle as O
from test_gpu_parity import random_patankar_system

pytestmark = pytest.mark.gpu


def pair(gpu, nx, ny, solver, block=0, tol=1e-16, maxiter=1000):
    o = O.Oracle(O.make_params(nx, ny, (0.0, 0.0), (1.0, 1.0), jacobi_tol=tol,
                               jacobi_maxiter=maxiter))
    s = gpu.Solver(nx=nx, ny=ny, x0=(0.0, 0.0), x1=(1.0, 1.0), solver=solver, jacobi_block=block,
                   jacobi_tol=tol, jacobi_maxiter=maxiter)
    return o, s


def check(o, s, mass, diag, rhs):
    ref, k_ref = o.jacobi(mass, diag, rhs)
    got, k, rc = s.debug_jacobi(mass, diag, rhs)
    assert k == k_ref
    assert np.array_equal(got, ref, equal_nan=True)
    return k, rc


# 48 x 32 tiles up to 148 of them, 56 x 40 at 700 x 420 (135; 210 of 48 x 32), three rounds of
# 48 x 32 at 1000 x 620, strips at 1100 x 1003
@pytest.mark.parametrize("nx,ny", [(3, 3), (5, 90), (48, 32), (49, 33), (64, 48), (97, 65),
                                   (224, 81), (700, 420), (701, 401), (1000, 620),
                                   (1100, 1003), (1101, 1000)])
@pytest.mark.parametrize("solver,block", [("stencil", 0), ("stencil", 3), ("csr", 0)])
def test_shapes(gpu, nx, ny, solver, block):
    o, s = pair(gpu, nx, ny, solver, block)
    check(o, s, *random_patankar_system(nx * ny, nx + ny))


@pytest.mark.parametrize("nx,ny", [(70, 61), (1100, 1003)])
@pytest.mark.parametrize("solver", ["stencil", "csr"])
def test_operands_outside_the_fast_division(gpu, nx, ny, solver):
    n = nx * ny
    o, s = pair(gpu, nx, ny, solver, maxiter=40)
    mass, diag, rhs = random_patankar_system(n, 5)
    zeros = rhs.copy()
    zeros[:: 7] = 0.0
    check(o, s, mass, diag, zeros)
    tiny = np.where(np.arange(n) % 11 == 0, 1e-150, rhs)  # below 2^-400, alone in its row
    alone = mass.reshape(n, 5).copy()
    alone[np.arange(n) % 11 == 0] = 0.0
    check(o, s, alone.reshape(-1), diag, tiny)
    big = diag.copy()
    big[n // 2] = 1e200
    check(o, s, mass, big, rhs)
    if solver == "csr":
        centre = mass.reshape(n, 5).copy()
        centre[n // 3, 2] = -0.25
        check(o, s, centre.reshape(-1), diag, rhs)


@pytest.mark.parametrize("solver", ["stencil", "csr"])
def test_zero_tolerance_takes_exact_sums(gpu, solver):
    # stops when every |dx| is below 2^-101: the last sweeps' sums are inside the band
    # where only the exact sum decides
    o, s = pair(gpu, 60, 50, solver, tol=0.0, maxiter=200)
    mass, diag, rhs = random_patankar_system(3000, 11)
    check(o, s, 0.1 * mass, diag, rhs)


def test_zero_right_hand_side(gpu):
    o, s = pair(gpu, 60, 50, "stencil")
    mass, diag, rhs = random_patankar_system(3000, 2)
    k, rc = check(o, s, mass, diag, 0.0 * rhs)
    assert k == 0 and rc == 0
