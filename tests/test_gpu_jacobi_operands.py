"""Operands that the Jacobi's fast divisions do not take cost their system IEEE divisions in
passes of the same length, not the one-sweep exact passes; a Diagonal whose low word is all
ones costs nothing.  Tiles and strips, one system among a group's and one member among an
ensemble's, bit for bit against the oracle.  The checked build says which passes ran; the
run is a child process, so that the checked library is the only one it loads."""
import json
import multiprocessing as mp
import os
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EXACT = {4, 9}  # sites of the one-sweep passes' checks (CSR columns, stencil neighbours)


def _child(q):
    try:
        sys.path.insert(0, os.path.join(ROOT, "sw-mpdec_b200"))
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        sys.path.insert(0, os.path.join(ROOT, "tests"))
        import numpy as np
        import build
        import cases
        import oracle as O
        import swm
        from test_gpu_parity import random_patankar_system
        swm.LIB_PATH = build.build(checked=True)
        out = {}

        def done(tag, same):
            out[tag] = [bool(same), bool(EXACT & swm.checked_sites()), swm.checked_status()[1]]

        def sweeps(nx, ny, mass, diag, rhs, n):
            """n sweeps in the reference's order."""
            M, D, B = mass.reshape(ny, nx, 5), diag.reshape(ny, nx), rhs.reshape(ny, nx)
            x = B
            for _ in range(n):
                p = M[..., 0] * np.roll(x, 1, 0) + M[..., 1] * np.roll(x, 1, 1)
                p = p + M[..., 3] * np.roll(x, -1, 1)
                x = (B - (p + M[..., 4] * np.roll(x, -1, 0))) / D
            return x.ravel()

        # tiles of 56 x 40 and 48 x 32 cells, strips
        for nx, ny, block in ((70, 61, 0), (70, 61, 4), (1101, 1003, 0)):
            n = nx * ny
            mass, diag, rhs = random_patankar_system(n, 7)
            at = np.arange(n) % 97 == 13
            alone = mass.reshape(n, 5).copy()
            alone[at] = 0.0
            alone = alone.reshape(-1)
            low = diag.copy()
            low[n // 3: n // 3 + 2] = (low[n // 3: n // 3 + 2].view(np.int64) | 0xffffffff).view(
                np.float64)
            ones = diag.copy()
            ones[n // 2] = np.nextafter(2.0, 0.0)  # significand all ones
            big, nan = diag.copy(), rhs.copy()
            big[n // 2] = 1e200
            nan[n // 2] = np.nan
            centre = mass.reshape(n, 5).copy()
            centre[n // 3, 2] = -0.25
            for solver in ("stencil", "csr"):
                o = O.Oracle(O.make_params(nx, ny, (0.0, 0.0), (1.0, 1.0), jacobi_maxiter=40))
                s = swm.Solver(nx=nx, ny=ny, x0=(0.0, 0.0), x1=(1.0, 1.0), solver=solver,
                               jacobi_block=block, jacobi_maxiter=40)
                for tag, args in (("low word", (mass, low, rhs)), ("all ones", (mass, ones, rhs)),
                                  ("tiny", (alone, diag, np.where(at, 1e-150, rhs))),
                                  ("big", (mass, big, rhs)), ("nan", (mass, diag, nan)),
                                  ("centre", (centre.reshape(-1), diag, rhs))):
                    if tag == "centre" and solver == "stencil":
                        continue
                    # (the library goes on to the last sweep on a NaN residual, the
                    # reference's comparison ends its loop)
                    ref, k_ref = (sweeps(nx, ny, *args, 40), 40) if tag == "nan" else o.jacobi(*args)
                    got, k, _ = s.debug_jacobi(*args)
                    done(f"{tag} {solver} {nx} {block}",
                         k == k_ref and np.array_equal(got, ref, equal_nan=True))
                s.close()

        # one step of still water, of water with a patch of 1e-150 depths (whose limiter makes
        # the state non-finite) and of 1e-150 throughout (at rest below the tolerance): as
        # members of an ensemble in both forms and alone.  The persistent form divides and
        # sums by code of its own; finite states are the oracle's too.
        def water(nx, ny, tiny):
            P = np.zeros((3, ny, nx))
            P[0] = 1.0 + 0.1 * np.sin(np.arange(nx) * 2 * np.pi / nx)[None, :]
            if tiny == "patch":
                P[0, 15:29, 20:36] = 1e-150
            if tiny == "all":
                P[0] = 1e-150
            return P

        def step(f):
            try:
                f()
                return 0
            except swm.SwmError as e:
                return e.code

        shapes = [(60, 50, ""), (57, 44, "patch"), (130, 72, ""), (33, 40, "all")]
        kw = dict(x0=(0.0, 0.0), x1=(1.0, 1.0), cfl=0.4)
        b = swm.Batch([swm.make_params(nx, ny, solver="stencil", jacobi_block=4, **kw)
                       for nx, ny, _ in shapes])
        forms = []
        for per_phase in (False, True):
            b.set_launches(per_phase)
            for i, sh in enumerate(shapes):
                b.set_planes(i, water(*sh))
            step(b.step)
            forms.append([b.get_planes(i) for i in range(len(shapes))])
        b.close()
        done("ensemble", all(np.array_equal(x, y, equal_nan=True) for x, y in zip(*forms)))
        for (nx, ny, tiny), ref in zip(shapes, forms[0]):
            o = O.Oracle(O.make_params(nx, ny, kw["x0"], kw["x1"], cfl=0.4))
            o.set_planes(water(nx, ny, tiny))
            dt = o.timestep()
            s = swm.Solver(nx=nx, ny=ny, solver="stencil", **kw)
            s.set_planes(water(nx, ny, tiny))
            ok = s.timestep() == dt and step(lambda: s.step(0.0, dt)) == (
                -3 if tiny == "patch" else 0)
            ok = ok and np.array_equal(s.get_planes(), ref, equal_nan=True)
            if tiny != "patch":
                o.step(0.0, dt)
                ok = ok and np.array_equal(ref, o.get_planes())
            done("step " + tiny, ok)
            s.close()
        q.put(json.dumps(out))
    except Exception as exc:  # reported to the parent
        q.put(json.dumps({"error": repr(exc)}))


def test_operands_cost_ieee_divisions_not_single_sweeps(gpu):
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    p = ctx.Process(target=_child, args=(q,))
    p.start()
    res = json.loads(q.get(timeout=900))
    p.join(timeout=60)
    assert "error" not in res, res
    for tag, (same, exact, failing) in res.items():
        assert same and failing == 0, (tag, res[tag])
        # only the CSR centre slot needs the pattern's own products
        assert exact == tag.startswith("centre"), (tag, res[tag])
    assert len(res) == 3 * (5 + 6) + 3 + 1  # (the two waters share a tag)
