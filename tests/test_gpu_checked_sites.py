"""The checked build's index checks cover the Jacobi forms that the steps take: tiles of
both pass lengths, strips, the one-sweep exact passes (stencil and CSR) and the persistent
ensemble step's tiles each reach their sites, every check passes and the FP64 form still
matches the oracle bit for bit.  The run is a child process, so that the checked library is
the only one it loads."""
import json
import multiprocessing as mp
import os
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RHS, PAIRS, CELLS, CSR, ENS, TILE, STRIP, EXACT = 1, 2, 3, 4, 6, 7, 8, 9


def _child(q):
    try:
        sys.path.insert(0, os.path.join(ROOT, "sw-mpdec_b200"))
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import numpy as np
        import build
        import cases
        import oracle as O
        import swm
        swm.LIB_PATH = build.build(checked=True)
        out = {}

        def single(tag, name, nx, ny, solver, block=0, **kw):
            c = cases.case(name)
            c["nx"], c["ny"] = nx, ny
            P = cases.cell_averages(c)
            kw = dict(dict(g=c["g"], cfl=c["cfl"], bathy_flag=c["bathy_flag"],
                           bathy_par=c["bathy_par"]), **kw)
            o = O.Oracle(O.make_params(nx, ny, c["x0"], c["x1"], **kw))
            s = swm.Solver(nx=nx, ny=ny, x0=c["x0"], x1=c["x1"], solver=solver,
                           jacobi_block=block, **kw)
            o.set_planes(P)
            s.set_planes(P)
            dt = o.timestep()
            o.step(0.0, dt)
            s.step(0.0, dt)
            same = bool(np.array_equal(s.get_planes(), o.get_planes()))
            s.close()
            out[tag] = [same, sorted(swm.checked_sites()), swm.checked_status()[1]]

        def batch(tag, per_phase):
            b = swm.Batch([swm.make_params(n, m, (0.0, 0.0), (3.0, 3.0), precision="split",
                                           solver="stencil", jacobi_block=4)
                           for n, m in ((41, 37), (130, 72), (5, 90))])
            b.set_launches(per_phase)
            for i, (n, m) in enumerate(((41, 37), (130, 72), (5, 90))):
                P = np.zeros((3, m, n))
                P[0] = 1.0 + 0.1 * np.sin(np.arange(n) * 2 * np.pi / n)[None, :]
                b.set_planes(i, P)
            b.step()
            b.close()
            out[tag] = [True, sorted(swm.checked_sites()), swm.checked_status()[1]]

        for solver in ("stencil", "csr"):
            single("tiles8 " + solver, "vortex", 97, 65, solver)
            single("small " + solver, "vortex", 5, 7, solver)
            single("strips " + solver, "vortex", 701, 601, solver)
            single("exact " + solver, "vortex", 57, 40, solver, jacobi_tol=0.0,
                   jacobi_maxiter=40, cfl=0.01)
        single("tiles4 stencil", "vortex", 97, 65, "stencil", 4)
        batch("persistent", False)
        batch("phased", True)
        q.put(json.dumps(out))
    except Exception as exc:  # reported to the parent
        q.put(json.dumps({"error": repr(exc)}))


def test_every_jacobi_form_reaches_its_checks(gpu):
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    p = ctx.Process(target=_child, args=(q,))
    p.start()
    res = json.loads(q.get(timeout=600))
    p.join(timeout=60)
    assert "error" not in res, res
    reached = {"tiles8": TILE, "tiles4": TILE, "small": TILE, "strips": STRIP, "exact": EXACT,
               "persistent": PAIRS, "phased": STRIP}
    for tag, (same, sites, failing) in res.items():
        kind = tag.split()[0]
        assert same and failing == 0, (tag, res[tag])
        # (the exact passes of the CSR form go through its pattern arrays)
        want = CSR if tag == "exact csr" else reached[kind]
        assert want in sites and RHS in sites, (tag, sites)
        if kind in ("tiles8", "tiles4", "small"):
            assert STRIP not in sites, (tag, sites)
    assert CELLS in res["persistent"][1] and ENS in res["persistent"][1]
    assert len(res) == 11
