"""Ensembles: what the two step forms report, and the solves that only exact sums decide, in
both forms."""
import json
import multiprocessing as mp
import os
import sys

import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EXACT = 9  # site of the one-sweep passes' checks


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


def _child(q):
    try:
        sys.path.insert(0, os.path.join(ROOT, "sw-mpdec_b200"))
        sys.path.insert(0, os.path.join(ROOT, "oracle"))
        import build
        import oracle as O
        import swm
        swm.LIB_PATH = build.build(checked=True)
        out = {}
        # members whose solves end inside the band (tolerance 0, short steps), odd and even
        # widths, among ones that end by the usual tolerance
        members = [("vortex", 40, 0.4, 1e-16), ("vortex", 57, 0.01, 0.0), ("island", 50, 0.4, 1e-16),
                   ("vortex", 66, 0.01, 0.0), ("lake", 73, 0.4, 1e-16)]
        for precision in ("fp64", "split", "fp64_fma"):
            cs, params = [], []
            for name, n, cfl, tol in members:
                c = cases.case(name, n=n)
                kw = dict(g=c["g"], cfl=cfl, bathy_flag=c["bathy_flag"], bathy_par=c["bathy_par"],
                          jacobi_tol=tol, jacobi_maxiter=60)
                cs.append((c, kw))
                params.append(swm.make_params(c["nx"], c["ny"], c["x0"], c["x1"], solver="stencil",
                                              precision=precision, jacobi_block=4, **kw))
            b = swm.Batch(params)
            got, sites = {}, {}
            for per_phase in (False, True):
                b.set_launches(per_phase)
                for i, (c, _) in enumerate(cs):
                    b.set_planes(i, cases.cell_averages(c))
                swm.checked_sites()
                for _ in range(2):
                    b.step()
                sites[per_phase] = swm.checked_sites()
                got[per_phase] = [b.get_planes(i) for i in range(len(cs))], b.stats()[2]
            b.close()
            same = np.array_equal(got[False][1], got[True][1]) and all(
                np.array_equal(x, y) for x, y in zip(got[False][0], got[True][0]))
            # alone, and (FP64) by the oracle
            for i, (c, kw) in enumerate(cs):
                s = swm.Solver(params[i])
                s.set_planes(cases.cell_averages(c))
                o = O.Oracle(O.make_params(c["nx"], c["ny"], c["x0"], c["x1"], **kw))
                o.set_planes(cases.cell_averages(c))
                for _ in range(2):
                    s.step(0.0, s.timestep())
                    if precision == "fp64":
                        o.step(0.0, o.timestep())
                same = same and np.array_equal(s.get_planes(), got[True][0][i])
                same = same and s.stats()["jacobi_iters"] == list(got[True][1][:, i])
                if precision == "fp64":
                    same = same and np.array_equal(o.get_planes(), got[True][0][i])
                s.close()
            out[precision] = [bool(same), EXACT in sites[True], swm.checked_status()[1]]
        q.put(json.dumps(out))
    except Exception as exc:  # reported to the parent
        q.put(json.dumps({"error": repr(exc)}))


def test_solves_that_end_inside_the_band(gpu):
    # the checked build says that the batched solve's one-sweep passes ran; a child process,
    # so that the checked library is the only one it loads
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    p = ctx.Process(target=_child, args=(q,))
    p.start()
    res = json.loads(q.get(timeout=900))
    p.join(timeout=60)
    assert "error" not in res, res
    assert res == {k: [True, True, 0] for k in ("fp64", "split", "fp64_fma")}
