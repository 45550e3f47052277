"""Drop-in PBCGS2 and QMRCCG as iteration graphs (quiet) give bit for bit what the
same iterations give launch by launch (with the per-MATVEC output): solutions,
iteration and MATVEC counts, through reliable checks, restarts and MAXIT."""
import numpy as np
import pytest

import ddscat_b200 as D
from ddscat_b200 import targets


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["pbcgs2", "qmrccg"])
@pytest.mark.parametrize("dims,maxit,x0", [((9, 8, 7), 200, False), ((16, 14, 18), 200, True), ((24, 24, 24), 5, False),
                                           ((13, 17, 11), 1, False), ((26, 20, 24), 300, False)])
def test_graph_iterations_equal_launched_iterations(solver, dims, maxit, x0):
    prob = targets.make_problem(*dims, m=1.7 + 0.05j, x=0.35 * max(dims) / 2)
    k = prob.incid[0].k
    b, adia, aoff = prob.rhs(0), prob.adia(0), prob.aoff()
    start = (0.1 * b).astype(np.complex64) if x0 else None
    dda = D.DDA()
    dda.prepare_green(*dims, prob.iocc, k)
    got = []
    try:
        for level in (0, 1):
            dda.lib.ddscat_b200_set_verbose(level)
            n0 = dda.launch_count()
            o = dda.solve(solver, b, adia, aoff, x0=start, maxit=maxit, tol=1e-6, check=False)
            got.append((o, dda.launch_count() - n0))
    finally:
        dda.lib.ddscat_b200_set_verbose(-1)
    (a, na), (c, nc) = got
    assert (a.rc, a.itno, a.ncompte, a.tole) == (c.rc, c.itno, c.ncompte, c.tole)
    assert np.array_equal(a.x, c.x)
    assert na == nc  # the kernels a graph runs are counted like launched ones
    dda.release()
