"""Drop-in PBCGS2 and QMRCCG as iteration graphs (quiet, from the 4th and the 16th
iteration on) give bit for bit what the same iterations give launch by launch (with the
per-MATVEC output): solutions, iteration and MATVEC counts, through reliable
checks, restarts and MAXIT.  Shorter solves run launch by launch and pay nothing
for the graph."""
import time

import numpy as np
import pytest

import ddscat_b200 as D
from ddscat_b200 import targets
from oracle import ddscat_oracle as O


def _both_levels(dda, *args, **kw):
    got = []
    try:
        for level in (0, 1):
            dda.lib.ddscat_b200_set_verbose(level)
            n0 = dda.launch_count()
            o = dda.solve(*args, check=False, **kw)
            got.append((o, dda.launch_count() - n0))
    finally:
        dda.lib.ddscat_b200_set_verbose(-1)
    (a, na), (c, nc) = got
    assert (a.rc, a.itno, a.ncompte, a.tole) == (c.rc, c.itno, c.ncompte, c.tole)
    assert np.array_equal(a.x, c.x)
    assert na == nc  # the kernels a graph runs are counted like launched ones
    return a


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
    a = _both_levels(dda, solver, b, adia, aoff, x0=start, maxit=maxit, tol=1e-6)
    if dims == (26, 20, 24):  # 25 and 82 iterations in 64 bits
        assert a.itno > 16
    dda.release()


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["pbcgs2", "qmrccg"])
@pytest.mark.parametrize("maxit", [3, 4, 5, 15, 16, 17, 43])
def test_graph_on_a_caller_supplied_odd_grid(solver, maxit):
    """A Green tensor from the caller keeps the 2n grid, here of the generic
    transforms; strong scattering, so every solve runs to MAXIT."""
    dims = (13, 11, 9)
    prob = targets.make_problem(*dims, m=3 + 0.2j, x=2.5)
    k = prob.incid[0].k
    oct6 = O.green_octant(O.GreenParams(*dims, ak=tuple(float(np.float32(v)) for v in k))).astype(np.complex64)
    dda = D.DDA()
    dda.prepare(*dims, prob.iocc, oct6)
    a = _both_levels(dda, solver, prob.rhs(0), prob.adia(0), prob.aoff(), maxit=maxit, tol=1e-7)
    assert a.itno == maxit
    dda.release()


@pytest.mark.gpu
@pytest.mark.parametrize("solver", ["pbcgs2", "qmrccg"])
def test_short_solves_pay_for_no_graph(solver):
    """The 2nd and 3rd iteration take at most 150 us more than the 7th and 8th:
    recording a graph in one of them costs 350.  The fastest of calls taken in
    turn, so that a change of the host's clock meets all of them."""
    prob = targets.make_problem(16, 16, 16, m=2.5 + 0.02j, x=3.0)
    b, adia, aoff = prob.rhs(0), prob.adia(0), prob.aoff()
    dda = D.DDA()
    dda.prepare_green(16, 16, 16, prob.iocc, prob.incid[0].k)
    best = {1: 1.0, 3: 1.0, 6: 1.0, 8: 1.0}
    try:
        dda.lib.ddscat_b200_set_verbose(0)
        for _ in range(100):
            for maxit in best:
                t = time.perf_counter()
                o = dda.solve(solver, b, adia, aoff, maxit=maxit, tol=1e-7, check=False)
                best[maxit] = min(best[maxit], time.perf_counter() - t)
                assert o.itno == maxit
        assert best[3] - best[1] <= best[8] - best[6] + 150e-6
    finally:
        dda.lib.ddscat_b200_set_verbose(-1)
    dda.release()
