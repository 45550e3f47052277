"""The 5 * 2^k axis lengths (80, 160, 320) in every pass: natural (2n is the
length) and padded rows against the FP64 oracle, a CPU-supplied spectrum on such
a grid, FP64 residuals (80 only) and the compact batched form.  Tolerances as in
test_gpu_matvec.py."""
import numpy as np
import pytest

import ddscat_b200 as D
from oracle import ddscat_oracle as O


def _inputs(dims, seed=2):
    rng = np.random.default_rng(seed)
    nat = int(np.prod(dims))
    iocc = (rng.random(nat) < 0.7).astype(np.int16)
    iocc[0] = 1
    v = [(rng.normal(size=3 * nat) + 1j * rng.normal(size=3 * nat)).astype(np.complex64) for _ in range(3)]
    return iocc, (0.3, 0.2, -0.25), v


def _check(y, yr):
    assert np.linalg.norm(y - yr) <= 2e-5 * np.linalg.norm(yr)
    assert np.abs(y - yr).max() <= 1e-4 * np.abs(yr).max()


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(40, 6, 8), (6, 40, 8), (8, 6, 40), (37, 33, 39), (80, 8, 6), (6, 80, 8), (8, 6, 80),
                                  (71, 9, 66), (160, 6, 8), (8, 160, 6), (6, 8, 160), (129, 7, 6), (7, 157, 9),
                                  (9, 7, 133)])
def test_five_times_two_to_the_k_matches_oracle(dims):
    iocc, ak, (x, adia, aoff) = _inputs(dims)
    op = O.Operator.from_params(O.GreenParams(*dims, ak=tuple(float(np.float32(a)) for a in ak)), iocc)
    dda = D.DDA()
    dda.prepare_green(*dims, iocc, ak)
    for c in "NC":
        _check(dda.apply(x, adia, aoff, c), op.apply_full(x, adia, aoff, c))
    dda.release()


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(40, 8, 8), (8, 80, 8), (8, 8, 160)])
def test_cpu_supplied_spectrum(dims):
    iocc, ak, (x, adia, aoff) = _inputs(dims)
    gp = O.GreenParams(*dims, ak=tuple(float(np.float32(a)) for a in ak))
    dda = D.DDA()
    dda.prepare(*dims, iocc, O.green_octant(gp).astype(np.complex64))
    _check(dda.apply(x, adia, aoff), O.Operator.from_params(gp, iocc).apply_full(x, adia, aoff))
    dda.release()


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(40, 38, 37), (70, 9, 33), (9, 36, 75), (96, 5, 8), (48, 6, 6)])
def test_fp64_and_batches(dims):
    iocc, ak, _ = _inputs(dims)
    nat = iocc.size
    rng = np.random.default_rng(9)
    b = ((rng.normal(size=(5, 3 * nat)) + 1j * rng.normal(size=(5, 3 * nat))) * np.tile(iocc, 3)).astype(np.complex64)
    adia = np.full((5, 3 * nat), 16.0 - 3.0j, dtype=np.complex64)
    dda = D.DDA()
    dda.prepare_green(*dims, iocc, ak)
    x = np.zeros_like(b)
    out = dda.solve_batch("qmrccg", b, x, adia, maxit=300, tol=1e-5, replace=True, symmetric=True, graph=True)
    assert np.all(out.status == 0)
    assert np.all(dda.residual_f64(b, x, adia) <= 1.2e-5)
    dda.release()
