"""Green build: replica sums shared by thread groups (2 nx - 1 lags per row: one
group above 128 lags, several below) and mirrored lags of finite targets, against
the FP64 oracle operator (tolerance of test_gpu_matvec.py)."""
import numpy as np
import pytest

import ddscat_b200 as D
from oracle import ddscat_oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("dims,pyd,pzd", [((1, 3, 2), 3.0, 2.0), ((2, 3, 3), 3.0, 0.0), ((43, 2, 2), 2.0, 2.0),
                                          ((64, 2, 1), 0.0, 3.0), ((65, 1, 2), 2.0, 2.0)])
def test_periodic_green_matches_oracle(dims, pyd, pzd):
    nx, ny, nz = dims
    nat = nx * ny * nz
    rng = np.random.default_rng(nat)
    iocc = np.ones(nat, dtype=np.int16)
    ak = (0.5, 0.15, 0.1)
    gamma = 0.25
    dda = D.DDA()
    dda.prepare_green(nx, ny, nz, iocc, ak, ipbc=1, gamma=gamma, pyd=pyd, pzd=pzd)
    gp = O.GreenParams(nx, ny, nz, ipbc=1, gamma=gamma, pyd=pyd, pzd=pzd, ak=tuple(float(np.float32(a)) for a in ak))
    op = O.Operator.from_params(gp, iocc)
    x = (rng.normal(size=3 * nat) + 1j * rng.normal(size=3 * nat)).astype(np.complex64)
    adia = np.zeros(3 * nat, dtype=np.complex64)
    y = dda.apply(x, adia, adia)
    yr = op.apply_full(x, adia, adia)
    assert np.linalg.norm(y - yr) <= 2e-5 * np.linalg.norm(yr)
    dda.release()


@pytest.mark.gpu
@pytest.mark.parametrize("idipint", [0, 1])
@pytest.mark.parametrize("dims", [(1, 1, 2), (2, 1, 1), (3, 17, 9), (40, 5, 6), (5, 260, 1)])
def test_finite_green_matches_oracle(dims, idipint):
    """Axis lengths of one site up to one beyond the register transforms."""
    nx, ny, nz = dims
    nat = nx * ny * nz
    rng = np.random.default_rng(nat)
    iocc = np.ones(nat, dtype=np.int16)
    ak = (0.3, -0.2, 0.25)
    dda = D.DDA()
    dda.prepare_green(nx, ny, nz, iocc, ak, dx=(1.0, 0.9, 1.1), idipint=idipint)
    gp = O.GreenParams(nx, ny, nz, idipint=idipint, ak=tuple(float(np.float32(a)) for a in ak),
                       dx=tuple(float(np.float32(a)) for a in (1.0, 0.9, 1.1)))
    op = O.Operator.from_params(gp, iocc)
    x = (rng.normal(size=3 * nat) + 1j * rng.normal(size=3 * nat)).astype(np.complex64)
    adia = np.zeros(3 * nat, dtype=np.complex64)
    y = dda.apply(x, adia, adia)
    yr = op.apply_full(x, adia, adia)
    assert np.linalg.norm(y - yr) <= 2e-5 * np.linalg.norm(yr)
    dda.release()
