"""The batched z pass that stages Green lines and prefetches rows (kx_zg3r): one
and several RHS per block, masked RHS, odd row lengths and every axis length it
is built for, checked by the FP64 residuals of batched solves."""
import numpy as np
import pytest

import ddscat_b200 as D

# padded z lengths 16, 32, 48, 64, 128, 256; the last case has enough lines for
# one chunk of all RHS per block
CASES = [(9, 8, 7), (9, 10, 13), (12, 9, 23), (10, 11, 31), (9, 12, 57), (12, 10, 101), (32, 120, 99)]


@pytest.mark.gpu
@pytest.mark.parametrize("dims", CASES)
@pytest.mark.parametrize("least", ["1", "4"])
def test_zpass_with_staged_rows_solves(monkeypatch, dims, least):
    monkeypatch.setenv("DDSCAT_B200_ZG3R_MIN", least)
    rng = np.random.default_rng(4)
    nat = int(np.prod(dims))
    iocc = (rng.random(nat) < 0.5).astype(np.int16)
    iocc[0] = 1
    R = 5
    b = ((rng.normal(size=(R, 3 * nat)) + 1j * rng.normal(size=(R, 3 * nat))) * np.tile(iocc, 3)).astype(np.complex64)
    # different diagonals: the RHS converge, and are masked, at different iterations
    adia = np.stack([np.full(3 * nat, (14.0 + 8 * r) - 3.0j) for r in range(R)]).astype(np.complex64)
    dda = D.DDA()
    dda.prepare_green(*dims, iocc, (0.3, 0.0, 0.0))
    x = np.zeros_like(b)
    out = dda.solve_batch("qmrccg", b, x, adia, maxit=400, tol=1e-5, replace=True, symmetric=True, graph=True)
    assert np.all(out.status == 0) and len(set(out.itno.tolist())) > 1
    assert np.all(dda.residual_f64(b, x, adia) <= 1.2e-5)
    dda.release()
