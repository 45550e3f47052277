"""Index maps built on the device: rows shorter and longer than a warp, more rows
than one scan step (1024), vacant rows, and a wrong NAT0."""
import numpy as np
import pytest

import ddscat_b200 as D


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(1, 1, 3), (31, 3, 2), (33, 40, 30), (64, 33, 32), (100, 7, 5)])
def test_gather_and_scatter_follow_site_order(dims):
    """EVALQ sees the compact order of a solution the maps gathered: with CXADIA
    chosen per site, A x = b of isolated phases returns x site by site."""
    nx, ny, nz = dims
    nat = nx * ny * nz
    rng = np.random.default_rng(nat)
    iocc = (rng.random(nat) < 0.4).astype(np.int16)
    iocc.reshape(nz * ny, nx)[1::3] = 0
    iocc[0] = 1
    n0 = int(iocc.sum())
    k = (0.2, 0.1, 0.05)
    # a huge diagonal: x = b / adia to FP32 rounding, different on every site
    b = (np.tile(iocc, 3) * (1 + rng.random(3 * nat))).astype(np.complex64)
    adia = (1e8 * (1 + rng.random(3 * nat))).astype(np.complex64)
    dda = D.DDA()
    dda.prepare_green(nx, ny, nz, iocc, k)
    out = dda.solve("pbcgs2", b, adia, np.zeros_like(b), maxit=20, tol=1e-6)
    ref = b / adia
    assert np.abs(out.x - ref).max() <= 1e-5 * np.abs(ref).max()
    with pytest.raises(D.DDSCATError) as e:
        dda.prepare_green(nx, ny, nz, iocc, k, nat0=n0 - 1 if n0 > 1 else n0 + 1)
    assert e.value.code == 208 and str(n0) in str(e.value)
    dda.release()
