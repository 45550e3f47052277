"""Far-field sums at the edges of the row-contraction kernel: columns around its
64-column chunks, directions around its tiles of 64, odd row counts, vacant rows
and sparse targets, against direct FP64 sums.

Tolerance: an FP32 row sum is chains of 8 complex products (two roundings each in
either component) of factors rounded to FP32 (one more, the phase table), met in
a compensated sum (two); the y and z phases are FP64 and the amplitude is rounded
to FP32 once: 20 roundings per component, so an amplitude is within 20 sqrt(2) =
29 times 2^-24 of |k|^3 sum_j |P_j|.  FP64: chains of 64 products, phases and
their products, 136 roundings, and eps |k r| of the phase arguments (|k r| < 200)
on top: 200 + 200 times 2^-53."""
import numpy as np
import pytest

import ddscat_b200 as D

CASES = [((1, 1, 1), 1.0, 1), ((1, 5, 3), 0.5, 3), ((33, 4, 3), 0.6, 63), ((63, 3, 3), 0.9, 64), ((64, 2, 5), 0.6, 65),
         ((65, 5, 3), 0.6, 127), ((128, 3, 2), 0.02, 128), ((130, 5, 5), 0.1, 129), ((200, 7, 3), 0.5, 300),
         ((17, 40, 41), 0.3, 5), ((6, 9, 130), 0.5, 33)]


@pytest.mark.gpu
@pytest.mark.parametrize("dims,p_occ,ndir", CASES)
def test_farfield_sums_match_direct_sums(dims, p_occ, ndir):
    nx, ny, nz = dims
    rng = np.random.default_rng(sum(dims) + ndir)
    nat = nx * ny * nz
    iocc = (rng.random(nat) < p_occ).astype(np.int16)
    iocc.reshape(nz, ny, nx)[nz // 2] = 0  # a vacant plane
    iocc[0] = 1
    occ = np.flatnonzero(iocc)
    n0 = occ.size
    k = np.array([0.25, 0.125, -0.5])
    kk = np.linalg.norm(k)
    n = rng.normal(size=(ndir, 3))
    aks = (kk * n / np.linalg.norm(n, axis=1, keepdims=True)).astype(np.float32).astype(np.float64)
    em1, em2 = (rng.normal(size=(2, ndir, 3))).astype(np.float32).astype(np.float64)
    x0 = (-0.5, 0.25, -1.5)
    p = (rng.normal(size=(3, n0)) + 1j * rng.normal(size=(3, n0))).astype(np.complex64)
    pos = np.stack([occ % nx + 1 + x0[0], (occ // nx) % ny + 1 + x0[1], occ // (nx * ny) + 1 + x0[2]])
    S = np.exp(-1j * (aks @ pos)) @ p.astype(np.complex128).T
    f = np.stack([np.sum(em1 * S, axis=1), np.sum(em2 * S, axis=1)]) * kk ** 3
    bound = kk ** 3 * np.abs(p).sum() * max(np.abs(em1).max(), np.abs(em2).max())
    dda = D.DDA()
    dda.prepare_green(nx, ny, nz, iocc, k)
    ones, zero = np.ones(3 * n0, dtype=np.complex64), np.zeros(3 * n0, dtype=np.complex64)
    dda.evalq(k, use_resident=0, e=ones, p=p, adia=ones, aoff=zero)
    sc = dda.scat(k, (0, 0, 0), x0, jpbc=3, aks=aks, em1=em1, em2=em2)
    assert np.abs(np.stack([sc["f1"], sc["f2"]]) - f).max() <= 29 * 2.0 ** -24 * bound
    x = np.zeros((2, 3, nat), dtype=np.complex128)
    x[:, :, occ] = p
    x[1] *= 2
    f1, f2 = dda.scat_amplitudes_f64(x.reshape(2, -1), k, aks, em1, em2, x0)
    for r in range(2):
        assert np.abs(np.stack([f1[r], f2[r]]) - (1 + r) * f).max() <= (200 + 200) * 2.0 ** -53 * (1 + r) * bound
    dda.release()
