"""Targets with odd sides and sides whose 2n is no register-FFT length run on
padded axis lengths (x-first pipeline): MATVEC against the FP64 oracle, and
against the same target on the 2n grid (DDSCAT_B200_NOPAD=1).

Tolerances as in test_gpu_matvec.py: FP32 FFT errors grow like eps_f32 log2(M),
2e-5 in norm and 1e-4 of max|y| are two orders above; FP64 results agree to
1e-12 (eps_f64 log2(M) with the same margin)."""
import ctypes as ct

import numpy as np
import pytest

import ddscat_b200 as D
from oracle import ddscat_oracle as O

RTOL_L2, RTOL_MAX = 2e-5, 1e-4


def _case(dims, seed=3):
    rng = np.random.default_rng(seed)
    nat = int(np.prod(dims))
    iocc = (rng.random(nat) < 0.7).astype(np.int16)
    iocc[0] = 1

    def cn(s=1.0):
        return (s * (rng.normal(size=3 * nat) + 1j * rng.normal(size=3 * nat))).astype(np.complex64)

    return iocc, (0.31, -0.17, 0.22), cn(), cn(), cn(0.3)


def _close(y, yr):
    assert np.linalg.norm(y - yr) <= RTOL_L2 * np.linalg.norm(yr)
    assert np.abs(y - yr).max() <= RTOL_MAX * np.abs(yr).max()


# per-thread tiles: 11 -> 32, 17 -> 48, 33 -> 96, 13 -> 32; one TMA box (256):
# 101, 99; two boxes (512) on each axis: 131; rows that end in the first, a
# middle and the last element pair of a tile (97, 111, 127)
RAGGED = [(11, 7, 5), (17, 13, 33), (33, 17, 18), (18, 45, 11), (101, 9, 7), (9, 99, 7), (7, 9, 101), (9, 97, 111),
          (127, 111, 9), (131, 9, 7), (9, 131, 7), (7, 9, 131), (25, 27, 29)]


@pytest.mark.gpu
@pytest.mark.parametrize("layout", ["fft3d", "slices"])
@pytest.mark.parametrize("dims", RAGGED)
def test_ragged_apply_matches_oracle(layout, dims):
    iocc, ak, x, adia, aoff = _case(dims)
    gp = O.GreenParams(*dims, ak=tuple(float(np.float32(a)) for a in ak))
    op = O.Operator.from_params(gp, iocc)
    dda = D.DDA(layout)
    dda.prepare_green(*dims, iocc, ak)
    for cwhat in "NC":
        y = dda.apply(x, adia, aoff, cwhat)
        _close(y, op.apply_full(x, adia, aoff, cwhat))
        assert np.all(y.reshape(3, -1)[:, iocc == 0] == 0)
    dda.release()


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(17, 13, 11), (7, 33, 18), (20, 24, 18), (9, 65, 6), (65, 9, 7), (8, 6, 67)])
@pytest.mark.parametrize("pz", [0.0, 1.0])
def test_ragged_periodic_equals_unpadded(monkeypatch, dims, pz):
    iocc, ak, x, adia, aoff = _case(dims)
    out = []
    for nopad in ("0", "1"):
        monkeypatch.setenv("DDSCAT_B200_NOPAD", nopad)
        dda = D.DDA()
        dda.prepare_green(*dims, iocc, ak, ipbc=1, gamma=0.1, pyd=float(dims[1]), pzd=pz * dims[2])
        out.append([dda.apply(x, adia, aoff, c) for c in "NC"])
        dda.release()
    for a, b in zip(*out):
        _close(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(13, 17, 11), (33, 9, 21), (51, 7, 39)])
def test_ragged_fp64_and_batch_equal_unpadded(monkeypatch, dims):
    """FP64 residuals and compact multi-RHS solves (masks, fused x*y sums)."""
    rng = np.random.default_rng(8)
    nat = int(np.prod(dims))
    iocc = (rng.random(nat) < 0.6).astype(np.int16)
    iocc[0] = 1
    R = 6
    b = ((rng.normal(size=(R, 3 * nat)) + 1j * rng.normal(size=(R, 3 * nat))) * np.tile(iocc, 3)).astype(np.complex64)
    adia = np.full((R, 3 * nat), 12.0 - 3.0j, dtype=np.complex64)
    x0 = (b / adia).astype(np.complex64)
    res, sol = [], []
    for nopad in ("0", "1"):
        monkeypatch.setenv("DDSCAT_B200_NOPAD", nopad)
        dda = D.DDA()
        dda.prepare_green(*dims, iocc, (0.3, 0.0, 0.0))
        res.append(dda.residual_f64(b, x0, adia))
        for name, sym in (("qmrccg", True), ("pbcgs2", False)):
            x = np.zeros_like(b)
            out = dda.solve_batch(name, b, x, adia, maxit=300, tol=1e-5, replace=True, symmetric=sym, graph=True)
            assert np.all(out.status == 0)
            assert np.all(dda.residual_f64(b, x, adia) <= 1.2e-5)
            sol.append(x)
        dda.release()
    assert np.abs(res[0] - res[1]).max() <= 1e-12
    for k in range(2):  # iterates within 20 tol of the same solution each
        assert np.linalg.norm(sol[k] - sol[2 + k]) <= 40e-5 * np.linalg.norm(sol[k])


def _rel_errors(monkeypatch, dims, periodic=False):
    """Norm errors against the FP64 oracle on the default grid and on the 2n grid,
    with CXADIA of the size of an inverse polarisability (14 at m = 1.5)."""
    iocc, ak, x, _, aoff = _case(dims, seed=17)
    adia = np.full_like(x, 12.0 - 3.0j)
    per = dict(ipbc=1, gamma=0.1, pyd=float(dims[1]), pzd=float(dims[2])) if periodic else {}
    gp = O.GreenParams(*dims, ak=tuple(float(np.float32(a)) for a in ak),
                       **{k: float(np.float32(v)) if k == "gamma" else v for k, v in per.items()})
    ref = O.Operator.from_params(gp, iocc).apply_full(x, adia, aoff)
    out = []
    for nopad in ("0", "1"):
        monkeypatch.setenv("DDSCAT_B200_NOPAD", nopad)
        dda = D.DDA()
        dda.prepare_green(*dims, iocc, ak, **per)
        out.append(np.linalg.norm(dda.apply(x, adia, aoff) - ref) / np.linalg.norm(ref))
        dda.release()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("dims,periodic", [((13, 17, 11), False), ((25, 27, 29), False), ((35, 35, 35), False),
                                           ((47, 47, 47), False), ((66, 12, 10), False), ((45, 37, 31), False),
                                           ((8, 9, 65), False), ((7, 131, 6), False), ((13, 13, 13), True),
                                           ((15, 15, 15), True), ((20, 24, 18), True)])
def test_register_grid_is_no_less_precise_than_2n(monkeypatch, dims, periodic):
    """Targets that would run the generic transforms on their 2n grid, which sum
    prime-length DFTs in FP64, lose no precision on register lengths."""
    padded, generic = _rel_errors(monkeypatch, dims, periodic)
    assert padded <= generic


@pytest.mark.gpu
def test_80_points_are_no_less_precise_than_96(monkeypatch):
    """36^3 runs on 80 points per axis, 48^3 on 96: the shorter transform has no
    more roundings, so its twiddles must not make it less precise."""
    assert _rel_errors(monkeypatch, (36, 36, 36))[0] <= _rel_errors(monkeypatch, (48, 48, 48))[0]


@pytest.mark.gpu
@pytest.mark.parametrize("dims,planes", [((69, 69, 73), "some"), ((45, 37, 31), "all"), ((5, 255, 251), "some")])
def test_ragged_noalloc_equals_apply(dims, planes):
    """Ragged targets of up to 349,525 sites are accepted whatever their padded
    grid needs: the middle stage runs in plane batches where it does not fit."""
    torch = pytest.importorskip("torch")
    iocc, ak, x, adia, aoff = _case(dims)
    dda = D.DDA()
    dda.prepare_green(*dims, iocc, ak)
    t = [torch.from_numpy(a).cuda() for a in (x, adia, aoff)]
    y = torch.zeros_like(t[0])
    rc = dda.lib.ddscat_b200_apply_noalloc_f32(ord("C"), *[ct.c_void_p(v.data_ptr()) for v in (t[0], y, t[1], t[2])],
                                               ct.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    _close(y.cpu().numpy(), dda.apply(x, adia, aoff, "C"))
    dda.release()
