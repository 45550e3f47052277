"""Reused device blocks: repeated prepares, solves and far-field calls on targets
of changing size give the results of a fresh state, concurrent targets do not
share blocks, and ddscat_cuda_release returns the memory."""
import numpy as np
import pytest

import ddscat_b200 as D
from ddscat_b200 import targets


def _run(dda, n, seed):
    prob = targets.make_problem(n, n + 1, n + 2, m=1.4 + 0.03j, x=2.0)
    k = prob.incid[0].k
    dda.prepare_green(prob.nx, prob.ny, prob.nz, prob.iocc, k)
    b, adia, aoff = prob.rhs(0), prob.adia(0), prob.aoff()
    o = dda.solve("pbcgs2", b, adia, aoff, maxit=200, tol=1e-5)
    q = dda.evalq(k)
    s = dda.scat(k, prob.incid[0].e, prob.x0)
    r = dda.residual_f64(b[None], o.x[None], adia[None])
    return o.x, np.array([*q, s["csca"], s["cbksca"], r[0]])


@pytest.mark.gpu
def test_reused_blocks_give_the_same_results():
    torch = pytest.importorskip("torch")
    dda = D.DDA()
    dda.release()
    first = {n: _run(dda, n, 0) for n in (12, 20, 9)}
    dda.release()
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    for n in (20, 9, 12, 9, 20, 12):  # blocks of other sizes and owners
        x, v = _run(dda, n, 1)
        assert np.array_equal(x, first[n][0]) and np.array_equal(v, first[n][1])
    dda.release()
    assert torch.cuda.mem_get_info()[0] >= free0 - (4 << 20)


@pytest.mark.gpu
def test_refused_prepares_keep_no_memory():
    """A prepare whose NAT0 is not the occupied count (208) has built its index
    maps, 10 bytes per site, when it finds out; 60 of them at 96^3 (530 MB) return
    everything but the bounded reuse lists, and those with the release."""
    torch = pytest.importorskip("torch")
    n = 96
    iocc = np.ones(n ** 3, dtype=np.int16)
    dda = D.DDA()
    dda.prepare_green(8, 8, 8, np.ones(512, dtype=np.int16), (0.3, 0.0, 0.0))  # one-time set-up
    dda.release()
    free0 = torch.cuda.mem_get_info()[0]
    for _ in range(60):
        with pytest.raises(D.DDSCATError) as err:
            dda.prepare_green(n, n, n, iocc, (0.3, 0.0, 0.0), nat0=n ** 3 - 1)
        assert err.value.code == 208
    assert torch.cuda.mem_get_info()[0] >= free0 - (64 << 20)
    dda.release()
    assert torch.cuda.mem_get_info()[0] >= free0 - (4 << 20)


@pytest.mark.gpu
@pytest.mark.parametrize("layout,keep_mib", [("slices", 512), ("fft3d", 2048)])
def test_idle_blocks_stay_within_the_limit(layout, keep_mib):
    """A 160^3 target (3.4 GB) followed by a small one leaves at most the limit of
    the reuse lists; the SLICES build's is small."""
    torch = pytest.importorskip("torch")
    dda = D.DDA(layout)

    def prepare(n):
        dda.prepare_green(n, n, n, np.ones(n ** 3, dtype=np.int16), (0.3, 0.0, 0.0))

    prepare(16)
    dda.release()
    free0 = torch.cuda.mem_get_info()[0]
    prepare(160)
    big = free0 - torch.cuda.mem_get_info()[0]
    prepare(16)
    idle = free0 - torch.cuda.mem_get_info()[0]
    assert big > (2 << 30) and idle <= (keep_mib + 64) << 20
    dda.release()
    assert torch.cuda.mem_get_info()[0] >= free0 - (4 << 20)


@pytest.mark.gpu
def test_concurrent_targets_do_not_share_blocks():
    probs = [targets.make_problem(n, m=1.4 + 0.03j, x=1.5) for n in (8, 10, 12, 14, 16, 9)]

    def tlist():
        out = []
        for p in probs:
            b = np.stack([p.rhs(r) for r in range(2)])
            out.append(dict(dims=(p.nx, p.ny, p.nz), iocc=p.iocc, ak=p.incid[0].k, b=b, x=np.zeros_like(b),
                            adia=np.stack([p.adia(r) for r in range(2)])))
        return out

    dda = D.DDA()
    ref = tlist()
    dda.multi_solve(ref, nthreads=1)
    for _ in range(3):
        got = tlist()
        dda.multi_solve(got, nthreads=6)
        for a, b in zip(ref, got):
            assert np.array_equal(a["x"], b["x"])
