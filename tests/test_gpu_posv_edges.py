"""The factor + solve drivers and potrf_l beyond n = 64 at the edges of the 16-row
blocks and of the size ranges (64 | 65, 128 | 129, 160 | 161): uneven batches
against numpy's solution (1e-13, the FP64 bar of every routine, for matrices of
condition below 10; the mixed solver refines to the same), non-positive pivots, a
workspace aligned to 8 bytes, row offsets."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import relfro

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 7, 15, 16, 17, 31, 33, 48, 49, 63, 64, 65, 66, 67, 68, 79, 80, 81, 96, 97, 111, 113, 127, 128, 129, 143,
         144, 145, 160, 161, 175, 191, 193, 224, 225, 241, 255, 256, 257, 300]


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def spd(rng, n):
    G = rng.standard_normal((n, n))
    return G @ G.T / n + np.eye(n)


def batch(ns, mats, rhs):
    import torch
    from blasfeo_b200.workloads import SpdBatch
    by_n = {}
    for n in sorted(set(ns)):
        idx = np.array([i for i, v in enumerate(ns) if v == n])
        by_n[n] = (idx, torch.from_numpy(np.stack([mats[i] for i in idx])).cuda())
    return SpdBatch(np.array(ns, np.int32), by_n, rhs)


def solve(bf, W, ns, mixed, work=None, nbytes=0):
    import torch
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    info = torch.full((len(ns),), -9, dtype=torch.int32, device="cuda")
    wp = C.c_void_p(work) if work else None
    if mixed:
        st = bf.lib.blasfeo_dsposv_l_vbatch(len(ns), P(W.nvec), W.max_n, P(W.desc), P(W.bdesc), P(W.xdesc), 30, 1e-14,
                                            None, None, P(info), wp, nbytes, None)
    else:
        st = bf.lib.blasfeo_dposv_l_vbatch(len(ns), P(W.nvec), W.max_n, P(W.desc), P(W.bdesc), P(W.xdesc), P(info), wp,
                                           nbytes, None)
    assert st == 0
    torch.cuda.synchronize()
    x = W.x.cpu().numpy()
    return [x[o: o + n] for o, n in zip(W.voff, ns)], info.cpu().numpy()


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("cap", [64, 128, 300])
def test_solve(bf, mixed, cap):
    if mixed and cap > 256:
        cap = 256
    rng = np.random.default_rng(cap)
    ns = [n for n in SIZES if n <= cap] * 2
    mats, rhs = [spd(rng, n) for n in ns], [rng.standard_normal(n) for n in ns]
    low = [np.where(np.tril(np.ones_like(A)) > 0, A, np.nan) for A in mats]  # the upper part is not read
    x, info = solve(bf, batch(ns, low, rhs), ns, mixed)
    assert (info == 0).all()
    for i, n in enumerate(ns):
        assert relfro(x[i], np.linalg.solve(mats[i], rhs[i])) <= 1e-13, n


@pytest.mark.parametrize("n", [40, 80, 130])
def test_bad_pivots(bf, n):
    """Pivot j negative: info = j + 1; the other systems of the call are solved."""
    rng = np.random.default_rng(n)
    js = list(range(0, n, 3)) + [n - 1]
    A0 = spd(rng, n)
    L = np.linalg.cholesky(A0)
    mats = [A0.copy() for _ in js] + [spd(rng, 150), spd(rng, n)]
    for k, j in enumerate(js):
        mats[k][j, j] = L[j, :j] @ L[j, :j] - 1.0
    ns = [len(A) for A in mats]
    rhs = [rng.standard_normal(m) for m in ns]
    x, info = solve(bf, batch(ns, mats, rhs), ns, False)
    assert list(info) == [j + 1 for j in js] + [0, 0]
    for i in (-2, -1):
        assert relfro(x[i], np.linalg.solve(mats[i], rhs[i])) <= 1e-13


def test_workspace_aligned_to_8_bytes(bf):
    import torch
    rng = np.random.default_rng(5)
    ns = [n for n in SIZES if n <= 200]
    mats, rhs = [spd(rng, n) for n in ns], [rng.standard_normal(n) for n in ns]
    need = bf.lib.blasfeo_dposv_worksize_n(len(ns), max(ns), 0)
    work = torch.zeros(need // 8 + 4, dtype=torch.float64, device="cuda")
    x, info = solve(bf, batch(ns, mats, rhs), ns, False, work.data_ptr() + 8, need)
    assert (info == 0).all()
    for i, n in enumerate(ns):
        assert relfro(x[i], np.linalg.solve(mats[i], rhs[i])) <= 1e-13, n


@pytest.mark.parametrize("n", [65, 100, 144, 160, 161, 192, 193, 250, 257])
@pytest.mark.parametrize("off", [(0, 0), (3, 6), (4, 1)])
def test_potrf(bf, n, off):
    import torch
    rng = np.random.default_rng(n)
    ci, di = off
    A = np.stack([spd(rng, n) for _ in range(3)])
    full = np.zeros((3, n + 8, n))
    full[:, ci: ci + n] = np.where(np.tril(np.ones((n, n))) > 0, A, np.nan)
    c, d = bf.DMatBatch(n + 8, n, 3).pack_all(full), bf.DMatBatch(n + 8, n, 3)
    info = torch.full((3,), -9, dtype=torch.int32, device="cuda")
    assert bf.lib.blasfeo_dpotrf_l_batch(3, n, c.ref, ci, 0, d.ref, di, 0, C.c_void_p(info.data_ptr()), None) == 0
    torch.cuda.synchronize()
    assert (info.cpu().numpy() == 0).all()
    L = np.tril(d.unpack_all()[:, di: di + n])
    for k in range(3):
        assert relfro(L[k], np.linalg.cholesky(A[k])) <= 1e-13
