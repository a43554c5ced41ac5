"""trsm_rltn / rltu by a thread per row with 128 threads staging A (n > 48, launches that fill the GPU): up to and beyond
32 and 64 rows, the largest n of each kernel, row offsets off the panel grid; against numpy in FP64 with the
repository's tolerances.  And a call must not take longer than the same one on larger matrices."""
import numpy as np
import pytest

from tests.helpers import relfro, tol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def slab(bf, prec, X):
    return (bf.DMatBatch if prec == "d" else bf.SMatBatch)(X.shape[1], X.shape[2], X.shape[0]).pack_all(X)


@pytest.mark.parametrize("prec", ["d", "s"])
@pytest.mark.parametrize("unit", [False, True])
@pytest.mark.parametrize("m,n,batch,off", [(1, 49, 160, 0), (31, 64, 170, 1), (32, 112, 160, 0), (7, 113, 160, 4),
                                           (33, 50, 160, 2), (64, 96, 150, 0), (65, 97, 80, 3), (20, 176, 150, 0),
                                           (3, 177, 150, 1), (40, 160, 150, 4)])
def test_sizes(bf, prec, unit, m, n, batch, off):
    rng = np.random.default_rng(m * 1000 + n)
    f32 = lambda X: X.astype(np.float32).astype(np.float64) if prec == "s" else X  # noqa: E731
    L = np.tril(rng.uniform(-1, 1, (batch, n + off, n + off)) / np.sqrt(n))
    L[:, np.arange(n + off), np.arange(n + off)] = rng.uniform(1, 2, (batch, n + off))
    L, R = f32(L), f32(rng.standard_normal((batch, m, n)))
    Lg = L.copy()
    Lg[:, np.triu(np.ones((n + off, n + off), bool), 0 if unit else 1)] = np.nan  # not read
    sA, sB, sD = slab(bf, prec, Lg), slab(bf, prec, R), slab(bf, prec, np.zeros((batch, m, n)))
    f = getattr(bf.lib, "blasfeo_%strsm_rlt%s_batch" % (prec, "u" if unit else "n"))
    assert f(batch, m, n, 1.5, sA.ref, off, off, sB.ref, 0, 0, sD.ref, 0, 0, None) == 0
    X = sD.unpack_all()
    for i in (0, batch // 2, batch - 1):
        T = L[i, off:, off:].copy()
        if unit:
            np.fill_diagonal(T, 1.0)
        assert relfro(X[i], np.linalg.solve(T, 1.5 * R[i].T).T) <= tol(prec, 1), i


def test_time_grows_with_n(bf):
    import torch

    def time(n, m=8, batch=4000):
        A, B, D = bf.SMatBatch(n, n, batch), bf.SMatBatch(m, n, batch), bf.SMatBatch(m, n, batch)
        A.buf.zero_()
        B.buf.zero_()
        ts = []
        for _ in range(7):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            assert bf.lib.blasfeo_strsm_rltn_batch(batch, m, n, 1.0, A.ref, 0, 0, B.ref, 0, 0, D.ref, 0, 0, None) == 0
            e[1].record()
            torch.cuda.synchronize()
            ts.append(e[0].elapsed_time(e[1]))
        return sorted(ts)[3]

    assert time(176) < 1.2 * time(192)
