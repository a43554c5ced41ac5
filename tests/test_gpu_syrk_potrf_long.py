"""syrk_potrf_ln of a few matrices with a long k, on both sides of the rule that chooses between one kernel and two
launches: results against numpy in FP64, and no call much longer than syrk_ln and potrf_l called one after the other."""
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


def f32(prec, X):
    return X.astype(np.float32).astype(np.float64) if prec == "s" else X


@pytest.mark.parametrize("prec", ["d", "s"])
@pytest.mark.parametrize("batch,m,k", [(1, 64, 256), (1, 64, 257), (3, 41, 300), (2, 40, 300), (1, 48, 200), (1, 48, 201),
                                       (149, 50, 401), (75, 48, 210), (1, 49, 1000)])
def test_long_k(bf, prec, batch, m, k):
    import torch
    rng = np.random.default_rng(m + k)
    A = f32(prec, rng.standard_normal((batch, m, k)) / np.sqrt(k))
    Cm = f32(prec, np.repeat(2.0 * np.eye(m)[None], batch, 0))
    sA, sC, sD = slab(bf, prec, A), slab(bf, prec, Cm), slab(bf, prec, np.zeros_like(Cm))
    info = torch.full((batch,), -9, dtype=torch.int32, device="cuda")
    f = getattr(bf.lib, "blasfeo_%ssyrk_%spotrf_ln_batch" % (prec, prec))
    assert f(batch, m, k, sA.ref, 0, 0, sA.ref, 0, 0, sC.ref, 0, 0, sD.ref, 0, 0, info.data_ptr(), None) == 0
    L, inv = np.tril(sD.unpack_all().astype(np.float64)), sD.diag_all(m)
    assert (info.cpu().numpy() == 0).all()
    for i in {0, batch // 2, batch - 1}:
        ref = np.linalg.cholesky(Cm[i] + A[i] @ A[i].T)
        assert relfro(L[i], ref) <= tol(prec) and relfro(inv[i], 1 / np.diagonal(ref)) <= tol(prec)


@pytest.mark.parametrize("prec,m,k", [("d", 64, 2000), ("d", 48, 1000), ("s", 48, 1000), ("d", 40, 2000)])
def test_time(bf, prec, m, k):
    import torch
    A, Cm = slab(bf, prec, np.zeros((1, m, k))), slab(bf, prec, np.eye(m)[None])
    D = slab(bf, prec, np.zeros((1, m, m)))

    def time(f):
        ts = []
        for _ in range(9):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            for _ in range(10):
                f()
            e[1].record()
            torch.cuda.synchronize()
            ts.append(e[0].elapsed_time(e[1]))
        return sorted(ts)[4]

    one, syrk, potrf = (getattr(bf.lib, "blasfeo_%s_batch" % n.replace("?", prec))
                        for n in ("?syrk_?potrf_ln", "?syrk_ln", "?potrf_l"))

    def two():
        syrk(1, m, k, 1.0, A.ref, 0, 0, A.ref, 0, 0, 1.0, Cm.ref, 0, 0, D.ref, 0, 0, None)
        potrf(1, m, D.ref, 0, 0, D.ref, 0, 0, None, None)

    assert time(lambda: one(1, m, k, A.ref, 0, 0, A.ref, 0, 0, Cm.ref, 0, 0, D.ref, 0, 0, None, None)) < 1.1 * time(two)
