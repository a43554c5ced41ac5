"""syrk_potrf_ln (fused for m <= 64) and trsm_rltn / rltu on uniform batches at the
edges of their kernels: sizes around blocks of 8 and 16, every launch rule of
the solve, row offsets off the panel grid, k = 0, A and B equal or not, bad
pivots; against numpy in FP64 with the repository's tolerances (1e-13 FP64, 2e-5
FP32 relative Frobenius)."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import relfro, tol

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def slab(bf, prec, X):
    B = bf.DMatBatch if prec == "d" else bf.SMatBatch
    return B(X.shape[1], X.shape[2], X.shape[0]).pack_all(X)


def f32(prec, X):
    return X.astype(np.float32).astype(np.float64) if prec == "s" else X


@pytest.mark.parametrize("prec", ["d", "s"])
@pytest.mark.parametrize("same", [True, False])
@pytest.mark.parametrize("n,k,off", [(1, 1, 0), (5, 0, 0), (8, 8, 0), (9, 7, 1), (16, 33, 4), (23, 9, 0), (32, 16, 3),
                                     (40, 17, 0), (47, 40, 4), (50, 37, 0), (57, 5, 2), (64, 64, 0), (65, 20, 0)])
def test_syrk_potrf(bf, prec, same, n, k, off):
    import torch
    rng = np.random.default_rng(100 * n + k)
    b = 5
    A = f32(prec, rng.standard_normal((b, n + off, max(k, 1) + 1)))
    # B near A keeps C + A B^T positive definite
    B = A if same else f32(prec, A + 0.01 * rng.standard_normal(A.shape))
    G = rng.standard_normal((b, n + off, n + off + 1))
    Cm = f32(prec, G @ G.transpose(0, 2, 1) / n + 3 * np.eye(n + off))
    sA, sC, sD = slab(bf, prec, A), slab(bf, prec, Cm), slab(bf, prec, np.zeros_like(Cm))
    sB = sA if same else slab(bf, prec, B)
    info = torch.full((b,), -9, dtype=torch.int32, device="cuda")
    f = getattr(bf.lib, "blasfeo_%ssyrk_%spotrf_ln_batch" % (prec, prec))
    assert f(b, n, k, sA.ref, off, 1 if k else 0, sB.ref, off, 1 if k else 0, sC.ref, off, off, sD.ref, off, off, P(info),
             None) == 0
    torch.cuda.synchronize()
    L = sD.unpack_all().astype(np.float64)
    assert (info == 0).all()
    j = 1 if k else 0
    for i in range(b):
        S = np.tril(Cm[i, off:, off:] + A[i, off:, j:j + k] @ B[i, off:, j:j + k].T)
        ref = np.linalg.cholesky(S + np.tril(S, -1).T)
        assert relfro(np.tril(L[i, off:, off:]), ref) <= tol(prec), i
        assert not L[i, :off].any() and not np.triu(L[i, off:, off:], 1).any()
        if off == 0:
            assert relfro(sD.diag_all(n)[i], 1 / np.diagonal(ref)) <= tol(prec)


@pytest.mark.parametrize("prec", ["d", "s"])
@pytest.mark.parametrize("n", [7, 64])
def test_syrk_potrf_bad_and_infinite(bf, prec, n):
    import torch
    rng = np.random.default_rng(n)
    A = f32(prec, rng.standard_normal((3, n, 4)))
    Cm = np.repeat(2.0 * np.eye(n)[None], 3, 0)
    Cm[1, 4, 4] = -100.0
    Cm[2, 2, 1] = np.inf  # reaches pivot 3 as -inf: the columns before it stay as they are
    sA, sC, sD = slab(bf, prec, A), slab(bf, prec, Cm), slab(bf, prec, np.zeros_like(Cm))
    info = torch.full((3,), -9, dtype=torch.int32, device="cuda")
    f = getattr(bf.lib, "blasfeo_%ssyrk_%spotrf_ln_batch" % (prec, prec))
    assert f(3, n, 4, sA.ref, 0, 0, sA.ref, 0, 0, sC.ref, 0, 0, sD.ref, 0, 0, P(info), None) == 0
    torch.cuda.synchronize()
    L = sD.unpack_all().astype(np.float64)
    assert info.tolist() == [0, 5, 3]
    ref = np.linalg.cholesky(2.0 * np.eye(n) + A[2] @ A[2].T)
    assert L[1, 4, 4] == 0
    assert relfro(L[2, :, :1], ref[:, :1]) <= tol(prec)


@pytest.mark.parametrize("prec", ["d", "s"])
@pytest.mark.parametrize("unit", [False, True])
@pytest.mark.parametrize("m,n,batch,off", [(1, 1, 3, 0), (5, 15, 200, 0), (33, 16, 200, 4), (64, 17, 170, 1),
                                           (65, 31, 160, 0), (20, 48, 200, 0), (40, 65, 3, 2), (100, 96, 160, 0),
                                           (70, 130, 100, 0), (33, 200, 3, 0), (70, 161, 80, 0)])
def test_trsm(bf, prec, unit, m, n, batch, off):
    import torch
    rng = np.random.default_rng(m * 1000 + n)
    L = np.tril(rng.uniform(-1, 1, (batch, n + off, n + off)) / np.sqrt(n))
    L[:, np.arange(n + off), np.arange(n + off)] = rng.uniform(1, 2, (batch, n + off))
    L = f32(prec, L)
    Lg = L.copy()
    Lg[:, np.triu(np.ones((n + off, n + off), bool), 0 if unit else 1)] = np.nan  # not read
    R = f32(prec, rng.standard_normal((batch, m, n)))
    sA, sB, sD = slab(bf, prec, Lg), slab(bf, prec, R), slab(bf, prec, np.zeros((batch, m, n)))
    f = getattr(bf.lib, "blasfeo_%strsm_rlt%s_batch" % (prec, "u" if unit else "n"))
    assert f(batch, m, n, 1.5, sA.ref, off, off, sB.ref, 0, 0, sD.ref, 0, 0, None) == 0
    # and in place
    assert f(batch, m, n, 1.5, sA.ref, off, off, sB.ref, 0, 0, sB.ref, 0, 0, None) == 0
    torch.cuda.synchronize()
    X, Y = sD.unpack_all(), sB.unpack_all()
    assert np.array_equal(X, Y)
    for i in sorted({0, batch // 2, batch - 1}):
        T = L[i, off:, off:].copy()
        if unit:
            np.fill_diagonal(T, 1.0)
        ref = np.linalg.solve(T, 1.5 * R[i].T).T
        assert relfro(X[i], ref) <= tol(prec, 1), i
