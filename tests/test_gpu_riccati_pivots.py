"""Batched Riccati factorization, both slab layouts, with pivots that the fragment panels hand to the row form or mark:
exact zeros at even and odd places of a pair, infinite, NaN and subnormal pivots.  Against the recursion with the
library's pivot rule (c > 0 -> sqrt(c) and its reciprocal, else 0 and 0) in numpy (1e-13, the FP64 bar of every
routine).  info names the first pivot that is not positive; an infinite one counts back to back, where L_jj is NaN,
and not interleaved, where the pivot is looked at."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import relfro

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
N = 2


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def chol(S):
    n, S = len(S), S.copy()
    L, inv = np.zeros((n, n)), np.zeros(n)
    for j in range(n):
        c = S[j, j]
        if c > 0:
            inv[j] = 1.0 / np.sqrt(c)
            L[j, j] = c * inv[j]
        L[j + 1:, j] = S[j + 1:, j] * inv[j]
        S[j + 1:, j + 1:] -= np.outer(L[j + 1:, j], L[j + 1:, j])
    return L, inv


def recursion(BA, RSQ, nx, nu):
    """L_k, 1 / L_jj and the two info values of one problem."""
    out, info, m = {}, [0, 0], nx + nu
    for k in range(N, -1, -1):
        S = RSQ[k, :nx, :nx] if k == N else RSQ[k, :m, :m]
        if k < N:
            Lx = out[k + 1][0][-nx:, -nx:]
            W = np.array([[sum(BA[k, i, l] * Lx[l, j] for l in range(j, nx)) for j in range(nx)] for i in range(m)])
            S = S + W @ W.T
        S = np.tril(S) + np.tril(S, -1).T
        with np.errstate(all="ignore"):
            out[k] = chol(S)
        L, inv = out[k]
        for w in range(2):
            bad = [j for j in range(len(L)) if (not L[j, j] > 0 if w == 0 else inv[j] == 0 and L[j, j] == 0)]
            if bad and not info[w]:
                info[w] = 16 * (N - k) + bad[0] + 1
    return out, info


@pytest.mark.parametrize("nx,nu", [(5, 2), (8, 8), (12, 4), (11, 1)])
def test_pivots(bf, nx, nu):
    import torch
    m, rng = nx + nu, np.random.default_rng(nx)
    nbt = 12
    BA = rng.standard_normal((nbt, N, 16, nx)) / np.sqrt(nx)
    G = rng.standard_normal((nbt, N + 1, m, m))
    RSQ = np.zeros((nbt, N + 1, 16, 16))
    RSQ[:, :, :m, :m] = G @ G.transpose(0, 1, 3, 2) / m + np.eye(m)
    j = min(nx, 10) - 1
    RSQ[1, N, j, j] = np.inf                       # then every later stage is NaN
    RSQ[2, 0, 3, 3] = np.inf                       # last stage: the others of it stay finite
    RSQ[3, 0, m - 1, m - 1] = np.inf
    for p, z in ((4, 0), (5, 1), (6, j), (7, min(j, 2))):  # exact zeros
        RSQ[p, N, z, :] = RSQ[p, N, :, z] = 0.0
    RSQ[8, 0, 2, 1] = np.nan
    RSQ[9] = np.ldexp(RSQ[9], -1040)               # subnormal
    RSQ[10, 0, 1, 1] = -np.inf
    RSQ[11, 0, 3, 2] = np.inf                      # off the diagonal: pivot 3 becomes -inf
    slab = lambda X: bf.DMatBatch(X.shape[-2], X.shape[-1], X.shape[0] * X.shape[1]).pack_all(  # noqa: E731
        X.reshape((-1,) + X.shape[2:]))
    sBA, sRSQ, sL = slab(BA), slab(RSQ), bf.DMatBatch(16, 16, nbt * (N + 1))
    info, iinfo = (torch.full((nbt,), -9, dtype=torch.int32, device="cuda") for _ in range(2))
    assert bf.lib.blasfeo_dric_trf_batch(nbt, N, nx, nu, sBA.ref, sRSQ.ref, sL.ref, P(info), None) == 0
    bs = 16
    stage = lambda X: np.concatenate([np.concatenate([X[:, k], np.zeros((bs - nbt,) + X.shape[2:])])  # noqa: E731
                                      for k in range(X.shape[1])])
    il = lambda X: bf.DMatBatchIL(X.shape[1], X.shape[2], X.shape[0]).pack_all(X)  # noqa: E731
    iBA, iRSQ, iL = il(stage(BA)), il(stage(RSQ)), bf.DMatBatchIL(16, 16, (N + 1) * bs)
    assert bf.lib.blasfeo_dric_trf_batch_il(nbt, N, nx, nu, iBA.ref, iRSQ.ref, iL.ref, P(iinfo), None) == 0
    torch.cuda.synchronize()
    L, dA = sL.unpack_all().reshape(nbt, N + 1, 16, 16), sL.diag_all(16).reshape(nbt, N + 1, 16)
    Li = iL.unpack_all().reshape(N + 1, bs, 16, 16)
    ref = [recursion(BA[p], RSQ[p], nx, nu) for p in range(nbt)]
    assert info.cpu().tolist() == [r[1][0] for r in ref]
    assert iinfo.cpu().tolist() == [r[1][1] for r in ref]
    for p in range(nbt):
        # subnormal pivots: about 34 bits left
        tol, scale = (1e-9, 2.0 ** 520) if p == 9 else (1e-13, 1.0)
        for k in range(N + 1):
            R, inv = ref[p][0][k]
            mm = len(R)
            for X in (L[p, k, :mm, :mm], Li[k, p, :mm, :mm]):
                X = np.tril(X)
                ok = np.isfinite(np.tril(R))
                assert np.array_equal(np.isfinite(X), ok), (p, k)
                assert relfro(np.where(ok, X, 0) * scale, np.where(ok, np.tril(R), 0) * scale) <= tol, (p, k)
            d = dA[p, k, :mm]
            assert np.array_equal(d == 0, inv == 0) and not np.signbit(d[inv == 0]).any(), (p, k)
            assert relfro(d / scale, inv / scale) <= tol, (p, k)
