"""The reciprocal square root of the fragment Cholesky's pivots and its exact zeros.  The inverse pivot of a 1 x 1 potrf_l
is that root itself: against the 80-bit value and CUDA's rsqrt over the normal range, with a bound of 2 ulp (the
approximation's 2^-20 enters with its third power; what remains are the roundings of c y, of the product with it and of
the sum: 1.5 units of 2^-53).  Subnormal and infinite pivots leave no finite root there and go to the row form.  Zero
pivots, at even and odd places of a pair and both, give L_jj = dA_j = 0, info = j + 1 and leave the other rows' factor."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import relfro, tol

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def potrf(bf, prec, A):
    import torch
    b, n, _ = A.shape
    B = bf.DMatBatch if prec == "d" else bf.SMatBatch
    c, d = B(n, n, b).pack_all(A), B(n, n, b)
    info = torch.full((b,), -9, dtype=torch.int32, device="cuda")
    assert getattr(bf.lib, "blasfeo_%spotrf_l_batch" % prec)(b, n, c.ref, 0, 0, d.ref, 0, 0, P(info), None) == 0
    return np.tril(d.unpack_all()), d.diag_all(n), info.cpu().numpy()


@pytest.mark.parametrize("lo,hi", [(-1022, -1000), (-1000, -10), (-2, 2), (10, 1000), (1000, 1024)])
def test_rsqrt(bf, lo, hi):
    import torch
    rng = np.random.default_rng(abs(hi))
    c = np.ldexp(rng.uniform(1, 2, 300000), rng.integers(lo, hi, 300000))
    edge = np.array([1.0, np.nextafter(1.0, 2), np.nextafter(2.0, 1), 2.0, np.nextafter(2.0, 3), 3.0, np.nextafter(4.0, 3)])
    e = np.ldexp(edge[:, None], np.arange(lo, hi - 1)[None] if lo >= -1000 else np.arange(lo, hi)[None]).ravel()
    c = np.concatenate([c, e[np.isfinite(e)], [np.finfo(float).tiny, np.finfo(float).max]])
    L, inv, info = potrf(bf, "d", c.reshape(-1, 1, 1))
    inv, L = inv.ravel(), L.ravel()
    assert (info == 0).all()
    exact = 1 / np.sqrt(c.astype(np.longdouble))
    assert (np.abs(inv.astype(np.longdouble) - exact) <= 2 * np.spacing(exact.astype(float))).all()
    cuda = torch.rsqrt(torch.from_numpy(c).cuda()).cpu().numpy()
    assert (np.abs(inv - cuda) <= 2 * np.spacing(cuda)).all()
    # L = c times it, with one more rounding
    assert (np.abs(L.astype(np.longdouble) - np.sqrt(c.astype(np.longdouble))) <= 3 * np.spacing(np.sqrt(c))).all()


def test_rsqrt_outside_the_normal_range(bf):
    c = np.concatenate([[5e-324, 1e-320, np.nextafter(np.finfo(float).tiny, 0)], [np.inf, 0.0, -1.0, np.nan]])
    L, inv, info = potrf(bf, "d", c.reshape(-1, 1, 1))
    inv, L = inv.ravel(), L.ravel()
    assert info.tolist() == [0, 0, 0, 0, 1, 1, 1]
    exact = 1 / np.sqrt(c[:3].astype(np.longdouble))
    assert (np.abs(inv[:3].astype(np.longdouble) - exact) <= 2 * np.spacing(exact.astype(float))).all()
    assert (inv[3:] == 0).all() and np.isnan(L[3]) and (L[4:] == 0).all()


@pytest.mark.parametrize("prec", ["d", "s"])
@pytest.mark.parametrize("n", [5, 16, 40, 64, 65, 100, 161])
def test_exact_zeros(bf, prec, n):
    rng = np.random.default_rng(n)
    G = rng.standard_normal((n, n))
    A0 = G @ G.T / n + np.eye(n)
    A0 = A0.astype(np.float32).astype(np.float64) if prec == "s" else A0
    sets = [(0,), (1,), (0, 1), (2, 3), (n // 2,), (n - 1,), (n - 2, n - 1), (1, 2), tuple(range(n))]
    A = np.repeat(A0[None], len(sets), 0)
    for i, z in enumerate(sets):
        A[i, list(z)] = 0.0
        A[i, :, list(z)] = 0.0
    L, inv, info = potrf(bf, prec, A)
    for i, z in enumerate(sets):
        keep = np.setdiff1d(np.arange(n), z)
        assert info[i] == z[0] + 1
        assert not L[i, list(z)].any() and not L[i][:, list(z)].any() and not inv[i, list(z)].any()
        if len(keep):
            ref = np.linalg.cholesky(A0[np.ix_(keep, keep)])
            assert relfro(L[i][np.ix_(keep, keep)], ref) <= tol(prec)
            assert relfro(inv[i, keep], 1 / np.diagonal(ref)) <= tol(prec)
