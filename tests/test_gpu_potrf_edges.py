"""FP64 potrf_l on uniform batches at the edges of the kernels' block grids, with
non-positive pivots at every position of a block, subnormal and infinite
pivots; against numpy's Cholesky (1e-13, the FP64 bar of every routine)."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import relfro

pytestmark = pytest.mark.gpu
SIZES = [1, 2, 3, 7, 8, 9, 16, 17, 24, 31, 33, 40, 41, 48, 49, 56, 57, 63, 64, 65, 72, 80, 81, 96, 113, 129, 161]


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def potrf(bf, A, in_place=False):
    import torch
    b, n, _ = A.shape
    c = bf.DMatBatch(n, n, b).pack_all(A)
    d = c if in_place else bf.DMatBatch(n, n, b)
    info = torch.full((b,), -9, dtype=torch.int32, device="cuda")
    assert bf.lib.blasfeo_dpotrf_l_batch(b, n, c.ref, 0, 0, d.ref, 0, 0, C.c_void_p(info.data_ptr()), None) == 0
    torch.cuda.synchronize()
    return np.tril(d.unpack_all()), d.diag_all(n), info.cpu().numpy()


def spd(rng, b, n):
    G = rng.standard_normal((b, n, n))
    return G @ G.transpose(0, 2, 1) / n + np.eye(n)


@pytest.mark.parametrize("n", SIZES)
def test_sizes(bf, n):
    A = spd(np.random.default_rng(n), 5, n)
    A[:, np.triu(np.ones((n, n), bool), 1)] = np.nan  # the upper part is not read
    for in_place in (False, True):
        L, d, info = potrf(bf, A, in_place)
        ref = np.linalg.cholesky(np.tril(A) + np.tril(A, -1).transpose(0, 2, 1))
        assert (info == 0).all()
        for k in range(5):
            assert relfro(L[k], ref[k]) <= 1e-13
            assert relfro(d[k], 1 / np.diagonal(ref[k])) <= 1e-13


@pytest.mark.parametrize("n", [9, 16, 40, 64, 80])
def test_bad_pivots(bf, n):
    """Pivot j made negative (zero for odd j): L_jj = dA_j = 0, info = j + 1, column j zero, the columns before it as
    of the clean matrix."""
    rng = np.random.default_rng(n)
    A = np.repeat(spd(rng, 1, n), n, axis=0)
    ref = np.linalg.cholesky(A[0])
    for j in range(n):
        s = ref[j, :j] @ ref[j, :j]
        A[j, j, j] = s - 1.0 if j % 2 == 0 or j > 0 else 0.0
    L, d, info = potrf(bf, A)
    assert np.array_equal(info, np.arange(1, n + 1))
    for j in range(n):
        assert L[j, j, j] == 0 and d[j, j] == 0 and (L[j, j:, j] == 0).all()
        assert relfro(L[j, :, :j], ref[:, :j]) <= 1e-13


@pytest.mark.parametrize("n", [1, 7, 20, 64, 72])
def test_pivots_outside_the_fast_range(bf, n):
    rng = np.random.default_rng(7 * n)
    A = spd(rng, 3, n)
    # subnormal pivots: about 34 bits left, each update rounds at 2^-1074, so
    # entries of order 2^-520 carry errors of a few times 2^-34
    A[1] = np.ldexp(A[1], -1040)
    ref = [np.linalg.cholesky(A[0]), np.ldexp(np.linalg.cholesky(np.ldexp(A[1], 1040)), -520)]
    A[2, 0, 0] = np.inf  # 1 / sqrt(inf) = 0: a positive pivot whose column is 0 (and NaN where inf meets it)
    L, d, info = potrf(bf, A)
    assert info[0] == 0 and info[1] == 0
    assert relfro(L[0], ref[0]) <= 1e-13
    assert relfro(np.ldexp(L[1], 520), np.ldexp(ref[1], 520)) <= 1e-9
    assert d[2, 0] == 0 and np.isnan(L[2, 0, 0])
    if n > 1:
        assert (L[2, 1:, 0] == 0).all()
