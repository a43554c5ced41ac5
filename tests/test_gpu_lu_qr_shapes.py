"""FP64 getrf (with and without pivoting) and geqrf by the built-in rule at flat, wide and tiny shapes, uniform batches on
both sides of its lines, and beyond the 512 rows of the register panels; against the oracle (1e-13, the FP64 bar of
every routine)."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import oracle_api, relfro

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
SHAPES = [(2, 4, 3), (2, 9, 3), (3, 3, 3), (3, 8, 3), (3, 9, 700), (4, 48, 3), (4, 49, 3), (4, 257, 3), (6, 16, 3),
          (6, 17, 3), (8, 90, 160), (7, 300, 2), (9, 60, 2), (16, 353, 2), (17, 103, 3), (20, 140, 2), (30, 1, 700),
          (48, 2, 1300), (33, 240, 160), (48, 288, 160), (66, 260, 150), (40, 290, 2), (65, 460, 2), (130, 210, 150),
          (260, 370, 150), (129, 1300, 2), (513, 40, 2), (530, 530, 2), (600, 20, 3), (40, 600, 2)]


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def host(A):
    from oracle.pyoracle import HostMat
    return HostMat(*A.shape).set(A), HostMat(*A.shape)


def some(b):
    return sorted({0, b // 2, b - 1})


@pytest.mark.parametrize("m,n,batch", SHAPES)
def test_getrf(bf, m, n, batch):
    import torch
    rng = np.random.default_rng(m * 1000 + n)
    A, k = rng.uniform(-1, 1, (batch, m, n)), min(m, n)
    c, d = bf.DMatBatch(m, n, batch).pack_all(A), bf.DMatBatch(m, n, batch)
    piv = torch.full((batch, k), -1, dtype=torch.int32, device="cuda")
    info = torch.full((batch,), -9, dtype=torch.int32, device="cuda")
    assert bf.lib.blasfeo_dgetrf_rp_batch(batch, m, n, c.ref, 0, 0, d.ref, 0, 0, P(piv), P(info), None) == 0
    F, piv = d.unpack_all(), piv.cpu().numpy()
    assert (info.cpu().numpy() == 0).all()
    for i in some(batch):
        h, o = host(A[i])
        p = np.asarray(oracle_api().getrf_rp("d", m, n, h, 0, 0, o, 0, 0))[:k]
        assert np.array_equal(piv[i], p) and relfro(F[i], o.get()) <= 1e-13
    # without pivoting: dominant diagonals, against the factors multiplied out
    A[:, np.arange(k), np.arange(k)] += 2.0 * max(m, n)
    c.pack_all(A)
    info.fill_(-9)
    assert bf.lib.blasfeo_dgetrf_np_batch(batch, m, n, c.ref, 0, 0, d.ref, 0, 0, P(info), None) == 0
    F, inv = d.unpack_all(), d.diag_all(k)
    assert (info.cpu().numpy() == 0).all()
    for i in some(batch):
        L, U = np.tril(F[i], -1)[:, :k], np.triu(F[i])[:k]
        L[np.arange(k), np.arange(k)] = 1.0
        assert relfro(L @ U, A[i]) <= 1e-13
        assert np.array_equal(inv[i], 1.0 / np.diagonal(F[i])[:k])


@pytest.mark.parametrize("m,n,batch", SHAPES)
def test_geqrf(bf, m, n, batch):
    rng = np.random.default_rng(m * 1000 + n + 1)
    A, k = rng.uniform(-1, 1, (batch, m, n)), min(m, n)
    c, d = bf.DMatBatch(m, n, batch).pack_all(A), bf.DMatBatch(m, n, batch)
    assert bf.lib.blasfeo_dgeqrf_batch(batch, m, n, c.ref, 0, 0, d.ref, 0, 0, None) == 0
    F, tau = d.unpack_all(), d.diag_all(k)
    for i in some(batch):
        h, o = host(A[i])
        oracle_api().geqrf("d", m, n, h, 0, 0, o, 0, 0)
        assert relfro(F[i], o.get()) <= 1e-13 and relfro(tau[i], o.diag(k)) <= 1e-13
