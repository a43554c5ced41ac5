"""FP64 gemm_nt and syrk_ln at the edges of the 64 x 64 and 32 x 32 tiles, of the 8 x 8 fragments and of the k steps:
uniform batches with row offsets, and uneven batches whose instances have more tiles than CTAs; against numpy (1e-13,
the FP64 bar of every routine).  What lies outside the result is not written."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import relfro

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (8, 9, 3), (33, 31, 16), (40, 72, 17), (64, 64, 15), (65, 57, 64),
                                   (97, 128, 5), (130, 3, 33)])
@pytest.mark.parametrize("off", [0, 1, 4])
@pytest.mark.parametrize("batch", [2, 400])
def test_uniform(bf, m, n, k, off, batch):
    rng = np.random.default_rng(m + n + k)
    A, B, S = (rng.uniform(-1, 1, (batch, r + 4, c)) for r, c in ((m, k), (n, k), (m, n)))
    a, b, c = (bf.DMatBatch(X.shape[1], X.shape[2], batch).pack_all(X) for X in (A, B, S))
    d = bf.DMatBatch(m + 4, n, batch).pack_all(np.full((batch, m + 4, n), 7.0))
    assert bf.lib.blasfeo_dgemm_nt_batch(batch, m, n, k, 1.5, a.ref, off, 0, b.ref, off, 0, -0.5, c.ref, off, 0, d.ref,
                                         off, 0, None) == 0
    D = d.unpack_all()
    ref = 1.5 * A[:, off: off + m] @ B[:, off: off + n].transpose(0, 2, 1) - 0.5 * S[:, off: off + m]
    assert relfro(D[:, off: off + m], ref) <= 1e-13
    assert (D[:, :off] == 7).all() and (D[:, off + m:] == 7).all()
    if m != n:
        return
    d.pack_all(np.full((batch, m + 4, n), 7.0))
    assert bf.lib.blasfeo_dsyrk_ln_batch(batch, m, k, 1.5, a.ref, off, 0, b.ref, off, 0, -0.5, c.ref, off, 0, d.ref, off,
                                         0, None) == 0
    D = d.unpack_all()[:, off: off + m]
    assert relfro(np.tril(D), np.tril(ref)) <= 1e-13
    assert (np.triu(D, 1) == np.triu(np.full((m, m), 7.0), 1)).all()


@pytest.mark.parametrize("seed", [0, 1])
def test_uneven(bf, seed):
    import torch
    rng = np.random.default_rng(seed)
    sizes = [(300, 260, 20), (257, 5, 65), (0, 8, 8), (8, 8, 0), (1, 300, 1)]
    sizes += [tuple(int(v) for v in rng.integers(1, 140, 3)) for _ in range(120)]
    A, B = [rng.uniform(-1, 1, (m, k)) for m, n, k in sizes], [rng.uniform(-1, 1, (n, k)) for m, n, k in sizes]
    mk = lambda X: bf.DMat(max(X.shape[0], 1), max(X.shape[1], 1)).pack(  # noqa: E731
        np.pad(X, [(0, max(1 - X.shape[0], 0)), (0, max(1 - X.shape[1], 0))]))
    a, b = [mk(X) for X in A], [mk(X) for X in B]
    d = [mk(np.full((m, n), 7.0)) for m, n, k in sizes]
    da, db, dd = (bf.descriptor_array(x) for x in (a, b, d))
    s = torch.tensor(sizes, dtype=torch.int32).t().contiguous().cuda()
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    mx = [max(v) for v in zip(*sizes)]
    assert bf.lib.blasfeo_dgemm_nt_vbatch(len(sizes), P(s[0]), P(s[1]), P(s[2]), *mx, 1.0, P(da), P(db), 0.0, P(dd),
                                          P(dd), None) == 0
    torch.cuda.synchronize()
    for i, (m, n, k) in enumerate(sizes):
        if m and n:
            D, ref = d[i].unpack(), A[i] @ B[i].T
            assert np.linalg.norm(D - ref) <= 1e-13 * max(np.linalg.norm(ref), 1e-300), sizes[i]
