"""FP32 potrf_l and syrk_potrf_ln: an infinite pivot counts in info on both sides of n = 64 (L_jj is NaN, 1 / L_jj 0),
and the rest of its matrix, which it does not reach, is factored."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


@pytest.mark.parametrize("n", [1, 8, 17, 40, 64, 65, 100])
@pytest.mark.parametrize("fused", [False, True])
def test_infinite_pivot_fp32(bf, n, fused):
    import torch
    js = sorted({0, n // 2, n - 1})
    A = np.repeat(np.eye(n)[None] * 4.0, len(js) + 1, 0)
    for i, j in enumerate(js):
        A[i, j, j] = np.inf
    b = len(A)
    c, d, k = bf.SMatBatch(n, n, b).pack_all(A), bf.SMatBatch(n, n, b), bf.SMatBatch(n, 3, b).pack_all(np.zeros((b, n, 3)))
    info = torch.full((b,), -9, dtype=torch.int32, device="cuda")
    if fused:
        st = bf.lib.blasfeo_ssyrk_spotrf_ln_batch(b, n, 3, k.ref, 0, 0, k.ref, 0, 0, c.ref, 0, 0, d.ref, 0, 0, P(info), None)
    else:
        st = bf.lib.blasfeo_spotrf_l_batch(b, n, c.ref, 0, 0, d.ref, 0, 0, P(info), None)
    assert st == 0
    L, inv = np.tril(d.unpack_all()), d.diag_all(n)
    assert info.cpu().tolist() == [j + 1 for j in js] + [0]
    for i, j in enumerate(js):
        assert np.isnan(L[i, j, j]) and inv[i, j] == 0
        L[i, j, j] = 2.0
        assert np.array_equal(L[i], 2.0 * np.eye(n))
