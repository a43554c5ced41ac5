"""FP64 geqrf: the last row has no reflector (tau = 0) whatever its column holds, so a last column of infinities or NaN
leaves the columns right of it alone; against the oracle (1e-13, the FP64 bar of every routine)."""
import numpy as np
import pytest

from tests.helpers import oracle_api, relfro

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


@pytest.mark.parametrize("m,n", [(3, 5), (16, 16), (16, 20), (17, 30), (64, 70), (100, 130), (300, 320)])
@pytest.mark.parametrize("value", [np.inf, np.nan])
def test_last_row_has_no_reflector(bf, m, n, value):
    rng = np.random.default_rng(m)
    A = rng.uniform(-1, 1, (2, m, n))
    B = A.copy()
    B[0, :, m - 1] = value  # the last column with a row on the diagonal
    c, d = bf.DMatBatch(m, n, 2).pack_all(B), bf.DMatBatch(m, n, 2)
    assert bf.lib.blasfeo_dgeqrf_batch(2, m, n, c.ref, 0, 0, d.ref, 0, 0, None) == 0
    F, tau = d.unpack_all(), d.diag_all(m)
    from oracle.pyoracle import HostMat
    for i in range(2):
        h, o = HostMat(m, n).set(A[i]), HostMat(m, n)
        oracle_api().geqrf("d", m, n, h, 0, 0, o, 0, 0)
        R, t = o.get(), o.diag(m)
        assert tau[i, m - 1] == 0 and t[m - 1] == 0
        assert relfro(tau[i], t) <= 1e-13
        keep = [j for j in range(n) if i == 1 or j != m - 1]
        assert relfro(F[i][:, keep], R[:, keep]) <= 1e-13
        if i == 0:
            assert not np.isfinite(F[0, :, m - 1]).any()
