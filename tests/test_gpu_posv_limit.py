"""The largest systems of the plain solver's global-memory kernel: max_n at its limit is solved, one more is refused
with ENOTSUP and nothing is written (the small systems of the call included).  The limit is what the panel, the
diagonal block and the right-hand side leave of 227 KB: n = 1591."""
import numpy as np
import pytest

from tests.helpers import relfro
from tests.test_gpu_posv_edges import batch, solve

pytestmark = pytest.mark.gpu
LIMIT, ENOTSUP = 1591, 4


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def systems(ns):
    rng = np.random.default_rng(ns[0])
    mats = []
    for n in ns:
        G = rng.standard_normal((n, n))
        mats.append(G @ G.T / n + np.eye(n))
    return mats, [rng.standard_normal(n) for n in ns]


@pytest.mark.parametrize("n", [1589, 1590, LIMIT])
def test_at_the_limit(bf, n):
    ns = [n, 20, n - 1, 100]
    mats, rhs = systems(ns)
    x, info = solve(bf, batch(ns, mats, rhs), ns, False)
    assert (info == 0).all()
    for i in range(len(ns)):
        assert relfro(x[i], np.linalg.solve(mats[i], rhs[i])) <= 1e-13, ns[i]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [LIMIT + 1, 1640, 1680, 1700])
def test_beyond(bf, mixed, n):
    import ctypes as C
    import torch
    ns = [n, 20]
    mats, rhs = systems(ns)
    W = batch(ns, mats, rhs)
    W.x.fill_(7.0)
    P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    if mixed:
        st = bf.lib.blasfeo_dsposv_l_vbatch(2, P(W.nvec), n, P(W.desc), P(W.bdesc), P(W.xdesc), 30, 1e-14, None, None,
                                            None, None, 0, None)
    else:
        st = bf.lib.blasfeo_dposv_l_vbatch(2, P(W.nvec), n, P(W.desc), P(W.bdesc), P(W.xdesc), None, None, 0, None)
    assert st == ENOTSUP
    torch.cuda.synchronize()
    assert (W.x == 7.0).all() and bf.lib.blasfeo_b200_last_error() == 0
