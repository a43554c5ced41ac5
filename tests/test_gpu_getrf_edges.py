"""FP64 getrf with register panels at the edges: sizes around the panels, warps and
threads per matrix, tall and wide blocks, every thread count, ties, zero, NaN
and infinite columns, in place, size classes of uneven launches; pivots equal
to and factors within 1e-13 of the oracle's."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import oracle_api, relfro

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


def oracle_lu(A):
    from oracle.pyoracle import HostMat
    m, n = A.shape
    h, d = HostMat(m, n).set(A), HostMat(m, n)
    piv = oracle_api().getrf_rp("d", m, n, h, 0, 0, d, 0, 0)
    return d.get(), np.asarray(piv)[: min(m, n)]


def run(bf, mats, variant, in_place=False):
    import torch
    b = len(mats)
    src = [bf.DMat(*A.shape).pack(A) for A in mats]
    dst = src if in_place else [bf.DMat(*A.shape) for A in mats]
    dims = lambda i: torch.tensor([A.shape[i] for A in mats], dtype=torch.int32, device="cuda")
    mv, nv = dims(0), dims(1)
    maxm, maxn = int(mv.max()), int(nv.max())
    st = min(maxm, maxn)
    piv = torch.full((b, st), -1, dtype=torch.int32, device="cuda")
    info = torch.full((b,), -9, dtype=torch.int32, device="cuda")
    assert bf.lib.blasfeo_dgetrf_rp_vbatch_variant(b, P(mv), P(nv), maxm, maxn, P(bf.descriptor_array(src)),
                                                   P(bf.descriptor_array(dst)), P(piv), st, P(info), variant, None) == 0
    torch.cuda.synchronize()
    return dst, piv.cpu().numpy(), info.cpu().numpy()


def check(bf, mats, variant, in_place=False):
    dst, piv, info = run(bf, mats, variant, in_place)
    for i, A in enumerate(mats):
        ref, rp = oracle_lu(A)
        k = min(A.shape)
        assert np.array_equal(piv[i, :k], rp), (i, A.shape)
        assert relfro(dst[i].unpack(), ref) <= 1e-13, (i, A.shape)
        # dA is the reciprocal of the pivots as stored (how far a small pivot is
        # from the oracle's is its conditioning's, not the routine's)
        assert np.array_equal(dst[i].diag_array(k), 1.0 / np.diagonal(dst[i].unpack())[:k]), (i, A.shape)
        assert info[i] == 0


@pytest.mark.parametrize("variant", [-1, 0, 1, 2])
@pytest.mark.parametrize("shape", [(1, 1), (3, 7), (15, 15), (16, 17), (17, 16), (31, 40), (32, 32), (33, 5), (64, 64),
                                   (65, 130), (127, 128), (129, 129), (200, 33), (256, 100), (257, 257), (130, 300),
                                   (511, 40), (512, 64)])
def test_shapes(bf, shape, variant):
    rng = np.random.default_rng(shape[0] * 1000 + shape[1])
    check(bf, [rng.uniform(-1, 1, shape) for _ in range(2)], variant, in_place=variant == 0)


@pytest.mark.parametrize("top", [65, 190, 300])
def test_uneven(bf, top):
    rng = np.random.default_rng(top)
    ns = [1, top, 2, 5, 16, 33, top // 2, top // 4, top // 4 + 1, 3 * top // 4, top - 1, 48]
    check(bf, [rng.uniform(-1, 1, (n, n)) for n in ns], -1)


@pytest.mark.parametrize("n", [20, 70, 140])
def test_ties_zero_columns_and_nan(bf, n):
    rng = np.random.default_rng(n)
    ties = rng.choice([-1.0, 0.0, 1.0], (n, n)) + 2.0 * np.eye(n)[::-1]
    ref, rp = oracle_lu(ties)
    zero = rng.uniform(-1, 1, (n, n))
    zero[:, 3] = 0.0
    nan = rng.uniform(-1, 1, (n, n))
    nan[:, n - 2] = np.nan  # the column in which every candidate is NaN: the row stays
    dst, piv, info = run(bf, [ties, zero, nan], -1)
    assert np.array_equal(piv[0], rp) and relfro(dst[0].unpack(), ref) <= 1e-13
    zref, zp = oracle_lu(zero)
    assert np.array_equal(piv[1], zp) and relfro(dst[1].unpack(), zref) <= 1e-13 and info[1] == 4
    clean = np.nan_to_num(nan)
    cref, cp = oracle_lu(clean)
    assert np.array_equal(piv[2, : n - 2], cp[: n - 2]) and piv[2, n - 2] == n - 2
    assert relfro(dst[2].unpack()[:, : n - 2][: n - 2], cref[:, : n - 2][: n - 2]) <= 1e-13
