"""FP64 geqrf with register panels at the edges: sizes around the panels, column
chunks, lanes per column and threads per matrix, tall, square and wide blocks,
odd row offsets, in place, zero columns, size classes of uneven launches;
against the oracle (1e-13, the FP64 bar of every routine)."""
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


def oracle_qr(A):
    from oracle.pyoracle import HostMat
    m, n = A.shape
    h, d = HostMat(m, n).set(A), HostMat(m, n)
    oracle_api().geqrf("d", m, n, h, 0, 0, d, 0, 0)
    return d.get(), d.diag(min(m, n))


def run(bf, mats, variant, in_place=False):
    import torch
    b = len(mats)
    src = [bf.DMat(*A.shape).pack(A) for A in mats]
    dst = src if in_place else [bf.DMat(*A.shape) for A in mats]
    dims = lambda i: torch.tensor([A.shape[i] for A in mats], dtype=torch.int32, device="cuda")
    mv, nv = dims(0), dims(1)
    assert bf.lib.blasfeo_dgeqrf_vbatch_variant(b, P(mv), P(nv), int(mv.max()), int(nv.max()),
                                                P(bf.descriptor_array(src)), P(bf.descriptor_array(dst)), variant,
                                                None) == 0
    torch.cuda.synchronize()
    return dst


def check(bf, mats, variant, in_place=False):
    for i, (d, A) in enumerate(zip(run(bf, mats, variant, in_place), mats)):
        ref, tau = oracle_qr(A)
        assert relfro(d.unpack(), ref) <= 1e-13, (i, A.shape)
        assert relfro(d.diag_array(min(A.shape)), tau) <= 1e-13, (i, A.shape)


@pytest.mark.parametrize("variant", [-1, 0, 1, 2])
@pytest.mark.parametrize("shape", [(1, 1), (2, 1), (7, 3), (16, 16), (17, 16), (31, 20), (32, 48), (33, 17), (64, 33),
                                   (65, 65), (20, 100), (127, 50), (129, 40), (200, 97), (256, 128), (257, 30),
                                   (384, 64), (385, 20), (512, 49), (100, 300)])
def test_shapes(bf, shape, variant):
    rng = np.random.default_rng(shape[0] * 1000 + shape[1])
    check(bf, [rng.uniform(-1, 1, shape) for _ in range(2)], variant, in_place=variant == 0)


@pytest.mark.parametrize("top", [40, 96, 150])
def test_uneven(bf, top):
    rng = np.random.default_rng(top)
    ns = [1, top, 2, 5, 16, 33, top // 2, top // 4, top // 4 + 1, 3 * top // 4, top - 1]
    check(bf, [rng.uniform(-1, 1, (2 * n, n)) for n in ns], -1)


@pytest.mark.parametrize("off", [(1, 2), (4, 1), (2, 0)])
def test_offsets(bf, off):
    """A block at an offset of a larger matrix, single instance: the rest is not touched."""
    rng = np.random.default_rng(off[0])
    ai, aj = off
    m, n = 70, 41
    A = rng.uniform(-1, 1, (m + ai + 3, n + aj + 2))
    d = bf.DMat(*A.shape).pack(A)
    bf.blasfeo_dgeqrf(m, n, d, ai, aj, d, ai, aj)
    got = d.unpack()
    ref, tau = oracle_qr(A[ai:ai + m, aj:aj + n])
    assert relfro(got[ai:ai + m, aj:aj + n], ref) <= 1e-13
    assert relfro(d.diag_array(ai + n)[ai:], tau) <= 1e-13
    got[ai:ai + m, aj:aj + n] = A[ai:ai + m, aj:aj + n]
    assert np.array_equal(got, A)


def test_zero_columns_and_nan(bf):
    rng = np.random.default_rng(3)
    z = rng.uniform(-1, 1, (60, 40))
    z[5:, 5] = z[:, 20] = 0.0
    z[:, :5] = np.triu(z[:, :5])  # no reflector in the first columns
    nan = rng.uniform(-1, 1, (60, 40))
    nan[7, 30] = np.nan
    out = run(bf, [z, nan], -1)
    ref, tau = oracle_qr(z)
    assert relfro(out[0].unpack(), ref) <= 1e-13 and relfro(out[0].diag_array(40), tau) <= 1e-13
    assert not out[0].diag_array(40)[:6].any()
    clean, ctau = oracle_qr(nan[:, :30])
    # the columns before the one with the NaN do not see it
    assert relfro(out[1].unpack()[:, :30], clean) <= 1e-13 and relfro(out[1].diag_array(40)[:30], ctau) <= 1e-13
