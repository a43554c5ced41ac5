"""FP64 gemm_nt on uneven batches of many instances, whose tiles beyond an instance's first ones are taken from a list by
helper CTAs: sizes around the tiles, the fragments and the k slices, large instances at the ends of the batch and of the
groups of 128 that a helper looks at together, empty ones between; and syrk_ln / syrk_ln_mn of more tiles than one row
(the triangle's numbering).  Against numpy (1e-13, the FP64 bar of every routine); what lies outside the result is not
written."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import relfro

pytestmark = pytest.mark.gpu
P = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731


@pytest.fixture(scope="module")
def bf():
    import blasfeo_b200
    return blasfeo_b200


class Uneven:
    """Descriptors of instances (m, n, k) with operands cut from shared random matrices."""

    def __init__(self, bf, sizes, seed):
        import torch
        from blasfeo_b200.workloads import DESC_DTYPE, to_panel_major
        rng = np.random.default_rng(seed)
        self.bf, self.sizes = bf, sizes
        up = lambda x: (max(x, 1) + 3) // 4 * 4  # noqa: E731
        mx = [up(max(v)) for v in zip(*sizes)]
        self.A, self.B = rng.uniform(-1, 1, (mx[0], mx[2])), rng.uniform(-1, 1, (mx[1], mx[2]))
        self.src = [to_panel_major(torch.from_numpy(X)[None], *X.shape)[0].contiguous().cuda() for X in (self.A, self.B)]
        self.off = np.concatenate([[0], np.cumsum([up(m) * up(n) for m, n, k in sizes])])
        self.out = torch.full((int(self.off[-1]),), 7.0, dtype=torch.float64, device="cuda")

        def desc(pA, m, n, pm, cn):
            d = np.zeros(len(sizes), DESC_DTYPE)
            d["mem"], d["pA"], d["dA"], d["m"], d["n"], d["pm"], d["cn"] = pA, pA, pA, m, n, pm, cn
            return torch.from_numpy(d.view(np.uint8).copy()).cuda()
        m, n, k = (np.array(v) for v in zip(*sizes))
        self.d = [desc(self.src[0].data_ptr(), m, k, mx[0], mx[2]), desc(self.src[1].data_ptr(), n, k, mx[1], mx[2]),
                  desc(self.out.data_ptr() + 8 * self.off[:-1], m, n, [up(v) for v in m], [up(v) for v in n])]
        self.s = torch.tensor(sizes, dtype=torch.int32).t().contiguous().cuda()
        self.mx = [int(max(v)) for v in (m, n, k)]

    def run(self, variant=-1):
        assert self.bf.lib.blasfeo_dgemm_nt_vbatch_variant(
            len(self.sizes), P(self.s[0]), P(self.s[1]), P(self.s[2]), *self.mx, 1.0, P(self.d[0]), P(self.d[1]), 0.0,
            P(self.d[2]), P(self.d[2]), variant, None) == 0

    def check(self):
        out = self.out.cpu().numpy()
        for i, (m, n, k) in enumerate(self.sizes):
            pm, cn = (max(m, 1) + 3) // 4 * 4, (max(n, 1) + 3) // 4 * 4
            D = out[self.off[i]: self.off[i + 1]].reshape(pm // 4, cn, 4).transpose(0, 2, 1).reshape(pm, cn)
            ref = self.A[:m, :k] @ self.B[:n, :k].T
            assert np.linalg.norm(D[:m, :n] - ref) <= 1e-13 * max(np.linalg.norm(ref), 1e-300), (i, self.sizes[i])
            assert (D[m:] == 7).all() and (D[:, n:] == 7).all(), (i, self.sizes[i])


BIG = [(385, 321, 0), (400, 390, 1), (383, 384, 15), (384, 257, 16), (449, 330, 17), (390, 449, 49), (450, 450, 100)]


@pytest.mark.parametrize("variant,batch", [(-1, 1500), (-1, 700), (4, 1500), (5, 300)])
def test_lists(bf, variant, batch):
    rng = np.random.default_rng(batch)
    sizes = [tuple(int(v) for v in rng.integers(0, 21, 3)) for _ in range(batch)]
    # the ends of the batch and of the groups of 128 and 32, two in a row, the rest anywhere
    at = [0, 127, 128, 129, batch - 1, 31, int(rng.integers(130, batch - 1))]
    for i, s in zip(at, BIG):
        sizes[i] = s
    for i in rng.integers(200, batch - 1, 40):
        sizes[i] = tuple(int(v) for v in rng.integers(60, 200, 3))
    U = Uneven(bf, sizes, batch)
    U.run(variant)
    U.check()


def test_one_large_instance(bf):
    """One large instance among many small ones takes about as long as by itself."""
    import torch

    def time(sizes):
        U, ts = Uneven(bf, sizes, 1), []
        for _ in range(7):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            U.run()
            e[1].record()
            torch.cuda.synchronize()
            ts.append(e[0].elapsed_time(e[1]))
        return sorted(ts)[3]

    big, small = (1000, 1000, 1000), (8, 8, 8)
    alone = time([big] * 2) / 2
    assert time([small] * 300 + [big] + [small] * 299) < 4 * alone


@pytest.mark.parametrize("m,n,k,batch", [(129, 129, 20, 40), (200, 200, 65, 40), (320, 320, 70, 3), (257, 257, 16, 60),
                                         (300, 129, 33, 40), (129, 64, 70, 100), (70, 65, 5, 200), (160, 33, 80, 2)])
def test_syrk_tiles(bf, m, n, k, batch):
    rng = np.random.default_rng(m + n)
    A, S = rng.uniform(-1, 1, (batch, m, k)), rng.uniform(-1, 1, (batch, m, n))
    a, c = bf.DMatBatch(m, k, batch).pack_all(A), bf.DMatBatch(m, n, batch).pack_all(S)
    d = bf.DMatBatch(m, n, batch).pack_all(np.full((batch, m, n), 7.0))
    ref = 1.5 * A @ A[:, :n].transpose(0, 2, 1) - 0.5 * S
    f = bf.lib.blasfeo_dsyrk_ln_mn_batch
    assert f(batch, m, n, k, 1.5, a.ref, 0, 0, a.ref, 0, 0, -0.5, c.ref, 0, 0, d.ref, 0, 0, None) == 0
    D = d.unpack_all()
    assert relfro(np.tril(D), np.tril(ref)) <= 1e-13
    assert (np.triu(D, 1) == np.triu(np.full((m, n), 7.0), 1)).all()
