"""Batched Riccati kernels at the edges of their ranges: nu + nx = 16 with
every split of the fragment blocks, nu = 0, batches around the 8 problems of a
CTA and the 2 of a warp, N = 1, padding that holds NaN, slabs off the 16-byte
grid; against the oracle's factorization and solve (1e-13, the FP64 bar of
every routine)."""
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


def problems(rng, nbt, N, nx, nu):
    """(b, N, 16, nx), (b, N+1, 16, 16): what the routines must not read is NaN."""
    m = nx + nu
    BA = np.full((nbt, N, 16, nx), np.nan)
    RSQ = np.full((nbt, N + 1, 16, 16), np.nan)
    BA[:, :, :m] = rng.standard_normal((nbt, N, m, nx)) / np.sqrt(nx)
    G = rng.standard_normal((nbt, N + 1, m, m))
    S = np.tril(G @ G.transpose(0, 1, 3, 2) / m + np.eye(m))
    S[..., np.triu(np.ones((m, m), bool), 1)] = np.nan
    RSQ[:, :, :m, :m] = S
    RSQ[:, N] = np.nan
    RSQ[:, N, :nx, :nx] = S[:, N, :nx, :nx]
    return BA, RSQ


@pytest.mark.parametrize("dims", [(16, 0), (15, 1), (1, 15), (9, 7), (8, 8), (12, 3), (13, 3), (3, 1)])
@pytest.mark.parametrize("nbt,N", [(1, 1), (7, 3), (9, 2), (17, 4)])
def test_factor_solve_gains(bf, dims, nbt, N):
    import torch
    from blasfeo_b200.api import DMatBatchIL
    from tests.ric_oracle import ric_trf, ric_trs
    nx, nu = dims
    m = nx + nu
    rng = np.random.default_rng(1000 * nx + 10 * nbt + N)
    BA, RSQ = problems(rng, nbt, N, nx, nu)
    b, rq = rng.standard_normal((nbt, N, nx)), rng.standard_normal((nbt, N + 1, m))
    slab = lambda X: bf.DMatBatch(X.shape[-2], X.shape[-1], X.shape[0] * X.shape[1]).pack_all(
        X.reshape((-1,) + X.shape[2:]))
    sBA, sRSQ, sL = slab(BA), slab(RSQ), bf.DMatBatch(16, 16, nbt * (N + 1))
    info = torch.full((nbt,), -9, dtype=torch.int32, device="cuda")
    assert bf.lib.blasfeo_dric_trf_batch(nbt, N, nx, nu, sBA.ref, sRSQ.ref, sL.ref, P(info), None) == 0
    # interleaved: stage k of problem p at k * bs + p
    bs = (nbt + 15) // 16 * 16
    stage = lambda X: np.concatenate([np.concatenate([X[:, k], np.zeros((bs - nbt,) + X.shape[2:])])
                                      for k in range(X.shape[1])])
    il = lambda X: DMatBatchIL(X.shape[1], X.shape[2], X.shape[0]).pack_all(X)
    iBA, iRSQ, iL = il(stage(BA)), il(stage(RSQ)), DMatBatchIL(16, 16, (N + 1) * bs)
    iinfo = torch.full((nbt,), -9, dtype=torch.int32, device="cuda")
    assert bf.lib.blasfeo_dric_trf_batch_il(nbt, N, nx, nu, iBA.ref, iRSQ.ref, iL.ref, P(iinfo), None) == 0
    db, drq = torch.from_numpy(b).cuda(), torch.from_numpy(rq).cuda()
    ux, pi = torch.zeros_like(drq), torch.zeros_like(db)
    assert bf.lib.blasfeo_dric_trs_batch(nbt, N, nx, nu, sBA.ref, sL.ref, P(db), nx, P(drq), m, P(ux), m, P(pi), nx,
                                         None) == 0
    # the same solve with both slabs 8 bytes off the 16-byte grid
    off = []
    for s in (sBA, sL):
        buf = torch.zeros(s.buf.numel() + 16, dtype=torch.uint8, device="cuda")
        buf[8: 8 + s.buf.numel()] = s.buf
        d = type(s.s).from_buffer_copy(s.s)
        d.pA = buf.data_ptr() + 8
        off.append((buf, d))
    ux2, pi2 = torch.zeros_like(ux), torch.zeros_like(pi)
    assert bf.lib.blasfeo_dric_trs_batch(nbt, N, nx, nu, C.byref(off[0][1]), C.byref(off[1][1]), P(db), nx, P(drq), m,
                                         P(ux2), m, P(pi2), nx, None) == 0
    K = None
    if nu:
        sK = bf.DMatBatch(nu, nx, nbt * N)
        assert bf.lib.blasfeo_dric_gains_batch(nbt, N, nx, nu, sL.ref, sK.ref, None) == 0
        K = sK.unpack_all().reshape(nbt, N, nu, nx)
    torch.cuda.synchronize()
    assert (info == 0).all() and (iinfo == 0).all()
    assert torch.equal(ux, ux2) and torch.equal(pi, pi2)
    L, dA = sL.unpack_all().reshape(nbt, N + 1, 16, 16), sL.diag_all(16).reshape(nbt, N + 1, 16)
    L_il = iL.unpack_all()
    orc = oracle_api()
    clean = lambda X: np.nan_to_num(X)
    sym = lambda X: np.tril(X) + np.tril(X, -1).swapaxes(-1, -2)
    for p in sorted({0, nbt // 2, nbt - 1}):
        R = sym(clean(RSQ[p]))
        Lr = ric_trf(orc, clean(BA[p]), R, N, nx, nu)
        pad = lambda X: np.concatenate([X, np.zeros((X.shape[0], 16 - X.shape[1]))], 1)
        uxr, pir = ric_trs(orc, Lr, clean(BA[p]), pad(b[p]), pad(rq[p]), N, nx, nu)
        for k in range(N + 1):
            mm = nx if k == N else m
            ref = np.tril(Lr[k].get())[:mm, :mm]
            assert relfro(np.tril(L[p, k, :mm, :mm]), ref) <= 1e-13, (p, k)
            assert relfro(np.tril(L_il[k * bs + p, :mm, :mm]), ref) <= 1e-13, (p, k)
            assert relfro(dA[p, k, :mm], 1.0 / np.diagonal(ref)) <= 1e-13, (p, k)
            assert relfro(ux[p, k, :mm].cpu().numpy(), uxr[k][:mm]) <= 1e-12, (p, k)
            if K is not None and k < N:
                Kr = -np.linalg.solve(ref[:nu, :nu].T, ref[nu:, :nu].T)
                assert relfro(K[p, k], Kr) <= 1e-12, (p, k)
        assert relfro(pi[p].cpu().numpy(), np.stack(pir)[:, :nx]) <= 1e-12, p
