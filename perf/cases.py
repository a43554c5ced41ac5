"""The work that programs have this library do, as cases that can be timed and
whose results can be compared: single drop-in calls, the fused small-matrix
kernels, uniform batches, uneven batches and the factor+solve drivers, in FP64
and FP32.

listed() names the standing cases, draw() gives more of the same ranges,
prepare() makes the inputs and buffers of one, run() is one pass through the
public entry points, work() what a pass cannot do without, exact() the results
in 64 bits from plain torch.
"""
import ctypes as C
import math

import numpy as np
import torch

import blasfeo_b200 as bf
from blasfeo_b200.api import DMat, DMatBatch, DMatBatchIL, SMatBatch
from blasfeo_b200.workloads import DESC_DTYPE, SpdBatch

F64, F32 = torch.float64, torch.float32


def listed():
    return [
        # One step of an embedded solver that calls the routines one by one:
        # dgemm_nt, dpotrf_l and dtrsm_rltn on 64 x 64, asynchronous on a stream.
        {"name": "single_64", "kind": "single", "n": 64},
        # The fused syrk + potrf + trsm + gemm chain of 16 x 16 blocks,
        # interleaved slab.
        {"name": "chain_il", "kind": "chain_il", "batch": 20000, "k": 32},
        # Linear MPC: backward Riccati factorization, interleaved slab.
        {"name": "riccati_il", "kind": "riccati_il", "batch": 4096, "N": 30, "nx": 12, "nu": 4},
        # The whole LQ problem on the back-to-back slab: factorization, solve
        # with linear terms, feedback gains.
        {"name": "lq_solve", "kind": "lq", "batch": 4096, "N": 30, "nx": 12, "nu": 4},
        # Uniform batches of one routine.
        {"name": "gemm_128", "kind": "gemm", "batch": 2000, "m": 128, "n": 128, "k": 128, "beta": 0.0},
        {"name": "potrf_64", "kind": "potrf", "batch": 8000, "n": 64},
        # Uneven batches (sizes log-uniform up to nmax), as a mixed stream of
        # small problems launches them.
        {"name": "gemm_uneven", "kind": "vgemm", "batch": 2048, "nmax": 384, "shapes": 1},
        {"name": "lu_uneven", "kind": "vgetrf", "batch": 1024, "nmax": 384, "shapes": 2},
        {"name": "qr_uneven", "kind": "vgeqrf", "batch": 1024, "nmax": 192, "shapes": 3},
        # Uneven SPD systems A x = b, n ~ U{4..nmax}, condition number up to
        # 10^logcond: plain FP64, and FP32 factor with FP64 refinement.
        {"name": "spd_plain", "kind": "posv", "mixed": False, "num": 5000, "nmax": 256, "logcond": 6, "sizes": 4},
        {"name": "spd_mixed", "kind": "posv", "mixed": True, "num": 20000, "nmax": 256, "logcond": 5, "sizes": 5},
        # Single precision: one condensing stage, L = chol(C + A A^T), X = R L^-T.
        {"name": "s_stage_50", "kind": "sstage", "batch": 6000, "n": 50, "k": 37, "m": 60},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["single", "chain_il", "riccati_il", "lq", "gemm", "potrf", "vgemm", "vgetrf", "vgeqrf", "posv",
                       "posv", "sstage"])
    if kind == "single":
        return {"kind": kind, "n": _log_int(rng, 5, 160)}
    if kind == "chain_il":
        return {"kind": kind, "batch": _log_int(rng, 1000, 40000), "k": rng.randint(4, 64)}
    if kind in ("riccati_il", "lq"):
        nu = rng.randint(1, 4)
        return {"kind": kind, "batch": _log_int(rng, 100, 4096), "N": rng.randint(5, 40), "nx": rng.randint(3, 16 - nu),
                "nu": nu}
    if kind == "gemm":
        m, n, k = (_log_int(rng, 8, 256) for _ in range(3))
        return {"kind": kind, "batch": max(64, min(40000, int(1e9 / (m * n * k)))), "m": m, "n": n, "k": k,
                "beta": rng.choice([0.0, 1.0])}
    if kind == "potrf":
        n = _log_int(rng, 8, 300)
        return {"kind": kind, "batch": max(100, min(40000, int(rng.uniform(0.2, 1.0) * 1.5e9 / n ** 2.5))), "n": n}
    if kind in ("vgemm", "vgetrf", "vgeqrf"):
        cap = 192 if kind == "vgeqrf" else 384
        return {"kind": kind, "batch": _log_int(rng, 256, 1024), "nmax": rng.randint(24, cap),
                "shapes": rng.randrange(1 << 20)}
    if kind == "posv":
        mixed = rng.random() < 0.5
        return {"kind": kind, "mixed": mixed, "num": _log_int(rng, 300, 5000), "nmax": rng.randint(40, 256),
                "logcond": rng.randint(2, 5 if mixed else 6), "sizes": rng.randrange(1 << 20)}
    n = _log_int(rng, 8, 128)
    return {"kind": kind, "batch": max(100, min(20000, int(2e8 / n ** 2.5))), "n": n, "k": rng.randint(4, 2 * n),
            "m": rng.randint(4, 2 * n)}


# ---- sizes of the uneven cases (from the case alone) ----

GROUPS = 64  # different shapes in an uneven launch


def _shapes(case):
    """Uneven launch: [(m, n, k), instances] per group, and the order of the
    instances in the descriptor array."""
    rng = np.random.default_rng(case["shapes"])
    nmax = case["nmax"]

    def size():
        return int(min(nmax, math.exp(rng.uniform(math.log(4), math.log(nmax + 1)))))

    count = [len(x) for x in np.array_split(np.arange(case["batch"]), GROUPS)]
    out = []
    for c in count:
        if case["kind"] == "vgemm":
            out.append(((size(), size(), size()), c))
        elif case["kind"] == "vgeqrf":
            n = size()
            out.append(((2 * n, n, n), c))
        else:
            n = size()
            out.append(((n, n, n), c))
    return out, rng.permutation(case["batch"])


def _spd_sizes(case):
    return np.random.default_rng(case["sizes"]).integers(4, case["nmax"] + 1, size=case["num"]).astype(np.int32)


# ---- panel-major layout (panel size 4) ----

def _up(x, a):
    return (x + a - 1) // a * a


def _panels(X):
    """(B, m, n) -> (B, pm/4, 4, cn): row panel, row in the panel, column; zero padded."""
    B, m, n = X.shape
    P = torch.zeros((B, _up(m, 4), _up(n, 4)), dtype=X.dtype, device=X.device)
    P[:, :m, :n] = X
    return P.view(B, _up(m, 4) // 4, 4, _up(n, 4))


def _flat(X, diag=None):
    """(B, m, n) -> (B, stride): the storage of each instance, dA after pA."""
    B, m, n = X.shape
    pa = _panels(X).permute(0, 1, 3, 2).reshape(B, -1)
    out = torch.zeros((B, _stride(m, n)), dtype=X.dtype, device=X.device)
    out[:, : pa.shape[1]] = pa
    if diag is not None:
        out[:, pa.shape[1]: pa.shape[1] + diag.shape[1]] = diag
    return out


def _stride(m, n):
    """Elements of one FP64 instance."""
    return _up((_up(m, 4) * _up(n, 4) + _up(min(m, n), 16)) * 8, 64) // 8


def _view(M, dtype):
    """A uniform batch's matrices, (batch, pm/4, 4, cn), and their dA, (batch, min(m, n)): views of its storage."""
    st, pm, cn = M.s.stride, M.s.pm, M.s.cn
    t = M.buf[: M.batch * st * dtype.itemsize].view(dtype)
    return (t.as_strided((M.batch, pm // 4, 4, cn), (st, 4 * cn, 1, 4)),
            t.as_strided((M.batch, min(M.m, M.n)), (st, 1), t.storage_offset() + pm * cn))


def _put(M, X):
    _view(M, X.dtype)[0].copy_(_panels(X))
    return M


def _view_il(M):
    """An interleaved slab's matrices, (groups, 16, pm/4, 4, cn), and their dA, (groups, 16, min(m, n))."""
    gs, pm, cn, G = M.s.gstride, M.s.pm, M.s.cn, _up(M.batch, 16) // 16
    t = M.buf[: G * gs * 8].view(F64)
    return (t.as_strided((G, 16, pm // 4, 4, cn), (gs, 1, 64 * cn, 16, 64)),
            t.as_strided((G, 16, min(M.m, M.n)), (gs, 1, 16), t.storage_offset() + 16 * pm * cn))


def _groups(X):
    """(B, ...) -> (groups, 16, ...), zero padded."""
    G = _up(X.shape[0], 16) // 16
    out = torch.zeros((G * 16,) + X.shape[1:], dtype=X.dtype, device=X.device)
    out[: X.shape[0]] = X
    return out.view((G, 16) + X.shape[1:])


def _put_il(M, X):
    _view_il(M)[0].copy_(_groups(_panels(X)))
    return M


def _ptr(t):
    return C.c_void_p(t.data_ptr())


# ---- inputs (from the seed alone) ----

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.randn(shape, generator=g, dtype=F64, device="cuda")


def _uniform(g, *shape):
    return torch.rand(shape, generator=g, dtype=F64, device="cuda") * 2 - 1


def _spd(g, B, n):
    G = _randn(g, B, n, n)
    return G @ G.mT / n + torch.eye(n, dtype=F64, device="cuda")


def _spd_cond(g, B, n, logcond):
    """A = Q diag(lambda) Q^T, log10(lambda) ~ U[0, logcond], Q a product of three random reflections."""
    A = torch.diag_embed(10.0 ** (torch.rand((B, n), generator=g, dtype=F64, device="cuda") * logcond))
    for _ in range(3):
        v = _randn(g, B, n, 1)
        v /= v.norm(dim=1, keepdim=True)
        A = A - 2 * v @ (v.mT @ A)
        A = A - 2 * (A @ v) @ v.mT
    return 0.5 * (A + A.mT)


def _stable(g, case):
    """Random stable dynamics and stage costs of LQ problems: BAbt (batch, N, nu+nx, nx), RSQ (batch, N+1, nu+nx,
    nu+nx) with Q_N in the top-left block of the last."""
    b, N, nx, nu = case["batch"], case["N"], case["nx"], case["nu"]
    M = nu + nx
    BA = torch.empty((b, N, M, nx), dtype=F64, device="cuda")
    BA[:, :, :nu] = 0.5 * _randn(g, b, N, nu, nx)
    BA[:, :, nu:] = 0.9 * torch.eye(nx, dtype=F64, device="cuda") + 0.3 / math.sqrt(nx) * _randn(g, b, N, nx, nx)
    R = _randn(g, b, N + 1, M, M)
    RSQ = 0.1 * (R @ R.mT) + torch.eye(M, dtype=F64, device="cuda")
    RSQ[:, N, nx:, :] = 0
    RSQ[:, N, :, nx:] = 0
    return BA, RSQ


def _pad16(X):
    """(..., M, n) -> (..., 16, n)"""
    out = torch.zeros(X.shape[:-2] + (16, X.shape[-1]), dtype=X.dtype, device=X.device)
    out[..., : X.shape[-2], :] = X
    return out


def _pad16x16(X):
    return _pad16(_pad16(X).mT).mT


def _inputs(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind == "single":
        n = case["n"]
        return _uniform(g, 1, n, n), _uniform(g, 1, n, n), _spd(g, 1, n), _randn(g, 1, n, n)
    if kind == "chain_il":
        b, k = case["batch"], case["k"]
        return _randn(g, b, 16, k), _randn(g, b, 16, 16), _randn(g, b, 16, 16), _randn(g, b, 16, 16)
    if kind in ("riccati_il", "lq"):
        b, N, nx, nu = case["batch"], case["N"], case["nx"], case["nu"]
        BA, RSQ = _stable(g, case)
        if kind == "riccati_il":
            return BA, RSQ
        rq = _randn(g, b, N + 1, nu + nx)
        rq[:, N, nx:] = 0
        return BA, RSQ, rq, _randn(g, b, N, nx)
    if kind == "gemm":
        b, m, n, k = case["batch"], case["m"], case["n"], case["k"]
        return _uniform(g, b, m, k), _uniform(g, b, n, k), _uniform(g, b, m, n)
    if kind == "potrf":
        return (_spd(g, case["batch"], case["n"]),)
    if kind == "vgemm":
        return [(_uniform(g, c, m, k), _uniform(g, c, n, k)) for (m, n, k), c in _shapes(case)[0]]
    if kind in ("vgetrf", "vgeqrf"):
        return [_uniform(g, c, m, n) for (m, n, _), c in _shapes(case)[0]]
    if kind == "posv":
        ns, mats = _spd_sizes(case), {}
        for n in np.unique(ns):
            idx = np.nonzero(ns == n)[0]
            mats[int(n)] = (idx, _spd_cond(g, len(idx), int(n), case["logcond"]))
        rng = np.random.default_rng(seed)
        return ns, mats, [rng.standard_normal(int(n)) for n in ns]
    b, n, k, m = case["batch"], case["n"], case["k"], case["m"]
    return (_randn(g, b, n, k) / math.sqrt(k)).to(F32), _spd(g, b, n).to(F32), _randn(g, b, m, n).to(F32)


# ---- one uneven batch in device memory ----

class _Slab:
    """The instances of all groups one after the other; desc: device array of descriptors in the launch's order."""

    def __init__(self, dims, order, mats=None):
        strides = [_stride(m, n) for (m, n), c in dims]
        self.start = np.concatenate([[0], np.cumsum([s * c for s, (_, c) in zip(strides, dims)])])
        self.buf = torch.zeros(int(self.start[-1]) + 8, dtype=F64, device="cuda")
        d = np.zeros(len(order), dtype=DESC_DTYPE)
        at = 0
        for gi, ((m, n), c) in enumerate(dims):
            if mats is not None:
                self.buf[int(self.start[gi]): int(self.start[gi + 1])].view(c, -1).copy_(_flat(mats[gi]))
            e = d[at: at + c]
            e["mem"] = self.buf.data_ptr() + 8 * (int(self.start[gi]) + strides[gi] * np.arange(c))
            e["pA"] = e["mem"]
            e["dA"] = e["mem"] + 8 * _up(m, 4) * _up(n, 4)
            e["m"], e["n"], e["pm"], e["cn"], e["memsize"] = m, n, _up(m, 4), _up(n, 4), 8 * strides[gi]
            at += c
        self.desc = torch.from_numpy(d[order].view(np.uint8).copy()).cuda()


def prepare(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    s = {"case": case}
    if kind == "single":
        n = case["n"]
        bf.set_stream(torch.cuda.current_stream())
        bf.set_sync(False)  # the calls of a step follow each other on the stream
        for name, X in zip("ABSR", x):
            s[name] = DMat(n, n)
            s[name].buf[: 8 * _up(n, 4) ** 2].view(F64).copy_(_panels(X).permute(0, 1, 3, 2).reshape(-1))
        for name in "CDLX":
            s[name] = DMat(n, n)
        pa = lambda M: M.buf[: 8 * _up(n, 4) ** 2].view(F64).view(_up(n, 4) // 4, _up(n, 4), 4)  # noqa: E731
        da = s["L"].buf[8 * _up(n, 4) ** 2:].view(F64)[:n]
        s["out"] = {"D": pa(s["D"]), "L": pa(s["L"]), "dL": da, "X": pa(s["X"])}
    elif kind == "chain_il":
        b, k = case["batch"], case["k"]
        for name, X in zip("ARCG", x):
            s[name] = _put_il(DMatBatchIL(16, X.shape[2], b), X)
        for name in "LXD":
            s[name] = DMatBatchIL(16, 16, b)
        s["info"] = torch.zeros(b, dtype=torch.int32, device="cuda")
        L, dL = _view_il(s["L"])
        s["out"] = {"L": L, "dL": dL, "X": _view_il(s["X"])[0], "D": _view_il(s["D"])[0], "info": s["info"]}
    elif kind == "riccati_il":
        b, N, nx = case["batch"], case["N"], case["nx"]
        bs = _up(b, 16)
        BA, RSQ = _pad16(x[0]), _pad16x16(x[1])
        stage = lambda X: _groups(X).reshape((bs,) + X.shape[1:]).transpose(0, 1).reshape((-1,) + X.shape[2:])  # noqa: E731
        s["BA"] = _put_il(DMatBatchIL(16, nx, N * bs), stage(BA))
        s["RSQ"] = _put_il(DMatBatchIL(16, 16, (N + 1) * bs), stage(RSQ))
        s["L"] = DMatBatchIL(16, 16, (N + 1) * bs)
        s["info"] = torch.zeros(b, dtype=torch.int32, device="cuda")
        L, dL = _view_il(s["L"])
        s["out"] = {"L": L, "dL": dL, "info": s["info"]}
    elif kind == "lq":
        b, N, nx, nu = case["batch"], case["N"], case["nx"], case["nu"]
        s["BA"] = _put(DMatBatch(16, nx, b * N), _pad16(x[0]).reshape(b * N, 16, nx))
        s["RSQ"] = _put(DMatBatch(16, 16, b * (N + 1)), _pad16x16(x[1]).reshape(b * (N + 1), 16, 16))
        s["L"], s["K"] = DMatBatch(16, 16, b * (N + 1)), DMatBatch(nu, nx, b * N)
        s["rq"], s["b"] = x[2].contiguous(), x[3].contiguous()
        s["ux"], s["pi"] = torch.zeros_like(s["rq"]), torch.zeros_like(s["b"])
        s["info"] = torch.zeros(b, dtype=torch.int32, device="cuda")
        L, dL = _view(s["L"], F64)
        s["out"] = {"L": L, "dL": dL, "ux": s["ux"], "pi": s["pi"], "K": _view(s["K"], F64)[0], "info": s["info"]}
    elif kind == "gemm":
        b, m, n, k = case["batch"], case["m"], case["n"], case["k"]
        s["A"], s["B"] = _put(DMatBatch(m, k, b), x[0]), _put(DMatBatch(n, k, b), x[1])
        s["C"], s["D"] = _put(DMatBatch(m, n, b), x[2]), DMatBatch(m, n, b)
        s["out"] = {"D": _view(s["D"], F64)[0]}
    elif kind == "potrf":
        b, n = case["batch"], case["n"]
        s["C"], s["L"] = _put(DMatBatch(n, n, b), x[0]), DMatBatch(n, n, b)
        s["info"] = torch.zeros(b, dtype=torch.int32, device="cuda")
        L, dL = _view(s["L"], F64)
        s["out"] = {"L": L, "dL": dL, "info": s["info"]}
    elif kind in ("vgemm", "vgetrf", "vgeqrf"):
        groups, order = _shapes(case)
        sizes = np.repeat(np.array([g[0] for g in groups], dtype=np.int32), [g[1] for g in groups], axis=0)[order]
        s["m"], s["n"], s["k"] = (torch.from_numpy(sizes[:, i].copy()).cuda() for i in range(3))
        s["max"] = [int(v) for v in sizes.max(axis=0)]
        mn, mk, nk = ([((g[0][i], g[0][j]), g[1]) for g in groups] for i, j in ((0, 1), (0, 2), (1, 2)))
        s["D"] = _Slab(mn, order)
        if kind == "vgemm":
            s["A"], s["B"] = _Slab(mk, order, [p[0] for p in x]), _Slab(nk, order, [p[1] for p in x])
            s["out"] = {"D": s["D"].buf}
        else:
            s["A"] = _Slab(mn, order, x)
            s["out"] = {"D": s["D"].buf}
            if kind == "vgetrf":
                s["piv"] = torch.zeros((case["batch"], s["max"][1]), dtype=torch.int32, device="cuda")
                s["info"] = torch.zeros(case["batch"], dtype=torch.int32, device="cuda")
                s["out"].update(piv=s["piv"], info=s["info"])
    elif kind == "posv":
        s["W"] = SpdBatch(*x)
        s["info"] = torch.zeros(case["num"], dtype=torch.int32, device="cuda")
        s["out"] = {"x": s["W"].x, "info": s["info"]}
    else:
        b, n, k, m = case["batch"], case["n"], case["k"], case["m"]
        s["A"], s["C"], s["R"] = (_put(SMatBatch(X.shape[1], X.shape[2], b), X) for X in x)
        s["L"], s["X"] = SMatBatch(n, n, b), SMatBatch(m, n, b)
        s["info"] = torch.zeros(b, dtype=torch.int32, device="cuda")
        L, dL = _view(s["L"], F32)
        s["out"] = {"L": L, "dL": dL, "X": _view(s["X"], F32)[0], "info": s["info"]}
    return s


def run(s):
    case, lib = s["case"], bf.lib
    kind = case["kind"]
    if kind == "single":
        n = case["n"]
        bf.blasfeo_dgemm_nt(n, n, n, 1.0, s["A"], 0, 0, s["B"], 0, 0, 0.0, s["C"], 0, 0, s["D"], 0, 0)
        bf.blasfeo_dpotrf_l(n, s["S"], 0, 0, s["L"], 0, 0)
        bf.blasfeo_dtrsm_rltn(n, n, 1.0, s["L"], 0, 0, s["R"], 0, 0, s["X"], 0, 0)
        return s["out"]
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    if kind == "chain_il":
        bf.check(lib.blasfeo_dsyrk_dpotrf_dtrsm_dgemm_batch_il(
            case["batch"], 16, case["k"], 16.0, s["A"].ref, s["R"].ref, s["C"].ref, s["G"].ref, s["L"].ref, s["X"].ref,
            s["D"].ref, _ptr(s["info"]), stream))
    elif kind == "riccati_il":
        bf.check(lib.blasfeo_dric_trf_batch_il(case["batch"], case["N"], case["nx"], case["nu"], s["BA"].ref,
                                               s["RSQ"].ref, s["L"].ref, _ptr(s["info"]), stream))
    elif kind == "lq":
        dims = case["batch"], case["N"], case["nx"], case["nu"]
        M, nx = case["nu"] + case["nx"], case["nx"]
        bf.check(lib.blasfeo_dric_trf_batch(*dims, s["BA"].ref, s["RSQ"].ref, s["L"].ref, _ptr(s["info"]), stream))
        bf.check(lib.blasfeo_dric_trs_batch(*dims, s["BA"].ref, s["L"].ref, _ptr(s["b"]), nx, _ptr(s["rq"]), M,
                                            _ptr(s["ux"]), M, _ptr(s["pi"]), nx, stream))
        bf.check(lib.blasfeo_dric_gains_batch(*dims, s["L"].ref, s["K"].ref, stream))
    elif kind == "gemm":
        bf.check(lib.blasfeo_dgemm_nt_batch(case["batch"], case["m"], case["n"], case["k"], 1.0, s["A"].ref, 0, 0,
                                            s["B"].ref, 0, 0, case["beta"], s["C"].ref, 0, 0, s["D"].ref, 0, 0, stream))
    elif kind == "potrf":
        bf.check(lib.blasfeo_dpotrf_l_batch(case["batch"], case["n"], s["C"].ref, 0, 0, s["L"].ref, 0, 0,
                                            _ptr(s["info"]), stream))
    elif kind == "vgemm":
        bf.check(lib.blasfeo_dgemm_nt_vbatch(case["batch"], _ptr(s["m"]), _ptr(s["n"]), _ptr(s["k"]), *s["max"], 1.0,
                                             _ptr(s["A"].desc), _ptr(s["B"].desc), 0.0, _ptr(s["D"].desc),
                                             _ptr(s["D"].desc), stream))
    elif kind == "vgetrf":
        bf.check(lib.blasfeo_dgetrf_rp_vbatch(case["batch"], _ptr(s["m"]), _ptr(s["n"]), s["max"][0], s["max"][1],
                                              _ptr(s["A"].desc), _ptr(s["D"].desc), _ptr(s["piv"]), s["max"][1],
                                              _ptr(s["info"]), stream))
    elif kind == "vgeqrf":
        bf.check(lib.blasfeo_dgeqrf_vbatch(case["batch"], _ptr(s["m"]), _ptr(s["n"]), s["max"][0], s["max"][1],
                                           _ptr(s["A"].desc), _ptr(s["D"].desc), stream))
    elif kind == "posv":
        W = s["W"]
        if case["mixed"]:
            # refined to where the residual's own FP64 rounding begins: as good an answer as the plain solver's
            bf.check(lib.blasfeo_dsposv_l_vbatch(case["num"], _ptr(W.nvec), W.max_n, _ptr(W.desc), _ptr(W.bdesc),
                                                 _ptr(W.xdesc), 30, 1e-14, None, None, _ptr(s["info"]), None, 0, stream))
        else:
            bf.check(lib.blasfeo_dposv_l_vbatch(case["num"], _ptr(W.nvec), W.max_n, _ptr(W.desc), _ptr(W.bdesc),
                                                _ptr(W.xdesc), _ptr(s["info"]), None, 0, stream))
    else:
        b, n = case["batch"], case["n"]
        bf.check(lib.blasfeo_ssyrk_spotrf_ln_batch(b, n, case["k"], s["A"].ref, 0, 0, s["A"].ref, 0, 0, s["C"].ref, 0, 0,
                                                   s["L"].ref, 0, 0, _ptr(s["info"]), stream))
        bf.check(lib.blasfeo_strsm_rltn_batch(b, case["m"], n, 1.0, s["L"].ref, 0, 0, s["R"].ref, 0, 0, s["X"].ref, 0, 0,
                                              stream))
    return s["out"]


def work(case):
    """Each operand read once and each result written once (lower triangles where only they count); standard flop
    counts."""
    kind = case["kind"]
    chol = lambda n: n ** 3 / 3 + n ** 2 / 2 + n / 6  # noqa: E731
    low = lambda n: n * (n + 1) / 2  # noqa: E731
    if kind == "single":
        n = case["n"]
        return {"bytes": 8 * (3 * n * n + 2 * low(n) + n + low(n) + 2 * n * n), "flops": 2 * n ** 3 + chol(n) + n ** 3}
    if kind == "chain_il":
        b, k = case["batch"], case["k"]
        return {"bytes": b * 8 * (16 * k + 5 * 256 + low(16) + 16),
                "flops": b * (k * 16 * 17 + chol(16) + 16 ** 3 + 2 * 16 ** 3)}
    if kind in ("riccati_il", "lq"):
        b, N, nx, M = case["batch"], case["N"], case["nx"], case["nu"] + case["nx"]
        nu = case["nu"]
        by = b * 8 * (N * (M * nx + 2 * low(M) + M) + 2 * low(nx) + nx)
        fl = b * (N * (M * nx * (nx + 1) + nx * M * (M + 1) + chol(M)) + chol(nx))
        if kind == "lq":
            by += b * 8 * (2 * ((N + 1) * M + N * nx) + N * nu * nx)
            fl += b * N * (8 * nx * nx + 4 * M * nx + 2 * (nu * nu + 2 * nu * nx) + nu * nu * nx)
        return {"bytes": by, "flops": fl}
    if kind == "gemm":
        b, m, n, k = case["batch"], case["m"], case["n"], case["k"]
        return {"bytes": b * 8 * (m * k + n * k + m * n * (2 if case["beta"] else 1)), "flops": b * 2 * m * n * k}
    if kind == "potrf":
        b, n = case["batch"], case["n"]
        return {"bytes": b * 8 * (2 * low(n) + n), "flops": b * chol(n)}
    if kind == "vgemm":
        g = _shapes(case)[0]
        return {"bytes": sum(8 * c * (m * k + n * k + m * n) for (m, n, k), c in g),
                "flops": sum(2 * c * m * n * k for (m, n, k), c in g)}
    if kind == "vgetrf":
        g = _shapes(case)[0]
        return {"bytes": sum(c * (16 * n * n + 12 * n) for (_, n, _), c in g),
                "flops": sum(c * (2 * n ** 3 / 3 - n ** 2 / 2 + 5 * n / 6) for (_, n, _), c in g)}
    if kind == "vgeqrf":
        g = _shapes(case)[0]
        return {"bytes": sum(c * (16 * m * n + 8 * n) for (m, n, _), c in g),
                "flops": sum(c * (2 * m * n * n - 2 * n ** 3 / 3 + m * n + n * n + 14 * n / 3) for (m, n, _), c in g)}
    if kind == "posv":
        n = _spd_sizes(case).astype(np.float64)
        return {"bytes": float((8 * low(n) + 16 * n).sum()), "flops": float((chol(n) + 4 * n * n).sum())}
    b, n, k, m = case["batch"], case["n"], case["k"], case["m"]
    return {"bytes": b * 4 * (n * k + 2 * low(n) + n + 2 * m * n), "flops": b * (k * n * (n + 1) + chol(n) + m * n * n)}


# ---- results in 64 bits ----

def _exact_riccati(BA, RSQ, case):
    """L_k (batch, N+1, 16, 16) and the inverse diagonals."""
    b, N, nx, nu = case["batch"], case["N"], case["nx"], case["nu"]
    M = nu + nx
    L = torch.zeros((b, N + 1, 16, 16), dtype=F64, device="cuda")
    d = torch.zeros((b, N + 1, 16), dtype=F64, device="cuda")
    for k in range(N, -1, -1):
        if k == N:
            m, S = nx, RSQ[:, N, :nx, :nx]
        else:
            o = 0 if k + 1 == N else nu
            W = BA[:, k] @ L[:, k + 1, o: o + nx, o: o + nx]
            m, S = M, RSQ[:, k] + W @ W.mT
        F = torch.linalg.cholesky(S)
        L[:, k, :m, :m] = F
        d[:, k, :m] = 1 / torch.diagonal(F, dim1=1, dim2=2)
    return L, d


def _exact_lq(x, case):
    BA, RSQ, rq, bb = x
    b, N, nx, nu = case["batch"], case["N"], case["nx"], case["nu"]
    M = nu + nx
    L, d = _exact_riccati(BA, RSQ, case)
    xx = lambda k: L[:, k, :nx, :nx] if k == N else L[:, k, nu:M, nu:M]  # noqa: E731
    P = [xx(k) @ xx(k).mT for k in range(N + 1)]
    p = [None] * N + [rq[:, N, :nx, None]]
    K, kff = [None] * N, [None] * N
    for k in range(N - 1, -1, -1):
        v = P[k + 1] @ bb[:, k, :, None] + p[k + 1]
        h = rq[:, k, :, None] + BA[:, k] @ v
        Luu, Lxu = L[:, k, :nu, :nu], L[:, k, nu:M, :nu]
        K[k] = -torch.linalg.solve_triangular(Luu.mT, Lxu.mT, upper=True)
        kff[k] = -torch.cholesky_solve(h[:, :nu], Luu)
        p[k] = h[:, nu:] + K[k].mT @ h[:, :nu]
    ux, pi = torch.zeros_like(rq), torch.zeros_like(bb)
    x0 = -torch.cholesky_solve(p[0], xx(0))
    for k in range(N):
        u = K[k] @ x0 + kff[k]
        ux[:, k] = torch.cat([u, x0], 1)[..., 0]
        x0 = BA[:, k].mT @ ux[:, k, :, None] + bb[:, k, :, None]
        pi[:, k] = (P[k + 1] @ x0 + p[k + 1])[..., 0]
    ux[:, N, :nx] = x0[..., 0]
    return {"L": _panels(L.view(-1, 16, 16)), "dL": d.view(-1, 16), "ux": ux, "pi": pi,
            "K": _panels(torch.stack(K, 1).reshape(b * N, nu, nx)), "info": None}


def exact(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    rsolve = lambda L, R: torch.linalg.solve_triangular(L, R.mT, upper=False).mT  # noqa: E731
    inv_diag = lambda L: 1 / torch.diagonal(L, dim1=1, dim2=2)  # noqa: E731
    if kind == "single":
        A, B, S, R = x
        L = torch.linalg.cholesky(S)
        pa = lambda X: _panels(X)[0].permute(0, 2, 1)  # noqa: E731
        return {"D": pa(A @ B.mT), "L": pa(L), "dL": inv_diag(L)[0], "X": pa(rsolve(L, R))}
    if kind == "chain_il":
        A, R, Cm, G = x
        L = torch.linalg.cholesky(A @ A.mT + 16.0 * torch.eye(16, dtype=F64, device="cuda"))
        X = rsolve(L, R)
        il = lambda Y: _groups(_panels(Y))  # noqa: E731
        return {"L": il(L), "dL": _groups(inv_diag(L)), "X": il(X), "D": il(Cm - X @ G.mT), "info": None}
    if kind == "riccati_il":
        L, d = _exact_riccati(x[0], x[1], case)
        bs, N = _up(case["batch"], 16), case["N"]
        L = _groups(L).reshape(bs, N + 1, 16, 16).transpose(0, 1).reshape(-1, 16, 16)
        d = _groups(d).reshape(bs, N + 1, 16).transpose(0, 1).reshape(-1, 16)
        return {"L": _groups(_panels(L)), "dL": _groups(d), "info": None}
    if kind == "lq":
        return _exact_lq(x, case)
    if kind == "gemm":
        return {"D": _panels(x[0] @ x[1].mT + case["beta"] * x[2])}
    if kind == "potrf":
        L = torch.linalg.cholesky(x[0])
        return {"L": _panels(L), "dL": inv_diag(L), "info": None}
    if kind in ("vgemm", "vgetrf", "vgeqrf"):
        parts = []
        for X in x:
            if kind == "vgemm":
                parts.append(_flat(X[0] @ X[1].mT))
            elif kind == "vgetrf":
                LU = torch.linalg.lu_factor(X).LU
                parts.append(_flat(LU, inv_diag(LU)))
            else:
                QR, tau = torch.geqrf(X.cpu())
                parts.append(_flat(QR.cuda(), tau.cuda()))
        D = torch.cat([p.reshape(-1) for p in parts] + [torch.zeros(8, dtype=F64, device="cuda")])
        return {"D": D} if kind != "vgetrf" else {"D": D, "piv": None, "info": None}
    if kind == "posv":
        ns, mats, rhs = x
        at = np.concatenate([[0], np.cumsum(_up(ns, 4))]).astype(np.int64)
        out = torch.zeros(int(at[-1]) + 4, dtype=F64, device="cuda")
        for n, (idx, A) in mats.items():
            b = torch.from_numpy(np.stack([rhs[i] for i in idx])).cuda()
            sol = torch.cholesky_solve(b[:, :, None], torch.linalg.cholesky(A))[..., 0]
            out[torch.from_numpy(at[idx][:, None] + np.arange(n)).cuda()] = sol
        return {"x": out, "info": None}
    A, S, R = (X.double() for X in x)
    L = torch.linalg.cholesky(S + A @ A.mT)
    return {"L": _panels(L), "dL": inv_diag(L), "X": _panels(rsolve(L, R)), "info": None}
