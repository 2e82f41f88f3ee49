"""The solver path's workloads, as a program that uses this framework calls them.

Every case goes through the public entry points (the C ABI behind
``senk_gb300.lib`` and ``senk_gb300.solver``). The matrices are the configurations
the repository solves (``senk_gb300/problems.py``); they and their host setup
(ordering, ILU factors) are made once per process and shared, as a program that
solves many right-hand sides keeps them. Vectors come from the seed.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from senk_gb300 import learned as LN
from senk_gb300 import lib as L
from senk_gb300 import problems as P
from senk_gb300 import setup as S
from senk_gb300.solver import System

BSIZE = 16          # rows per ABMC block, as in every scalar configuration
NODES = 4           # nodes per ABMC block of the block-3x3 system (12 rows)


def listed():
    return [
        # a user's own CG loop on the blas1 and SpMV calls, on the smallest
        # configuration: launches, synchronising dot products, latency
        dict(name="cg8_f64_poisson128", kind="cg", problem="poisson2d", n=128),
        # one SpMV on the headline matrix (FP64), and on the large
        # variable-coefficient one in FP32 (a refinement loop's inner products)
        dict(name="spmv_f64_convdiff128", kind="spmv", problem="convdiff", n=128, dtype="f64"),
        dict(name="spmv_f32_vardiff160", kind="spmv", problem="vardiff", n=160, dtype="f32"),
        # register-blocked SpMV of the block-3x3 system
        dict(name="bcsr3_f64_block48", kind="bcsr", problem="block27", n=48),
        # one ILU(0) application (L then U), the preconditioner of every solve:
        # FP32 on the headline system (refinement's inner solves), FP64 on an odd
        # size with variable coefficients, and the natural order's level sets on
        # the small 2D system
        dict(name="ilu_f32_convdiff128", kind="ilu", problem="convdiff", n=128, dtype="f32", order="abmc"),
        dict(name="ilu_f64_vardiff101", kind="ilu", problem="vardiff", n=101, dtype="f64", order="abmc"),
        dict(name="ilu_f64_natural_poisson128", kind="ilu", problem="poisson2d", n=128, dtype="f64", order="natural"),
        # one ILUB(3x3) application of the block system
        dict(name="ilub3_f64_block48", kind="ilub", problem="block27", n=48),
        # whole calls: the plain FP64 solve of the headline system to 1e-8, and
        # the FP32 inner solve of one refinement step (1e-4, at most two cycles)
        dict(name="gmres_f64_convdiff128", kind="gmres", problem="convdiff", n=128, dtype="f64", eps=1e-8, outer=20),
        dict(name="gmres_f32_convdiff128", kind="gmres", problem="convdiff", n=128, dtype="f32", eps=1e-4, outer=2),
        # the other Krylov methods, some iterations on an odd mid-size system
        dict(name="bicgstab8_f64_convdiff75", kind="bicgstab", problem="convdiff", n=75, its=8),
        # loss and gradient of the learned preconditioner on one system of its
        # family (forward and backward)
        dict(name="learned_grad_64", kind="learned", problem="vardiff", n=64),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cg", "spmv", "spmv", "bcsr", "ilu", "ilu", "natural", "ilub", "gmres", "krylov", "learned"])
    prob3 = rng.choice(["convdiff", "vardiff"])
    dt = rng.choice(["f64", "f32"])
    if kind == "cg":
        return dict(kind="cg", problem="poisson2d", n=_logint(rng, 33, 900))
    if kind == "spmv":
        if rng.random() < 0.3:
            return dict(kind="spmv", problem="poisson2d", n=_logint(rng, 65, 1500), dtype=dt)
        return dict(kind="spmv", problem=prob3, n=_logint(rng, 25, 160 if dt == "f32" else 128), dtype=dt)
    if kind == "bcsr":
        return dict(kind="bcsr", problem="block27", n=_logint(rng, 9, 47))
    if kind == "ilu":
        return dict(kind="ilu", problem=prob3, n=4 * _logint(rng, 6, 31) + rng.choice([0, 0, 1]), dtype=dt, order="abmc")
    if kind == "natural":
        return dict(kind="ilu", problem="poisson2d", n=_logint(rng, 40, 150), dtype=dt, order="natural")
    if kind == "ilub":
        return dict(kind="ilub", problem="block27", n=4 * _logint(rng, 3, 11))
    if kind == "gmres":
        return dict(kind="gmres", problem="convdiff", n=_logint(rng, 24, 112), dtype=dt,
                    eps=1e-8 if dt == "f64" else 1e-4, outer=20 if dt == "f64" else 2)
    if kind == "krylov":
        if rng.random() < 0.5:
            return dict(kind="gcr", problem=prob3, n=_logint(rng, 24, 100), its=20)
        return dict(kind="bicgstab", problem="convdiff", n=_logint(rng, 24, 110), its=8)
    return dict(kind="learned", problem="vardiff", n=4 * _logint(rng, 5, 16))


# ------------------------------------------------------------ host setup

@functools.lru_cache(maxsize=4)
def _matrix(problem, n):
    if problem == "poisson2d":
        return P.poisson2d(n)
    if problem == "convdiff":
        return P.convdiff3d(n, 0.5)
    if problem == "vardiff":
        return P.vardiff3d(n, 1.5, 8.0, 0)
    return P.block27(n, seed=0)


def _pad(A, m):
    """A with unit rows appended up to a multiple of m rows (an ABMC block's size)."""
    k = -A.n % m
    if not k:
        return A
    return P.Csr(np.concatenate([A.val, np.ones(k)]),
                 np.concatenate([A.cind, np.arange(A.n, A.n + k, dtype=np.int32)]),
                 np.concatenate([A.rptr, A.nnz + np.arange(1, k + 1, dtype=np.int32)]).astype(np.int32))


class _Setup:
    """Ordered matrix, its split ILU factors and colour pointers."""


@functools.lru_cache(maxsize=4)
def _setup(problem, n, order):
    A, s = _matrix(problem, n), _Setup()
    if order == "natural":
        s.A, s.cptr, s.cnum = A, None, 0
        s.Lf, s.Uf, _ = S.Split(S.Ilu0(A), "L-DU", True)
    elif problem == "block27":
        G = P.block27_node_graph(n)
        s.cnum, s.cptr, LPn, _ = S.GetABMCPermutation(G.cind, G.rptr, G.n, NODES, False, "connect")
        LP, RP = P.expand_node_permutation(LPn, 3)
        s.A = S.Reordering(A, LP, RP)
        Lf, Uf, _ = S.Split(S.Ilu0(S.AllocBlockZero(s.A, 3, 3)), "L-DU", True)
        s.Lb, s.Ub = S.Csr2Bcsr(Lf, 3, 3), S.Csr2Bcsr(Uf, 3, 3)
    else:
        A = _pad(A, BSIZE)
        s.cnum, s.cptr, LP, RP = S.GetABMCPermutation(A.cind, A.rptr, A.n, BSIZE, False, "connect")
        s.A = S.Reordering(A, LP, RP)
        s.Lf, s.Uf, _ = S.Split(S.Ilu0(s.A), "L-DU", True)
    return s


@functools.lru_cache(maxsize=2)
def _bcsr(n):
    return S.Csr2Bcsr(_matrix("block27", n), 3, 3)


def _order(case):
    return case.get("order", "abmc")


def _np(case):
    return np.float32 if case.get("dtype", "f64") == "f32" else np.float64


def _t(case):
    return torch.float32 if case.get("dtype", "f64") == "f32" else torch.float64


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _vec(n, seed, dtype=torch.float64):
    """U(-1, 1) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1).to(dtype)


def _params():
    p = LN.init_params(2)
    p[LN.OFF_WOUT:LN.OFF_BOUT] = 0.05
    return p


# --------------------------------------------------------- prepare and run

class _Handle:
    """An ILU or ILUB plan."""

    def __init__(self):
        self.h = C.c_void_p()

    def __del__(self):
        if self.h:
            L.lib().senk_ilu_plan_destroy(self.h)


class _View:
    """A system's device buffer for torch.as_tensor; keeps the system alive."""

    def __init__(self, owner, ptr, n, dtype):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=np.dtype(dtype).str, data=(int(ptr), False), version=3)


def _system(case, s, m):
    T = _np(case)
    cast = (lambda A: A) if T == np.float64 else (lambda A: A.astype(T))
    return System(cast(s.A), cast(s.Lf), cast(s.Uf), L.PC_ILU_ABMC, s.cptr, s.cnum, BSIZE, dtype=T, m_max=m)


def _rhs(case, s, seed):
    """(b, x_true) with b = A x_true, x_true ~ U(-1, 1)."""
    xt = np.random.default_rng(seed).uniform(-1.0, 1.0, s.A.n)
    return s.A.matvec(xt), xt


def prepare(case, seed):
    k, st = case["kind"], dict(case=case)
    if k in ("cg", "spmv"):
        A = _matrix(case["problem"], case["n"])
        st.update(n=A.n, nnz=A.nnz, val=_dev(A.val.astype(_np(case))), cind=_dev(A.cind), rptr=_dev(A.rptr),
                  x=_vec(A.n, seed, _t(case)))
        for v in ("y",) if k == "spmv" else ("sol", "r", "p", "q"):
            st[v] = torch.empty_like(st["x"])
    elif k == "bcsr":
        bval, bcind, brptr = _bcsr(case["n"])
        n = 3 * (len(brptr) - 1)
        st.update(n=n, val=_dev(bval), cind=_dev(bcind), rptr=_dev(brptr), x=_vec(n, seed))
        st["y"] = torch.empty_like(st["x"])
    elif k in ("ilu", "ilub"):
        s, T, h = _setup(case["problem"], case["n"], _order(case)), _np(case), _Handle()
        cptr = None if s.cptr is None else np.ascontiguousarray(s.cptr, np.int32)
        if k == "ilub":
            L.check("plan", L.lib().senk_ilub_plan_create(C.byref(h.h), s.A.n, 3, 3, *[L.ptr(a) for a in s.Lb + s.Ub],
                                                          L.ptr(cptr), s.cnum, 3 * NODES))
        else:
            lv, uv = s.Lf.val.astype(T), s.Uf.val.astype(T)
            L.check("plan", L.lib().senk_ilu_plan_create(
                C.byref(h.h), L.F32 if T == np.float32 else L.F64, s.A.n, L.ptr(lv), L.ptr(s.Lf.cind),
                L.ptr(s.Lf.rptr), L.ptr(uv), L.ptr(s.Uf.cind), L.ptr(s.Uf.rptr),
                L.PC_ILU if cptr is None else L.PC_ILU_ABMC, L.ptr(cptr), s.cnum, 1 if cptr is None else BSIZE))
        st.update(plan=h, x=_vec(s.A.n, seed, _t(case)))
        st["y"] = torch.empty_like(st["x"])
    elif k in ("gmres", "gcr", "bicgstab"):
        s, T = _setup(case["problem"], case["n"], "abmc"), _np(case)
        b, _ = _rhs(case, s, seed)
        st["sys"] = _system(case, s, 30 if k == "gmres" else 0)
        st["sys"].set_rhs(b)
        st["nrm_b"] = float(np.linalg.norm(b))
        st["x"] = torch.as_tensor(_View(st["sys"], st["sys"].x_ptr, s.A.n, T), device="cuda")
    else:
        s = _setup(case["problem"], case["n"], "abmc")
        st["sys"], st["net"] = _system(case, s, 0), LN.Net(_params())
        st["net"].bind(st["sys"])
        st["r"], st["e"] = _vec(s.A.n, seed), 0.05 * _vec(s.A.n, seed + (1 << 31))
    torch.cuda.synchronize()
    return st


def run(st):
    lib, case = L.lib(), st["case"]
    k = case["kind"]
    cu = torch.cuda.current_stream().cuda_stream
    if k == "spmv":
        f = lib.senk_dev_spmv_csr_s if case["dtype"] == "f32" else lib.senk_dev_spmv_csr_d
        L.check("spmv", f(st["val"].data_ptr(), st["cind"].data_ptr(), st["rptr"].data_ptr(), st["x"].data_ptr(),
                          st["y"].data_ptr(), st["n"], st["nnz"], cu))
        return st["y"]
    if k == "bcsr":
        L.check("bcsr", lib.senk_dev_spmv_bcsr_d(st["val"].data_ptr(), st["cind"].data_ptr(), st["rptr"].data_ptr(),
                                                 st["x"].data_ptr(), st["y"].data_ptr(), st["n"], 3, 3, cu))
        return st["y"]
    if k in ("ilu", "ilub"):
        L.check("apply", lib.senk_ilu_plan_apply(st["plan"].h, st["x"].data_ptr(), st["y"].data_ptr(), cu))
        return st["y"]
    if k == "cg":
        return _run_cg(lib, st, cu)
    if k == "learned":
        loss, grad = st["net"].loss_grad(st["sys"], st["r"].data_ptr(), st["e"].data_ptr())
        return dict(loss=np.float64(loss), grad=grad)
    sysm = st["sys"]
    sysm.zero_x()
    if k == "gmres":
        r = sysm.gmres(st["nrm_b"], case["outer"], 30, case["eps"])
    elif k == "gcr":
        r = sysm.gcr(st["nrm_b"], 1, case["its"], 1e-14)
    else:
        r = sysm.bicgstab(st["nrm_b"], case["its"], 1e-14)
    return dict(x=st["x"], iters=int(r.iters))


def _run_cg(lib, st, cu):
    """Eight CG iterations from x = 0 on the blas1 and SpMV calls."""
    n, d = st["n"], C.c_double()
    val, cind, rptr, b, x, r, p, q = (st[v].data_ptr() for v in ("val", "cind", "rptr", "x", "sol", "r", "p", "q"))

    def dot(u, v):
        L.check("dot", lib.senk_dev_dot_d(u, v, n, C.byref(d), cu))
        return d.value

    L.check("copy", lib.senk_dev_copy_d(b, r, n, cu))
    L.check("copy", lib.senk_dev_copy_d(b, p, n, cu))
    L.check("copy", lib.senk_dev_copy_d(b, x, n, cu))
    L.check("scal", lib.senk_dev_scal_d(0.0, x, n, cu))
    rr = dot(r, r)
    for _ in range(8):
        L.check("spmv", lib.senk_dev_spmv_csr_d(val, cind, rptr, p, q, n, st["nnz"], cu))
        a = rr / dot(p, q)
        L.check("axpy", lib.senk_dev_axpy_d(a, p, x, n, cu))
        L.check("axpy", lib.senk_dev_axpy_d(-a, q, r, n, cu))
        new = dot(r, r)
        L.check("axpby", lib.senk_dev_axpby_d(1.0, r, new / rr, p, n, cu))
        rr = new
    return dict(x=st["sol"], r=st["r"], rr=np.float64(rr))


# -------------------------------------------------------------------- work

def _sizes(case):
    """(rows, entries) of the case's matrix."""
    n = case["n"]
    if case["problem"] == "poisson2d":
        return n * n, 5 * n * n - 4 * n
    if case["problem"] == "block27":
        return 3 * n ** 3, 9 * (3 * n - 2) ** 3
    return n ** 3, 7 * n ** 3 - 6 * n * n


def work(case):
    k, vb = case["kind"], np.dtype(_np(case)).itemsize
    N, nnz = _sizes(case)
    spmv = (vb + 4) * nnz + 4 * N + 2 * vb * N
    ilu = (vb + 4) * (nnz - N) + 8 * N + 3 * vb * N       # both factors, x in, y out
    if k == "cg":                                          # per iteration: A p, two dots, three updates
        return dict(bytes=8 * (spmv + 10 * vb * N), flops=8 * (2 * nnz + 10 * N))
    if k == "spmv":
        return dict(bytes=spmv, flops=2 * nnz)
    if k == "bcsr":
        return dict(bytes=(8 + 4 / 9) * nnz + 4 * N / 3 + 16 * N, flops=2 * nnz)
    if k == "ilu":
        return dict(bytes=ilu, flops=2 * nnz)
    if k == "ilub":
        return dict(bytes=(8 + 4 / 9) * (nnz + 9 * N / 3) + 4 * 2 * N / 3 + 16 * N, flops=2 * nnz)
    if k == "learned":                                     # activations of 4 layers of width 64, forward and backward
        return dict(bytes=4 * (2 * 896 + 1200) * N + 40 * nnz, flops=3 * 4 * 2 * 128 * 64 * N)
    if k == "gmres":                                       # about 1.15 n iterations to 1e-8, a fifth of them to 1e-4
        its = 1.15 * case["n"] * (1.0 if case["eps"] < 1e-6 else 0.2)
        mean = 15.0                                        # basis vectors of a mid-cycle Arnoldi step, read twice
        return dict(bytes=its * (spmv + ilu + vb * N * (2 * mean + 2)), flops=its * (4 * nnz + 4 * mean * N))
    per = 2 if k == "bicgstab" else 1
    vec = 14 if k == "bicgstab" else 4 + 2 * case["its"]
    return dict(bytes=case["its"] * (per * (spmv + ilu) + vec * vb * N), flops=case["its"] * (per * 4 * nnz + 2 * vec * N))


# ------------------------------------------------------------------- exact
# The same results from plain torch in 64 bits.

def _rows(rptr):
    r = _dev(rptr).long()
    return torch.repeat_interleave(torch.arange(r.numel() - 1, device=r.device), r[1:] - r[:-1])


def _csr64(A, dtype=np.float64):
    """x -> A x in float64, the values rounded to `dtype` first."""
    rows, col, val = _rows(A.rptr), _dev(A.cind).long(), _dev(A.val.astype(dtype).astype(np.float64))
    return lambda x: torch.zeros_like(x).index_add_(0, rows, val * x[col])


def _levels(case, s):
    """Row sets of the forward sweep in order: the rows of a set depend on earlier sets only."""
    if _order(case) == "natural":                          # 5-point grid: diagonals i + j
        n = case["n"]
        i, j = np.arange(n * n) % n, np.arange(n * n) // n
        return [np.nonzero(i + j == d)[0] for d in range(2 * n - 1)]
    if case["problem"] == "block27":                       # block rows: k-th node of every block of a colour
        nb = s.A.n // 3
        return [b[b < nb] for c in range(s.cnum) for b in
                (np.arange(s.cptr[c], s.cptr[c + 1]) * NODES + k for k in range(NODES))]
    return [np.arange(s.cptr[c], s.cptr[c + 1]) * BSIZE + k for c in range(s.cnum) for k in range(BSIZE)]


def _ilu64(case, s, dtype=np.float64):
    """x -> U^-1 L^-1 x in float64 with the factors' values rounded to `dtype`."""
    steps = []
    for F, upper in ((s.Lf, False), (s.Uf, True)):
        val = F.val.astype(dtype).astype(np.float64)
        cnt = np.diff(F.rptr).astype(np.int64)
        lev = _levels(case, s)
        for rows in (lev[::-1] if upper else lev):
            m = cnt[rows]
            at = np.repeat(F.rptr[rows].astype(np.int64) - (np.cumsum(m) - m), m) + np.arange(m.sum())
            own = np.repeat(np.arange(rows.size), m)
            if upper:                                      # the inverted diagonal comes first
                off = F.cind[at] != rows[own]
                di = _dev(val[F.rptr[rows]])
                at, own = at[off], own[off]
            else:
                di = None
            steps.append((_dev(rows.astype(np.int64)), _dev(own), _dev(F.cind[at].astype(np.int64)), _dev(val[at]), di))

    def apply(x):
        y = x.clone()
        for rows, own, col, v, di in steps:
            t = y[rows].index_add_(0, own, v * y[col], alpha=-1.0)
            y[rows] = t if di is None else t * di
        return y
    return apply


def _ilub64(case, s, x):
    """The block sweeps as the reference's compiled code reads them: within an L
    block row, a column inside the row is read after the pairs of rows before it
    were updated."""
    lev, y = _levels(case, s), x.clone()
    nb = s.A.n // 3
    for (bval, bcind, brptr), upper in ((s.Lb, False), (s.Ub, True)):
        val, col, ptr = _dev(bval).reshape(-1, 3, 3), _dev(bcind).long(), _dev(brptr).long()
        for rows in (lev[::-1] if upper else lev):
            if not rows.size:
                continue
            br = _dev(rows.astype(np.int64))
            i0, b0, b1 = 3 * br, ptr[br], ptr[br + 1]
            lane = torch.arange(3, device=br.device)
            t = y.reshape(nb, 3)[br]
            first = 1 if upper else 0
            most = int((b1 - b0).max()) - first
            for u in range(most):
                j = b1 - 1 - u if upper else b0 + u
                on = (j >= b0 + first) if upper else (j < b1)
                j = torch.where(on, j, torch.zeros_like(j))
                for l in range(3):
                    c = 3 * col[j] + l
                    v = val[j, l] * on[:, None]
                    rel = c - i0
                    inside = (rel >= 0) & (rel < 3) & on
                    t_out = t - v * y[c][:, None]
                    if upper or not bool(inside.any()):
                        t = t_out
                        continue
                    at = rel.clamp(0, 2)[:, None]
                    t0 = t - v * t.gather(1, at)
                    t_in = torch.where((lane[None] >> 1) > (at >> 1), t - v * t0.gather(1, at), t0)
                    t = torch.where(inside[:, None], t_in, t_out)
            if upper:                                      # the diagonal block, its diagonal inverted
                d = val[b0]
                for q in (2, 1, 0):
                    t[:, q] *= d[:, q, q]
                    t[:, :q] -= d[:, q, :q] * t[:, q:q + 1]
            y.reshape(nb, 3)[br] = t
    return y


def exact(case, seed):
    k, T = case["kind"], _np(case)
    if k in ("spmv", "cg"):
        A = _matrix(case["problem"], case["n"])
        mv, b = _csr64(A, T), _vec(A.n, seed, _t(case)).double()
        if k == "spmv":
            return mv(b)
        x, r, p, rr = torch.zeros_like(b), b.clone(), b.clone(), b @ b
        for _ in range(8):
            q = mv(p)
            a = rr / (p @ q)
            x, r = x + a * p, r - a * q
            new = r @ r
            p, rr = r + (new / rr) * p, new
        return dict(x=x, r=r, rr=np.float64(float(rr)))
    if k == "bcsr":
        bval, bcind, brptr = _bcsr(case["n"])
        nb = len(brptr) - 1
        x = _vec(3 * nb, seed).reshape(nb, 3)
        part = torch.einsum("blr,bl->br", _dev(bval).reshape(-1, 3, 3), x[_dev(bcind).long()])
        return torch.zeros_like(x).index_add_(0, _rows(brptr), part).reshape(-1)
    s = _setup(case["problem"], case["n"], _order(case))
    if k == "ilu":
        return _ilu64(case, s, T)(_vec(s.A.n, seed, _t(case)).double())
    if k == "ilub":
        return _ilub64(case, s, _vec(s.A.n, seed))
    if k == "learned":
        return _learned64(case, s, seed)
    b, xt = _rhs(case, s, seed)
    if k == "gmres":                                       # the solution itself
        return dict(x=xt, iters=None)
    mv, pc, b = _csr64(s.A), _ilu64(case, s), _dev(b)
    x, r = torch.zeros_like(b), b.clone()
    if k == "gcr":
        ps, aps = [pc(r)], []
        aps.append(mv(ps[0]))
        for j in range(case["its"]):
            d = aps[j] @ aps[j]
            a = (aps[j] @ r) / d
            x, r = x + a * ps[j], r - a * aps[j]
            z = pc(r)
            az = mv(z)
            be = [-(ap @ az) / (ap @ ap) for ap in aps]
            ps.append(z + sum(c * p for c, p in zip(be, ps)))
            aps.append(az + sum(c * p for c, p in zip(be, aps)))
    else:
        rs, p, rho = r.clone(), r.clone(), r @ r
        for _ in range(case["its"]):
            kp = pc(p)
            akp = mv(kp)
            a = rho / (akp @ rs)
            t = r - a * akp
            ks = pc(t)
            aks = mv(ks)
            w = (aks @ t) / (aks @ aks)
            x, r = x + a * kp + w * ks, t - w * aks
            new = r @ rs
            p, rho = r + (a / w) * (new / rho) * (p - w * akp), new
    return dict(x=x, iters=None)


def _learned64(case, s, seed):
    """Loss and gradient of the network in float64 (no BF16 rounding), by autograd."""
    A, H = s.A, LN.HID
    n, rows, col = A.n, _rows(A.rptr), _dev(A.cind).long()
    val = _dev(A.val)
    r = _vec(n, seed)
    mv, ilu = _csr64(A), _ilu64(case, s)(r)
    off = torch.where(rows == col, torch.zeros_like(val), val.abs())
    diag = torch.zeros_like(r).index_add_(0, rows, torch.where(rows == col, val, torch.zeros_like(val)))
    osum = torch.zeros_like(r).index_add_(0, rows, off)
    w = off / osum.clamp_min(1e-300)[rows]
    d = float(diag.sum() / n)
    rms = float(torch.sqrt(r @ r / n))
    p = _dev(_params().astype(np.float64)).requires_grad_()
    feat = torch.stack([diag / d, (osum + diag.abs()) / d, r / rms], 1)
    h = torch.relu(feat @ p[LN.OFF_WIN:LN.OFF_BIN].reshape(LN.NIN, H) + p[LN.OFF_BIN:LN.OFF_LAYER])
    for l in range(LN.LAYERS):
        o = LN.OFF_LAYER + l * LN.LAYER_SIZE
        m = torch.zeros_like(h).index_add(0, rows, w[:, None] * h[col])
        z = torch.cat([h, m], 1) @ p[o:o + 2 * H * H].reshape(2 * H, H) + p[o + 2 * H * H:o + LN.LAYER_SIZE]
        h = h + torch.relu(z)
    c = h @ p[LN.OFF_WOUT:LN.OFF_BOUT] + p[LN.OFF_BOUT]
    q = (r - mv(ilu)) / rms
    res = torch.zeros_like(c).index_add(0, rows, val * c[col]) / d - q
    loss = (res @ res) / (q @ q)
    loss.backward()
    return dict(loss=np.float64(float(loss.detach())), grad=p.grad.detach().cpu().numpy())
