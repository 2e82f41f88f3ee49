"""Sweeps enqueued one after another without a wait between them, the output of
one being the input of the next: plans with different colourings, the same
triangle of a two-colour plan twice, a plan whose L and U have different layouts."""
import numpy as np
import pytest

from senk_gb300 import lib as L
from senk_gb300 import problems as P
from senk_gb300 import setup as S
from test_gpu_kernels import Plan, _factors
from test_gpu_krylov import IlubPlan

pytestmark = pytest.mark.gpu

ROUNDS, INPUTS = 40, 3
TOL = {np.float64: 1e-12, np.float32: 1e-5}


def _chain(calls, xs, want, tol):
    """calls: f(x, y) in order, each reading the output of the one before."""
    import torch
    xd = [torch.from_numpy(x).cuda() for x in xs]
    n = len(xs[0])
    out = torch.zeros((ROUNDS, n), dtype=xd[0].dtype, device="cuda")
    mid = torch.full((len(calls), n), 3.0, dtype=xd[0].dtype, device="cuda")   # rewritten in every round
    torch.cuda.synchronize()
    for i in range(ROUNDS):
        x = xd[i % INPUTS].data_ptr()
        for k, f in enumerate(calls):
            y = out[i].data_ptr() if k + 1 == len(calls) else mid[k].data_ptr()
            L.check("sweep", f(x, y))
            x = y
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    for i in range(ROUNDS):
        w = want[i % INPUTS]
        assert np.max(np.abs(got[i] - w)) <= tol * np.max(np.abs(w)), i


def _apply(h):
    return lambda x, y: L.lib().senk_ilu_plan_apply(h, x, y, None)


def _inputs(n, dtype):
    return [np.random.default_rng(i).uniform(-1, 1, n).astype(dtype) for i in range(INPUTS)]


# (schedule, block size, sweep) of the plan before and of the plan after
@pytest.mark.parametrize("before,after", [
    (("abmc", 16, L.SWEEP_AUTO), ("abmc", 8, L.SWEEP_AUTO)),
    (("abmc", 8, L.SWEEP_AUTO), ("abmc", 16, L.SWEEP_AUTO)),
    (("abmc", 16, L.SWEEP_COLOURS), ("abmc", 16, L.SWEEP_AUTO)),
    (("natural", 16, L.SWEEP_AUTO), ("abmc", 16, L.SWEEP_AUTO)),
    (("abmc", 4, L.SWEEP_COMPACT), ("abmc", 16, L.SWEEP_COMPACT)),
    (("abmc", 4, L.SWEEP_WIDE), ("abmc", 16, L.SWEEP_WIDE)),
    (("abmc", 16, L.SWEEP_AUTO), ("abmc", 16, L.SWEEP_ROWS_WIDE))])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_two_plans(port, before, after, dtype):
    A = P.convdiff3d(32, 0.5)       # 256 KB of FP64: the natural order runs level set by level set
    plans, fac = [], []
    for sched, bs, sweep in (before, after):
        _, Lf, Uf, sc, nc, pc, b = _factors(A, sched, bs)
        plans.append(Plan(Lf, Uf, pc, sc, nc, b, dtype, sweep=sweep))
        L.check("plan", plans[-1].code)
        fac.append((Lf.astype(dtype), Uf.astype(dtype)))
    xs = _inputs(A.n, dtype)
    want = []
    for x in xs:
        for Lf, Uf in fac:
            x = port.sptrsv(Uf, port.sptrsv(Lf, x, False), True)
        want.append(x)
    _chain([_apply(p.h) for p in plans], xs, want, 10 * TOL[dtype])
    for p in plans:
        L.check("status", L.lib().senk_ilu_plan_status(p.h, None))


def _two_colours(port, which, dtype):
    """Red-black colouring of a 5-point grid: two colours of single rows."""
    A = P.poisson2d(200)            # FP64 and FP32 vectors too large for the one-CTA sweep (FP32: 156 KB)
    _, Lf, Uf, sc, nc, pc, b = _factors(A, "amc", 16)
    assert nc == 2
    plan = Plan(Lf, Uf, pc, sc, nc, b, dtype, sweep=L.SWEEP_AUTO if dtype == np.float64 else L.SWEEP_ROWS)
    L.check("plan", plan.code)
    return plan, (Uf if which else Lf).astype(dtype), A.n


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("which", [0, 1])
def test_the_same_triangle_twice(port, which, dtype):
    plan, F, n = _two_colours(port, which, dtype)
    xs = _inputs(n, dtype)
    want = [port.sptrsv(F, port.sptrsv(F, x, bool(which)), bool(which)) for x in xs]
    f = lambda x, y: L.lib().senk_ilu_plan_sweep(plan.h, which, x, y, None)     # noqa: E731
    _chain([f, f], xs, want, 10 * TOL[dtype])


def _thinned(U, keep):
    """Rows of U with their diagonal and every keep-th other entry."""
    sel = np.zeros(len(U.val), bool)
    for i in range(U.n):
        sel[U.rptr[i]] = True
        sel[U.rptr[i] + 1:U.rptr[i + 1]:keep] = True
    rptr = np.concatenate([[0], np.cumsum(np.add.reduceat(sel, U.rptr[:-1]))]).astype(np.int32)
    return P.Csr(U.val[sel].copy(), U.cind[sel].copy(), rptr)


def test_row_slots_for_l_and_slices_for_u(port):
    """Groups of L too large for the slices' shared memory, groups of U within it."""
    A = S.AllocLevelZero(P.block27(8), 1)
    nc, sc, LP, RP = S.GetABMCPermutation(A.cind, A.rptr, A.n, 32, False, "connect")
    Lf, Uf, _ = S.Split(S.Ilu0(S.Reordering(A, LP, RP)), "L-DU", True)
    Uf = _thinned(Uf, 8)
    plan = Plan(Lf, Uf, L.PC_ILU_ABMC, sc, nc, 32, np.float64)
    L.check("plan", plan.code)
    xs = _inputs(A.n, np.float64)
    want = [port.sptrsv(Uf, port.sptrsv(Lf, x, False), True) for x in xs]
    _chain([_apply(plan.h)], xs, want, TOL[np.float64])


def test_two_ilub_plans(port):
    A, G = P.block27(8), P.block27_node_graph(8)
    plans, fac = [], []
    for nodes in (4, 8):
        nc, sc, LPn, _ = S.GetABMCPermutation(G.cind, G.rptr, G.n, nodes, False, "connect")
        LP, RP = P.expand_node_permutation(LPn, 3)
        Lf, Uf, _ = S.Split(S.Ilu0(S.AllocBlockZero(S.Reordering(A, LP, RP), 3, 3)), "L-DU", True)
        fac.append((S.Csr2Bcsr(Lf, 3, 3), S.Csr2Bcsr(Uf, 3, 3), sc, nc, 3 * nodes))
        plans.append(IlubPlan(*fac[-1][:2], A.n, 3, 3, *fac[-1][2:]))
        L.check("plan", plans[-1].code)
    for order in ((0, 1), (1, 0)):
        xs, want = _inputs(A.n, np.float64), []
        for x in xs:
            for k in order:
                bl, bu, sc, nc, bs = fac[k]
                x = port.ilub_sweep(bu, port.ilub_sweep(bl, x, False, 3, 3, sc, nc, bs), True, 3, 3, sc, nc, bs)
            want.append(x)
        _chain([_apply(plans[k].h) for k in order], xs, want, 10 * TOL[np.float64])
