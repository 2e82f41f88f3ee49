"""A plan built or used beside another one: each keeps what its kernels need of
the device, whatever plan of the same kind was built after it."""
import numpy as np
import pytest

from senk_gb300 import lib as L
from senk_gb300 import problems as P
from senk_gb300 import setup as S
from senk_gb300 import solver as SV
from test_gpu_ilub_slices import _block_system
from test_gpu_kernels import Plan, _factors
from test_gpu_krylov import IlubPlan

pytestmark = pytest.mark.gpu

# a factor with large groups, one with small groups, both on the same kernels
BIG_SMALL = {
    "slices": (lambda: P.block27(8), lambda: P.convdiff3d(16, 0.5), "abmc", 16, L.SWEEP_AUTO, np.float64),
    "rows": (lambda: P.block27(8), lambda: P.convdiff3d(16, 0.5), "abmc", 4, L.SWEEP_AUTO, np.float32),
    "rows, two chains a lane": (lambda: P.block27(8), lambda: P.convdiff3d(16, 0.5), "abmc", 4, L.SWEEP_ROWS_WIDE,
                                np.float32),
    "compact": (lambda: P.block27(8), lambda: P.convdiff3d(16, 0.5), "abmc", 4, L.SWEEP_COMPACT, np.float64),
    "wide": (lambda: P.block27(8), lambda: P.convdiff3d(16, 0.5), "abmc", 4, L.SWEEP_WIDE, np.float64),
    "cooperative": (lambda: P.block27(8), lambda: P.convdiff3d(16, 0.5), "abmc", 4, L.SWEEP_PERSISTENT, np.float32),
    "dataflow": (lambda: P.block27(8), lambda: P.convdiff3d(8, 0.5), "abmc", 4, L.SWEEP_DATAFLOW, np.float64),
    "one CTA": (lambda: P.poisson2d(128), lambda: P.poisson2d(4), "natural", 16, L.SWEEP_AUTO, np.float64),
}


def _apply(torch, h, x):
    y = torch.from_numpy(x).cuda()
    L.check("apply", L.lib().senk_ilu_plan_apply(h, y.data_ptr(), y.data_ptr(), None))
    L.check("status", L.lib().senk_ilu_plan_status(h, None))
    return y.cpu().numpy()


@pytest.mark.parametrize("kind", BIG_SMALL)
def test_ilu_plan_after_a_smaller_one(port, kind):
    import torch
    big, small, sched, bs, sweep, dtype = BIG_SMALL[kind]
    plans = []
    for A in (big(), small()):
        _, Lf, Uf, sc, nc, pc, b = _factors(A, sched, bs)
        plans.append((Plan(Lf, Uf, pc, sc, nc, b, dtype, sweep=sweep), Lf.astype(dtype), Uf.astype(dtype)))
        L.check("plan", plans[-1][0].code)
    tol = 1e-12 if dtype == np.float64 else 1e-5
    for pl, Lf, Uf in plans + plans[:1]:
        x = np.random.default_rng(Lf.n).uniform(-1, 1, Lf.n).astype(dtype)
        want = port.sptrsv(Uf, port.sptrsv(Lf, x, False), True)
        assert np.max(np.abs(_apply(torch, pl.h, x) - want)) <= tol * np.max(np.abs(want))


def test_ilub_plan_after_a_smaller_one(port):
    """Chains of eight 3x3 block rows (groups of 75 KB), then of four."""
    import torch
    A, G = P.block27(8), P.block27_node_graph(8)
    nc, sc, LPn, _ = S.GetABMCPermutation(G.cind, G.rptr, G.n, 8, False, "connect")
    LP, RP = P.expand_node_permutation(LPn, 3)
    Lf, Uf, _ = S.Split(S.Ilu0(S.AllocBlockZero(S.Reordering(A, LP, RP), 3, 3)), "L-DU", True)
    cases = [(S.Csr2Bcsr(Lf, 3, 3), S.Csr2Bcsr(Uf, 3, 3), sc, nc, 24, A.n)]
    Ar, bl, bu, sc, nc = _block_system(6)
    cases.append((bl, bu, sc, nc, 12, Ar.n))
    plans = [IlubPlan(bl, bu, n, 3, 3, sc, nc, bsize) for bl, bu, sc, nc, bsize, n in cases]
    for i in (0, 1, 0):
        bl, bu, sc, nc, bsize, n = cases[i]
        L.check("plan", plans[i].code)
        x = np.random.default_rng(n).uniform(-1, 1, n)
        want = port.ilub_sweep(bu, port.ilub_sweep(bl, x, False, 3, 3, sc, nc, bsize), True, 3, 3, sc, nc, bsize)
        assert np.max(np.abs(_apply(torch, plans[i].h, x) - want)) <= 1e-12 * np.max(np.abs(want))


def test_two_cached_systems_in_turn():
    """Two systems that the drop-in entries keep, used in turn; each call's
    restart length is new to its system, so its cycle is captured again."""
    L.lib().senk_dropin_cache(1)
    systems = []
    for A in (P.block27(8), P.convdiff3d(16, 0.5)):
        Ar, Lf, Uf, sc, nc, _, _ = _factors(A, "abmc", 16)
        systems.append((Ar, Lf, Uf, sc, nc, Ar.matvec(np.random.default_rng(2).uniform(-1, 1, Ar.n))))
    for i, m in ((0, 30), (1, 30), (0, 20), (1, 20)):
        Ar, Lf, Uf, sc, nc, b = systems[i]
        x = np.zeros(Ar.n)
        r = SV.AbmcIluGmresm(Ar.val, Ar.cind, Ar.rptr, Lf.val, Lf.cind, Lf.rptr, Uf.val, Uf.cind, Uf.rptr, sc, nc, 16,
                             b, x, float(np.linalg.norm(b)), 100, m, Ar.n, 1e-8)
        assert r.converged and np.linalg.norm(b - Ar.matvec(x)) <= 2e-8 * np.linalg.norm(b)
