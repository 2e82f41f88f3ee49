"""ABMC ILUB sweeps at the edges of the slice layout (k_ilub_slices): chains of
one to sixteen block rows and one past that (k_ilub_sweep), groups with few
chains, and the 27-point block system, against the oracle."""
import numpy as np
import pytest

from senk_gb300 import lib as L
from senk_gb300 import problems as P
from senk_gb300 import setup as S
from senk_gb300.solver import System
from test_gpu_krylov import IlubPlan, _ilub_factors

pytestmark = pytest.mark.gpu


def _block_system(n):
    A, G = P.block27(n), P.block27_node_graph(n)
    nc, sc, LPn, _ = S.GetABMCPermutation(G.cind, G.rptr, G.n, 4, False, "connect")
    LP, RP = P.expand_node_permutation(LPn, 3)
    Ar = S.Reordering(A, LP, RP)
    Lf, Uf, _ = S.Split(S.Ilu0(S.AllocBlockZero(Ar, 3, 3)), "L-DU", True)
    return Ar, S.Csr2Bcsr(Lf, 3, 3), S.Csr2Bcsr(Uf, 3, 3), sc, nc


@pytest.mark.parametrize("bnl,bnw,bsize", [(1, 1, 1), (1, 1, 16), (1, 1, 32), (2, 2, 2), (2, 1, 4), (3, 3, 48),
                                           (4, 2, 16), (8, 1, 16), (8, 2, 64), ("block", 3, 6), ("block", 3, 12)])
def test_abmc_slices(port, bnl, bnw, bsize):
    import torch
    if bnl == "block":        # 3x3 blocks, 4 nodes per ABMC block, n = bsize
        Ar, bl, bu, sc, nc = _block_system(bsize)
        bnl = bnw = 3
        bsize, n = 12, Ar.n
    else:
        A = P.convdiff3d(12, 0.5)
        bl, bu, sc, nc = _ilub_factors(A, bnl, bnw, bsize)
        n = A.n
    plan = IlubPlan(bl, bu, n, bnl, bnw, sc, nc, bsize)
    if plan.code == L.ERR_ARG:    # 1x1 blocks can borrow a later row's entry: refused
        assert (bnl, bnw) == (1, 1)
        return
    L.check("plan", plan.code)
    x = np.random.default_rng(bsize).uniform(-1, 1, n)
    xd = torch.from_numpy(x).cuda()
    yl, ya = torch.empty_like(xd), xd.clone()
    L.check("sweep", L.lib().senk_ilu_plan_sweep(plan.h, 0, xd.data_ptr(), yl.data_ptr(), None))
    L.check("apply", L.lib().senk_ilu_plan_apply(plan.h, ya.data_ptr(), ya.data_ptr(), None))   # in place
    L.check("status", L.lib().senk_ilu_plan_status(plan.h, None))
    wl = port.ilub_sweep(bl, x, False, bnl, bnw, sc, nc, bsize)
    want = port.ilub_sweep(bu, wl, True, bnl, bnw, sc, nc, bsize)
    for got, ref in ((yl, wl), (ya, want)):
        assert np.max(np.abs(got.cpu().numpy() - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("dtype,tol", [(np.float64, 1e-12), (np.float32, 1e-5)])
def test_system_precond(port, dtype, tol):
    """The block system's preconditioner in both precisions."""
    Ar, bl, bu, sc, nc = _block_system(8)
    cast = lambda F: (F[0].astype(dtype), *F[1:])     # noqa: E731
    sy = System(Ar.astype(dtype), cast(bl), cast(bu), L.PC_ILUB_ABMC, sc, nc, 12, dtype=dtype, m_max=1, block=(3, 3))
    x = np.random.default_rng(1).uniform(-1, 1, Ar.n).astype(dtype)
    got = sy.apply_precond(x)
    sy.close()
    wl = port.ilub_sweep(bl, x.astype(np.float64), False, 3, 3, sc, nc, 12)
    want = port.ilub_sweep(bu, wl, True, 3, 3, sc, nc, 12)
    assert np.max(np.abs(got - want)) <= tol * np.max(np.abs(want))


@pytest.mark.parametrize("rows", [67968, 68001, 68352])  # the last: more groups to an SM than the slices take
def test_many_groups(port, rows):
    """Two colours of single 2x2 block rows, red rows first, each black row
    coupled with two red ones, around the group count from which k_ilub_sweep runs."""
    import torch
    rng = np.random.default_rng(rows)
    red = (rows + 1) // 2
    black = np.arange(rows - red)
    pair = np.stack([black, np.minimum(black + 1, red - 1)], 1).astype(np.int32)
    lp = np.zeros(rows + 1, np.int32)
    lp[red + 1:] = 2 * np.arange(1, rows - red + 1)
    bl = (rng.uniform(-.3, .3, 8 * len(black)), pair.reshape(-1), lp)
    up, uc, uv = np.zeros(rows + 1, np.int32), [], []
    cnt = np.where(np.arange(rows) < red, 2, 1)
    cnt[:red][np.arange(red) >= rows - red] = 1    # a red row without a black partner
    up[1:] = np.cumsum(cnt)
    uc = np.zeros(up[-1], np.int32)
    uc[up[:-1]] = np.arange(rows)
    two = np.flatnonzero(cnt == 2)
    uc[up[two] + 1] = red + two
    uv = rng.uniform(-.3, .3, (up[-1], 4))
    uv[up[:-1]] = np.array([1.0, 0.0, 0.2, 0.5])   # inverted diagonal square, column-major
    bu = (uv.reshape(-1), uc, up)
    sc = np.array([0, red, rows], np.int32)
    plan = IlubPlan(bl, bu, 2 * rows, 2, 2, sc, 2, 2)
    L.check("plan", plan.code)
    x = rng.uniform(-1, 1, 2 * rows)
    y = torch.from_numpy(x).cuda()
    L.check("apply", L.lib().senk_ilu_plan_apply(plan.h, y.data_ptr(), y.data_ptr(), None))
    L.check("status", L.lib().senk_ilu_plan_status(plan.h, None))
    want = port.ilub_sweep(bu, port.ilub_sweep(bl, x, False, 2, 2, sc, 2, 2), True, 2, 2, sc, 2, 2)
    assert np.max(np.abs(y.cpu().numpy() - want)) <= 1e-12 * np.max(np.abs(want))
