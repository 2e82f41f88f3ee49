"""The one-CTA sweeps of small systems (k_ilu_small) in the natural order
against the oracle: one, two and four sets of consumers, rows of up to three
entries and longer ones, levels wider than a set."""
import ctypes as C

import numpy as np
import pytest

from senk_gb300 import lib as L
from senk_gb300 import problems as P
from senk_gb300 import setup as S

pytestmark = pytest.mark.gpu


def _factors(kind, n):
    A = P.poisson2d(n) if kind.startswith("poisson") else P.convdiff3d(n, 0.5)
    if kind == "poisson, one fill level":       # rows of more than three entries
        return S.Split(S.Ilu0(S.AllocLevelZero(A, 1)), "L-DU", True)[:2]
    return S.Split(S.Ilu0(A), "L-DU", True)[:2]


# widest levels: 1, 33, 128, 48, about 190, 430 and 590 rows
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind,n", [("poisson", 1), ("poisson", 33), ("poisson", 128), ("convdiff", 8),
                                    ("convdiff", 16), ("convdiff", 24), ("convdiff", 28),
                                    ("poisson, one fill level", 60)])
def test_small_sweeps(port, kind, n, dtype):
    import torch
    Lf, Uf = (F.astype(dtype) for F in _factors(kind, n))
    h = C.c_void_p()
    L.check("plan", L.lib().senk_ilu_plan_create(
        C.byref(h), L.F32 if dtype == np.float32 else L.F64, Lf.n, L.ptr(Lf.val), L.ptr(Lf.cind), L.ptr(Lf.rptr),
        L.ptr(Uf.val), L.ptr(Uf.cind), L.ptr(Uf.rptr), L.PC_ILU, None, 0, 1))
    try:
        x = np.random.default_rng(n).uniform(-1, 1, Lf.n).astype(dtype)
        xd = torch.from_numpy(x).cuda()
        yl, yu, ya = torch.empty_like(xd), torch.empty_like(xd), xd.clone()
        for _ in range(2):                       # the second run starts from the first's barriers
            L.check("sweep", L.lib().senk_ilu_plan_sweep(h, 0, xd.data_ptr(), yl.data_ptr(), None))
            L.check("sweep", L.lib().senk_ilu_plan_sweep(h, 1, xd.data_ptr(), yu.data_ptr(), None))
        L.check("apply", L.lib().senk_ilu_plan_apply(h, ya.data_ptr(), ya.data_ptr(), None))
        L.check("status", L.lib().senk_ilu_plan_status(h, None))
        wl = port.sptrsv(Lf, x, False)
        tol = 1e-12 if dtype == np.float64 else 1e-5
        for got, want in ((yl, wl), (yu, port.sptrsv(Uf, x, True)), (ya, port.sptrsv(Uf, wl, True))):
            assert np.max(np.abs(got.cpu().numpy() - want)) <= tol * np.max(np.abs(want))
    finally:
        L.lib().senk_ilu_plan_destroy(h)
