"""The row-sorted slice layout of the ILU sweeps: its CPU emulation
(tests/cpp/lv_emulate.cpp, every access of k_sweep_lv with its index checked)
and the kernel itself, against the oracle's sequential sweeps."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from senk_gb300 import lib as L
from senk_gb300 import problems as P
from senk_gb300 import setup as S

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# (problem, n, block size): chains of 1 to 32 rows, one partly filled group,
# rows of a dense stencil (smaller groups), several groups per colour
CASES = [("convdiff", 16, 16), ("convdiff", 40, 16), ("convdiff", 16, 2), ("convdiff", 12, 32), ("poisson", 64, 8),
         ("vardiff", 16, 4), ("convdiff", 12, 1), ("poisson", 200, 1), ("block", 8, 4), ("block", 8, 16),
         ("block", 8, 32)]


def _system(kind, n, bs):
    A = {"convdiff": lambda: P.convdiff3d(n, 0.5), "poisson": lambda: P.poisson2d(n),
         "vardiff": lambda: P.vardiff3d(n, 1.5, 4.0, 3), "block": lambda: P.block27(n)}[kind]()
    if bs == 1:
        nc, sc, LP, RP = S.GetAMCPermutation(A.cind, A.rptr, A.n, False)
    else:
        nc, sc, LP, RP = S.GetABMCPermutation(A.cind, A.rptr, A.n, bs, False, "connect")
    Ar = S.Reordering(A, LP, RP)
    Lf, Uf, _ = S.Split(S.Ilu0(Ar), "L-DU", True)
    return Ar, Lf, Uf, nc, np.ascontiguousarray(sc, np.int32)


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("lv") / "liblvemu.so")
    cmd = ["g++", "-O2", "-std=c++17", "-fopenmp", "-ffp-contract=off", "-shared", "-fPIC", "-I",
           os.path.join(ROOT, "senk_gb300", "csrc"), os.path.join(ROOT, "tests", "cpp", "lv_emulate.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind,n,bs", CASES)
def test_emulated_slice_sweep_equals_the_oracle(emu, port, kind, n, bs, dtype):
    Ar, Lf, Uf, nc, sc = _system(kind, n, bs)
    x = np.random.default_rng(7).uniform(-1, 1, Ar.n).astype(dtype)
    f = emu.lv_emulate_s if dtype == np.float32 else emu.lv_emulate_d
    # full groups, groups halved to fit a small buffer, and halved to make many
    for want, spread in ((32 * 1024, 1), (8 * 1024, 1), (32 * 1024, 100)):
        t = x
        for F, upper in ((Lf.astype(dtype), 0), (Uf.astype(dtype), 1)):
            y, err, info = np.zeros_like(t), C.create_string_buffer(256), (C.c_int * 2)()
            rc = f(Ar.n, L.ptr(F.val), L.ptr(F.cind), L.ptr(F.rptr), upper, L.ptr(sc), nc, bs, want, spread, L.ptr(t),
                   L.ptr(y), info, err, 256)
            assert rc == 0, err.value.decode()
            want_y = port.sptrsv(F, t, bool(upper))
            # the same operations, external entries before in-chain ones: rounding only
            tol = 1e-12 if dtype == np.float64 else 1e-5
            assert np.max(np.abs(y - want_y)) <= tol * np.max(np.abs(want_y))
            t = y
        if want < 9000:
            assert info[0] <= 256


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind,n,bs", CASES + [("convdiff", 72, 16)])
def test_slice_sweep_against_the_oracle(port, kind, n, bs, dtype):
    import torch
    Ar, Lf, Uf, nc, sc = _system(kind, n, bs)
    Lf, Uf = Lf.astype(dtype), Uf.astype(dtype)
    h = C.c_void_p()
    amc = bs == 1
    L.check("plan", L.lib().senk_ilu_plan_create(
        C.byref(h), L.F32 if dtype == np.float32 else L.F64, Ar.n, L.ptr(Lf.val), L.ptr(Lf.cind), L.ptr(Lf.rptr),
        L.ptr(Uf.val), L.ptr(Uf.cind), L.ptr(Uf.rptr), L.PC_ILU_AMC if amc else L.PC_ILU_ABMC, L.ptr(sc), nc, bs))
    try:
        x = np.random.default_rng(3).uniform(-1, 1, Ar.n).astype(dtype)
        xd = torch.from_numpy(x).cuda()
        yl, ya = torch.empty_like(xd), xd.clone()
        L.check("sweep", L.lib().senk_ilu_plan_sweep(h, 0, xd.data_ptr(), yl.data_ptr(), None))
        L.check("apply", L.lib().senk_ilu_plan_apply(h, ya.data_ptr(), ya.data_ptr(), None))  # in place
        L.check("status", L.lib().senk_ilu_plan_status(h, None))
        want_l = port.sptrsv(Lf, x, False)
        want = port.sptrsv(Uf, want_l, True)
        tol = 1e-12 if dtype == np.float64 else 1e-5
        assert np.max(np.abs(yl.cpu().numpy() - want_l)) <= tol * np.max(np.abs(want_l))
        assert np.max(np.abs(ya.cpu().numpy() - want)) <= tol * np.max(np.abs(want))
    finally:
        L.lib().senk_ilu_plan_destroy(h)
