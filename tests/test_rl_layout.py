"""The row-per-lane layout (row words, in-chain columns) on the CPU: its
emulation against the oracle's sequential sweeps, with columns repeated in a row
(which a factor may hold) and rows of 128 and more outside entries, whose counts
need two words; and the kernels on the same factors."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from senk_gb300 import lib as L
from senk_gb300 import problems as P
from test_lv_layout import _system

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("rl") / "librlemu.so")
    cmd = ["g++", "-O2", "-std=c++17", "-fopenmp", "-ffp-contract=off", "-shared", "-fPIC", "-I",
           os.path.join(ROOT, "senk_gb300", "csrc"), "-I", "/usr/local/cuda/include",
           os.path.join(ROOT, "tests", "cpp", "rl_emulate.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(out)


def repeated(F, upper, bs, times, which):
    """F with every entry of which(row, column) written `times` times, in equal
    exact parts (times a power of two); U's diagonal stays first and single."""
    val, col, ptr = [], [], [0]
    for i in range(F.n):
        for j in range(F.rptr[i], F.rptr[i + 1]):
            k = times if not (upper and j == F.rptr[i]) and which(i, F.cind[j]) else 1
            val += [F.val[j] / k] * k
            col += [F.cind[j]] * k
        ptr.append(len(col))
    return P.Csr(np.array(val, F.val.dtype), np.array(col, np.int32), np.array(ptr, np.int32))


def in_chain(bs):
    return lambda i, c: i // bs == c // bs


CASES = [("convdiff", 12, 16, 1, None), ("convdiff", 12, 32, 1, None), ("block", 6, 8, 1, None),
         ("convdiff", 12, 16, 8, "in"), ("block", 8, 16, 8, "in"), ("block", 6, 4, 16, "in"),
         ("convdiff", 12, 32, 8, "in"), ("convdiff", 12, 2, 64, "in"),
         ("convdiff", 12, 16, 32, "out"), ("block", 6, 4, 2, "out")]


def factors(kind, n, bs, times, part, dtype=np.float64):
    Ar, Lf, Uf, nc, sc = _system(kind, n, bs)
    which = in_chain(bs)
    if part == "out":                      # in the last row with outside entries only
        which = lambda i, c, f=which: i >= Ar.n - 5 * bs and not f(i, c)    # noqa: E731
    Lf, Uf = Lf.astype(dtype), Uf.astype(dtype)
    return (Lf, Uf, nc, sc) if part is None else (repeated(Lf, False, bs, times, which),
                                                  repeated(Uf, True, bs, times, which), nc, sc)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind,n,bs,times,part", CASES)
def test_emulated_rows_equal_the_oracle(emu, port, kind, n, bs, times, part, dtype):
    Lf, Uf, nc, sc = factors(kind, n, bs, times, part, dtype)
    f = emu.rl_emulate_s if dtype == np.float32 else emu.rl_emulate_d
    t = np.random.default_rng(5).uniform(-1, 1, Lf.n).astype(dtype)
    tol = 1e-12 if dtype == np.float64 else 1e-5
    for F, upper in ((Lf, 0), (Uf, 1)):
        y, err, info = np.zeros_like(t), C.create_string_buffer(256), (C.c_int * 1)()
        rc = f(F.n, L.ptr(F.val), L.ptr(F.cind), L.ptr(F.rptr), upper, L.ptr(sc), nc, bs, L.ptr(t), L.ptr(y), info,
               err, 256)
        assert rc == 0, err.value.decode()
        want = port.sptrsv(F, t, bool(upper)).astype(dtype)
        assert info[0] in (1, 2)           # words a row: the layout takes every factor
        if bs > 16 or (part is not None and not upper):
            assert info[0] == 2
        assert np.max(np.abs(y - want)) <= tol * np.max(np.abs(want))
        t = want


@pytest.mark.gpu
@pytest.mark.parametrize("sweep", [L.SWEEP_ROWS, L.SWEEP_ROWS_WIDE])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind,n,bs,times,part", [c for c in CASES if c[4]])
def test_sweeps_of_two_words_a_row(port, kind, n, bs, times, part, dtype, sweep):
    import torch
    from test_gpu_kernels import Plan
    Lf, Uf, nc, sc = factors(kind, n, bs, times, part, dtype)
    pl = Plan(Lf, Uf, L.PC_ILU_ABMC, sc, nc, bs, dtype, sweep=sweep)
    L.check("plan", pl.code)
    x = np.random.default_rng(6).uniform(-1, 1, Lf.n).astype(dtype)
    y = torch.from_numpy(x).cuda()
    L.check("apply", L.lib().senk_ilu_plan_apply(pl.h, y.data_ptr(), y.data_ptr(), None))
    L.check("status", L.lib().senk_ilu_plan_status(pl.h, None))
    want = port.sptrsv(Uf, port.sptrsv(Lf, x, False), True)
    tol = 1e-12 if dtype == np.float64 else 1e-5
    assert np.max(np.abs(y.cpu().numpy() - want)) <= tol * np.max(np.abs(want))
