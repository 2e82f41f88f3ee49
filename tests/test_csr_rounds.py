"""The tiles, rounds and copies of the CSR product at the ends of int's range:
the kernel's own index arithmetic (csr_rounds.hpp), walked on the host."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
INT_MAX = 2 ** 31 - 1


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("csr") / "libcsrwalk.so")
    cmd = ["g++", "-O1", "-std=c++17", "-fsanitize=undefined", "-fno-sanitize-recover", "-shared", "-fPIC", "-I",
           os.path.join(ROOT, "senk_gb300", "csrc"), os.path.join(ROOT, "tests", "cpp", "csr_rounds.cpp"), "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(out)

    def f(n, nnz, tile, rp, cap, size):
        rp, err = np.asarray(rp, np.int32), C.create_string_buffer(256)
        assert rp.min() >= 0 and rp.max() <= nnz
        rc = lib.csr_walk(n, nnz, tile, rp.ctypes.data_as(C.c_void_p), cap, size, err, 256)
        assert rc == 0, err.value.decode()
    return f


@pytest.mark.parametrize("size", [4, 8])
@pytest.mark.parametrize("nnz", [7 * 32, 2 ** 28 - 1, 2 ** 28, 2 ** 28 + 5, 2 ** 29 - 1, 2 ** 29, 2 ** 29 + 3, 2 ** 30,
                                 INT_MAX - 2000, INT_MAX])
@pytest.mark.parametrize("per", [7, 40, 1000])
def test_first_and_last_tile(walk, nnz, per, size):
    """The first tile, before which all entries lie, and the last one, in one
    round and in several."""
    per = min(per, nnz // 32)
    cap = max(256, (per * 36 + 63) // 64 * 64) if per <= 40 else 256
    n = nnz // 7
    rows = np.arange(33, dtype=np.int64) * per
    walk(n, nnz, 0, rows, cap, size)
    walk(n, nnz, n // 32 - 1, rows + nnz - 32 * per, cap, size)       # ends with the arrays


@pytest.mark.parametrize("n", [1, 31, 32, 33, INT_MAX - 32, INT_MAX - 31, INT_MAX - 1, INT_MAX])
def test_tiles_of_the_most_rows(walk, n):
    """The last tile, with rows past the last one, of matrices of up to 2^31 - 1 rows."""
    live = (n - 1) % 32 + 1
    rp = np.minimum(np.arange(33), live).astype(np.int64) + (n - live)
    walk(n, n, (n - 1) // 32, rp, 256, 8)
