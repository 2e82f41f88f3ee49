"""CSR SpMV on both sides of its dispatch (k_spmv_csr_rows for short mean rows
and aligned arrays, k_spmv_csr otherwise) against FP64 row sums on the host."""
import numpy as np
import pytest

from senk_gb300 import lib as L

pytestmark = pytest.mark.gpu


def _matrix(rng, lens, n):
    rptr = np.zeros(len(lens) + 1, np.int32)
    rptr[1:] = np.cumsum(lens)
    return rng.standard_normal(rptr[-1]), rng.integers(0, n, rptr[-1]).astype(np.int32), rptr


def _lens(kind, n, rng):
    if kind == "empty":
        return np.zeros(n, int)
    if kind == "stencil":
        return np.full(n, 7)
    if kind == "ragged":
        return rng.integers(0, 15, n)
    if kind == "one long row":            # longer than a buffer holds
        k = rng.integers(0, 9, n)
        k[n // 2] = 3001
        return k
    return np.full(n, {"mean 40": 40, "mean 41": 41}[kind])


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("kind,n", [("empty", 40), ("stencil", 1), ("stencil", 31), ("stencil", 33), ("stencil", 20011),
                                    ("ragged", 5000), ("one long row", 900), ("mean 40", 777), ("mean 41", 777)])
@pytest.mark.parametrize("shift", [0, 1])
def test_spmv_csr_rows(kind, n, dtype, shift):
    """shift: val and cind one entry off a 16-byte boundary (the general kernel)."""
    import torch
    rng = np.random.default_rng(n)
    val, cind, rptr = _matrix(rng, _lens(kind, n, rng), n)
    val = val.astype(dtype)
    x = rng.uniform(-1, 1, n).astype(dtype)
    v = torch.zeros(len(val) + 1, dtype=torch.from_numpy(val).dtype, device="cuda")
    c = torch.zeros(len(val) + 1, dtype=torch.int32, device="cuda")
    v, c = v[shift:shift + len(val)], c[shift:shift + len(val)]
    v.copy_(torch.from_numpy(val))
    c.copy_(torch.from_numpy(cind))
    r, xd = torch.from_numpy(rptr).cuda(), torch.from_numpy(x).cuda()
    y = torch.full((n,), 7.0, dtype=xd.dtype, device="cuda")
    f = L.lib().senk_dev_spmv_csr_s if dtype == np.float32 else L.lib().senk_dev_spmv_csr_d
    L.check("spmv", f(v.data_ptr() or r.data_ptr(), c.data_ptr() or r.data_ptr(), r.data_ptr(), xd.data_ptr(),
                      y.data_ptr(), n, int(rptr[-1]), None))
    torch.cuda.synchronize()
    prod = val.astype(np.float64) * x.astype(np.float64)[cind]
    rows = np.repeat(np.arange(n), np.diff(rptr))
    want = np.bincount(rows, weights=prod, minlength=n)
    mag = np.bincount(rows, weights=np.abs(prod), minlength=n)
    bound = (np.diff(rptr) + 1) * np.finfo(dtype).eps * mag   # any order of the additions
    assert np.all(np.abs(y.cpu().numpy() - want) <= bound)
