"""Rounding of the CSR product of short rows: over random rows, no further from
the exact sums than the general kernel (several lanes a row and a tree over
them), at every row length around those where its number of sums changes."""
import numpy as np
import pytest

from senk_gb300 import lib as L

pytestmark = pytest.mark.gpu


def _errors(lens, dtype, seed):
    """Root mean square error of each row class, relative to that of the exact
    sums, of the short-row kernel and of the general one (arrays off a 16-byte
    boundary)."""
    import torch
    rng = np.random.default_rng(seed)
    rptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    n, nnz = len(lens), int(rptr[-1])
    val, x = rng.uniform(-1, 1, nnz).astype(dtype), rng.uniform(-1, 1, n).astype(dtype)
    cind = rng.integers(0, n, nnz).astype(np.int32)
    wide = np.longdouble if dtype == np.float64 else np.float64
    exact = np.add.reduceat(val.astype(wide) * x.astype(wide)[cind], rptr[:-1])
    f = L.lib().senk_dev_spmv_csr_s if dtype == np.float32 else L.lib().senk_dev_spmv_csr_d
    err = []
    for shift in (0, 1):
        v = torch.zeros(nnz + 1, dtype=torch.from_numpy(val).dtype, device="cuda")[shift:shift + nnz]
        c = torch.zeros(nnz + 1, dtype=torch.int32, device="cuda")[shift:shift + nnz]
        v.copy_(torch.from_numpy(val))
        c.copy_(torch.from_numpy(cind))
        r, xd = torch.from_numpy(rptr).cuda(), torch.from_numpy(x).cuda()
        y = torch.empty_like(xd)
        L.check("spmv", f(v.data_ptr(), c.data_ptr(), r.data_ptr(), xd.data_ptr(), y.data_ptr(), n, nnz, None))
        err.append((y.cpu().numpy().astype(wide) - exact).astype(np.float64))
    return err


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("per", [5, 7, 8, 9, 13, 20, 27, 28, 29, 33, 40])
def test_rows_of_one_length(per, dtype):
    rows, general = _errors(np.full(100_000, per), dtype, per)
    assert np.sqrt(np.mean(rows ** 2)) <= np.sqrt(np.mean(general ** 2))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("mean,longer", [(6, (20, 40, 49, 80, 200)), (6, (300, 5000)), (20, (49, 60, 100, 1000))])
def test_longer_rows_among_short_ones(mean, longer, dtype):
    """Rows of one length with longer ones strewn in: four and more in some groups
    of 32 rows, none in others, rows that reach over several staged buffers; each
    length by itself, and the rows around them."""
    rng = np.random.default_rng(mean + len(longer))
    lens = np.full(120_000, mean)
    at = rng.choice(len(lens) // 2, 400 * len(longer), replace=False)     # the second half has none
    for i, k in enumerate(longer):
        lens[at[i::len(longer)]] = k
    assert lens.sum() <= 40 * len(lens)
    rows, general = _errors(lens, dtype, mean)
    for k in (mean, *longer):
        # 400 rows of a length: their root mean square is known to about 4 %
        slack = 1.0 if k == mean else 1.1
        sel = lens == k
        assert np.sqrt(np.mean(rows[sel] ** 2)) <= slack * np.sqrt(np.mean(general[sel] ** 2)), k
