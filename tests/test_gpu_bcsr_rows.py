"""The BCSR product with one thread per scalar row: every block shape, block
rows that straddle warps and CTAs, empty block rows, odd and even block counts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from senk_gb300 import lib as L


@pytest.mark.parametrize("bnl,bnw", [(1, 1), (2, 1), (2, 2), (3, 3), (4, 1), (4, 4), (8, 1)])
@pytest.mark.parametrize("rows", [1, 31, 42, 43, 129, 4097])
def test_bcsr_rows(bnl, bnw, rows):
    import torch
    rng = np.random.default_rng(1000 * bnl + 100 * bnw + rows)
    n, nbc = rows * bnl, rows * bnl // bnw if rows * bnl >= bnw else 1
    cnt = rng.integers(0, 8, rows)
    rptr = np.zeros(rows + 1, np.int32)
    rptr[1:] = np.cumsum(cnt)
    cind = rng.integers(0, nbc, int(rptr[-1])).astype(np.int32)
    val = rng.uniform(-1, 1, (len(cind), bnw, bnl))  # blocks by columns
    x = rng.uniform(-1, 1, max(n, nbc * bnw))
    prod = val * x[cind[:, None] * bnw + np.arange(bnw)][:, :, None]
    ref, mag = np.zeros((rows, bnl)), np.zeros((rows, bnl))
    br = np.repeat(np.arange(rows), cnt)
    np.add.at(ref, br, prod.sum(1))
    np.add.at(mag, br, np.abs(prod).sum(1))
    d = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (val.reshape(-1), cind, rptr, x)]
    y = torch.full((n + 1,), 7.0, dtype=torch.float64, device="cuda")
    L.check("bcsr", L.lib().senk_dev_spmv_bcsr_d(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(),
                                                 y.data_ptr(), n, bnl, bnw, torch.cuda.current_stream().cuda_stream))
    got = y.cpu().numpy()
    assert got[n] == 7.0
    # two sums of at most 8 * bnw products: 2 (k + 1) half-units of the magnitudes each
    assert np.all(np.abs(got[:n] - ref.reshape(-1)) <= 2 * (8 * bnw + 1) * 2.0 ** -53 * mag.reshape(-1) + 0.0)
