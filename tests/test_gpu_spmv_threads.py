"""CSR products of matrices with different row lengths from several host threads:
their kernels need different amounts of shared memory."""
import threading

import numpy as np
import pytest

from senk_gb300 import lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_row_lengths_in_threads(dtype):
    """The most shared memory that a CTA takes (rows of 15 or 32 entries in FP64, of 23 in FP32) beside less."""
    import torch
    n, rounds, bad = 3000, 3000, []
    f = L.lib().senk_dev_spmv_csr_s if dtype == np.float32 else L.lib().senk_dev_spmv_csr_d

    def work(per, stream):
        rng = np.random.default_rng(per)
        val = torch.from_numpy(rng.integers(-4, 5, n * per).astype(dtype)).cuda()      # exact sums
        col = rng.integers(0, n, n * per).astype(np.int32)
        x = rng.integers(-4, 5, n).astype(dtype)
        want = torch.from_numpy((val.cpu().numpy() * x[col]).reshape(n, per).sum(1)).cuda()
        c, r, xd = (torch.from_numpy(a).cuda() for a in (col, np.arange(n + 1, dtype=np.int32) * np.int32(per), x))
        y = torch.empty_like(want)
        torch.cuda.synchronize()
        for _ in range(rounds):
            if f(val.data_ptr(), c.data_ptr(), r.data_ptr(), xd.data_ptr(), y.data_ptr(), n, n * per, stream.cuda_stream):
                bad.append((per, L.lib().senk_last_error().decode()))
                return
        stream.synchronize()
        if not torch.equal(y, want):
            bad.append((per, "wrong rows"))

    ts = [threading.Thread(target=work, args=(per, torch.cuda.Stream())) for per in (14, 15, 21, 23, 32, 40)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
