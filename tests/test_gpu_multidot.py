"""Column dot products at the edges of k_multidot's work split: every column
count of a chunk and one past it, lengths around a thread's four elements and
the CTAs' slices, against FP64 sums on the host."""
import numpy as np
import pytest

from senk_gb300 import lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nv", [1, 2, 3, 4, 5, 6, 7, 8, 9, 16])
@pytest.mark.parametrize("n", [1, 255, 513, 4099, 311_297, 1_300_001])
def test_multidot_columns(nv, n):
    import ctypes as C

    import torch
    f = L.lib().senk_dev_multidot_d_noalloc
    f.argtypes = [C.c_void_p, C.c_longlong, C.c_int, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p]
    g = torch.Generator(device="cuda").manual_seed(n + nv)
    V = torch.rand((nv, n + 3), dtype=torch.float64, device="cuda", generator=g) - 0.5
    w = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) - 0.5
    out = torch.full((nv,), 9.0, dtype=torch.float64, device="cuda")
    L.check("multidot", f(V.data_ptr(), n + 3, nv, w.data_ptr(), n, out.data_ptr(), None))
    torch.cuda.synchronize()
    prod = (V[:, :n] * w).cpu().numpy()
    want = np.array([float(np.sum(p.astype(np.longdouble))) for p in prod])
    # products are fused; any order of n additions
    assert np.all(np.abs(out.cpu().numpy() - want) <= (n + 1) * 2.0 ** -53 * np.abs(prod).sum(axis=1))
    r = C.c_double()
    L.check("dot", L.lib().senk_dev_dot_d(V.data_ptr(), w.data_ptr(), n, C.byref(r), None))
    assert abs(r.value - want[0]) <= (n + 1) * 2.0 ** -53 * np.abs(prod[0]).sum()
