"""The uploads that a call reports: the arrays that it copied to the device, the
matrix, the factors and the vectors, not what kernels made of them there."""
import numpy as np
import pytest

from senk_gb300 import lib as L
from senk_gb300 import problems as P
from senk_gb300 import solver as SV
from test_gpu_kernels import _factors

pytestmark = pytest.mark.gpu


def test_fp64_abmc_solve():
    prev = L.lib().senk_dropin_cache(0)
    try:
        Ar, Lf, Uf, sc, nc, _, _ = _factors(P.block27(8), "abmc", 16)
        b = Ar.matvec(np.ones(Ar.n))
        x = np.zeros(Ar.n)
        r = SV.AbmcIluGmresm(Ar.val, Ar.cind, Ar.rptr, Lf.val, Lf.cind, Lf.rptr, Uf.val, Uf.cind, Uf.rptr, sc, nc, 16,
                             b, x, float(np.linalg.norm(b)), 10, 30, Ar.n, 1e-8)
        csr = sum(12 * len(F.val) + 4 * (Ar.n + 1) for F in (Ar, Lf, Uf))
        # beside the arrays only the groups' descriptors (32 bytes for 32 rows or more)
        assert csr + 16 * Ar.n <= r.h2d_bytes <= csr + 16 * Ar.n + 8 * Ar.n
    finally:
        L.lib().senk_dropin_cache(prev)
