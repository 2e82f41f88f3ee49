"""X^T dZ at the edges of its node chunks, with results that are and are not
16-byte aligned; the gradient at node counts that leave ragged passes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from senk_gb300 import lib as L


@pytest.mark.parametrize("n", [1, 63, 64, 65, 129, 20000])
@pytest.mark.parametrize("off", [0, 1, 4])
def test_gemm_tn_result_alignment(n, off):
    import torch
    g = torch.Generator().manual_seed(n)
    X = (torch.rand(n, 128, generator=g) - .5).to(torch.bfloat16).cuda()
    dZ = (torch.rand(n, 64, generator=g) - .5).to(torch.bfloat16).cuda()
    out = torch.full((128 * 64 + 8,), 7.0, device="cuda")
    L.check("gemm_tn", L.lib().senk_dev_gemm_tn_bf16(X.data_ptr(), dZ.data_ptr(), out.data_ptr() + 4 * off, n, None))
    torch.cuda.synchronize()
    ref, mag = X.double().T @ dZ.double(), X.double().abs().T @ dZ.double().abs()
    got = out[off:off + 128 * 64].double().reshape(128, 64)
    # products are exact in FP32; n additions, each within an FP32 unit of the magnitudes' sum
    assert bool(((got - ref).abs() <= n * 2.0 ** -23 * mag).all())
    assert out[:off].eq(7.0).all() and out[off + 128 * 64:].eq(7.0).all()


@pytest.mark.parametrize("n", [9, 11, 13])  # 729, 1331, 2197 nodes: remainders of the passes of 4, 16 and 128 nodes
def test_gradient_at_ragged_node_counts(n):
    import torch
    import oracle
    from oracle import mpnn as M
    from senk_gb300 import learned as LN
    mb = LN.family_member(n, 11, 1)
    sysm = LN.System(mb.A, mb.L, mb.U, L.PC_ILU_ABMC, mb.cptr, mb.cnum, 1, m_max=0)
    params = M.init_params(3)
    rng = np.random.default_rng(n)
    params[M.OFF_WOUT:M.OFF_BOUT] = rng.normal(0, 0.1, M.HID)
    net = LN.Net(params)
    try:
        net.bind(sysm)
        r, e = rng.standard_normal(mb.A.n), rng.standard_normal(mb.A.n) * 0.05
        rd, ed = torch.from_numpy(r).cuda(), torch.from_numpy(e).cuda()
        loss, grad = net.loss_grad(sysm, rd.data_ptr(), ed.data_ptr())
        ilu = oracle.port().ilu_apply(mb.L, mb.U, r, mb.cptr, mb.cnum, 1)
        want, gw = M.loss_grad(params, M.Graph(mb.A.val, mb.A.cind, mb.A.rptr), r, ilu, e, rounding=True, mode=1)
        # every activation passes BF16 operands, which round either way where the
        # FP32 sums before them differ in the last bit: half a BF16 unit (2e-3) of a
        # term, of which few of the hundred and more terms of a sum flip
        assert abs(loss - want) <= 1e-3 * want
        for lo, hi in ((0, M.OFF_BIN), (M.OFF_BIN, M.OFF_LAYER), (M.OFF_LAYER, M.OFF_WOUT), (M.OFF_WOUT, M.NPARAMS)):
            assert np.linalg.norm(grad[lo:hi] - gw[lo:hi]) <= 1e-3 * np.linalg.norm(gw[lo:hi])
    finally:
        net.close()
        sysm.close()
