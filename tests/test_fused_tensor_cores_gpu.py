"""The fused operator's 128-row kernels with the value products on the tensor cores (csrc/dense_softmax_v.cu): ragged ends of the tiles of 128
rows, 64 keys, 32 columns and 64 value columns, rows with and without TMA, and values that are not finite.  148 (batch, head) pairs
make those kernels the ones that fill the GPU."""
import numpy as np
import pytest
import torch

from conftest import assert_close

pytestmark = pytest.mark.gpu
SHAPES = [(65, 64, 64), (100, 33, 21), (127, 32, 32), (128, 64, 33), (200, 17, 64), (256, 64, 64), (193, 48, 40), (130, 96, 64), (128, 4, 1)]


def _inputs(n, w, wv, seed=60):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(37, n, 4, x, generator=gen, device="cuda") for x in (w, w, wv, wv)]


@pytest.mark.parametrize("mode", ["softmax", "softmax_plus_one", "exp"])
@pytest.mark.parametrize("n,w,wv", SHAPES)
def test_output_and_gradients(n, w, wv, mode):
    import l1attn_fused_cuda
    q, k, v, g = _inputs(n, w, wv)
    m = l1attn_fused_cuda.L1AttnSoftmaxV(mode)
    res = []
    for dt in (torch.float32, torch.float64):
        t = [x.to(dt).requires_grad_(True) for x in (q, k, v)]
        out = m(*t)
        res.append([out, *torch.autograd.grad(out, t, g.to(dt))])
    # pieces hold the operands exactly; what is left are fp32 sums and the rounding of scores of about sqrt(w), which exp() makes relative
    for x, r, name in zip(*res, ("vo", "dq", "dk", "dv")):
        assert_close(x.detach().cpu().numpy(), r.detach().cpu().numpy(), 1e-5, name)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
def test_values_that_are_not_finite(bad):
    """A value that is not finite has no pieces: the CTA computes its rows plainly, and the others are as ever."""
    import l1attn_fused_cuda
    q, k, v, g = _inputs(130, 64, 64)
    m = l1attn_fused_cuda.L1AttnSoftmaxV()
    v[3, 128, 2, 5] = g[5, 70, 1, 63] = bad
    res = []
    for dt in (torch.float32, torch.float64):
        t = [x.to(dt).requires_grad_(True) for x in (q, k, v)]
        out = m(*t)
        res.append([out, *torch.autograd.grad(out, t, g.to(dt))])
    for i, (x, r, name) in enumerate(zip(*res, ("vo", "dq", "dk", "dv"))):
        if i in (0, 3):  # (in dq and dk everything of the pair is NaN)
            assert torch.equal(x.isfinite(), r.isfinite()) and torch.equal(x.isnan(), r.isnan()), name
        fine = x.isfinite() & r.isfinite()
        assert_close(x[fine].detach().cpu().numpy(), r[fine].detach().cpu().numpy(), 1e-5, name)
        assert torch.isfinite(x[7]).all()


def test_wait_that_counts_polls_gives_up_and_is_reported():
    """The wait of these kernels is bounded by its polls: 500 of them on a barrier that nothing completes, then the kernel returns and the
    status reports a timeout, once.  More polls than a hundred thousand are refused."""
    import l1attn_cabi
    lib = l1attn_cabi.lib()
    torch.cuda.synchronize()
    assert lib.l1attn_device_status() == 0
    returned = torch.zeros(2, dtype=torch.int32, device="cuda")
    assert lib.l1attn_test_wait_polls(500, returned.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert returned.tolist() == [1, 500]
    assert lib.l1attn_device_status() == -7 and lib.l1attn_device_status() == 0
    assert lib.l1attn_test_wait_polls(0, returned.data_ptr(), None) == lib.l1attn_test_wait_polls(100001, returned.data_ptr(), None) == -1
