"""NHWC max-pool kernels against torch on the device (first GPU run is opt-in)."""
import os

import pytest
import torch
import torch.nn.functional as tF

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,k,s,p,hw", [(64, 3, 2, 1, (112, 112)), (8, 2, 2, 0, (9, 7)), (72, 3, 1, 1, (13, 11)), (16, 5, 2, 2, (31, 33))])
def test_forward_backward_match_torch(c, k, s, p, hw):
    from ferrotorch_b200.ops import pool as P

    torch.manual_seed(0)
    x = torch.randn(3, c, *hw, device="cuda", dtype=torch.bfloat16).contiguous(memory_format=torch.channels_last).requires_grad_()
    ref = tF.max_pool2d(x, k, s, p)
    gy = torch.randn_like(ref)
    ref.backward(gy)
    gref, x.grad = x.grad, None
    prev = P.use_native_pool(True)
    try:
        assert P.supported(x, k, s, p)
        y = P.max_pool2d(x, k, s, p)
        y.backward(gy)
    finally:
        P.use_native_pool(prev)
    assert torch.equal(y, ref)
    torch.testing.assert_close(x.grad.float(), gref.float(), rtol=2e-2, atol=2e-2)      # sums of up to 4 bf16 terms: order may differ


@pytest.mark.parametrize("n,c,h,w,k,stride,pad", [(5, 24, 33, 17, (3, 3), 2, (1, 1)), (1, 8, 2, 3, (2, 3), 1, (0, 1)), (2, 40, 31, 64, (5, 2), 3, (2, 0))])
def test_index_widths_agree(n, c, h, w, k, stride, pad):
    # 2^31 vectors, from which on the kernels count in 64 bits, would not fit a test: both widths on the same images, forward and backward
    from ferrotorch_b200 import _native
    from ferrotorch_b200.ops import functional as F

    lib = _native.kernels()
    ho, wo = (h + 2 * pad[0] - k[0]) // stride + 1, (w + 2 * pad[1] - k[1]) // stride + 1
    x = torch.randn(n, h, w, c, device="cuda").to(torch.bfloat16)
    gy = torch.randn(n, ho, wo, c, device="cuda").to(torch.bfloat16)
    results = []
    for wide in (0, 1):
        y, arg, gx = torch.empty_like(gy), torch.full((n, ho, wo, c), 255, device="cuda", dtype=torch.uint8), torch.empty_like(x)
        _native.check(lib.ft_maxpool2d_fwd_nhwc(x.data_ptr(), y.data_ptr(), arg.data_ptr(), n, h, w, c, *k, stride, *pad, wide, 0, F._stream()), "fwd")
        _native.check(lib.ft_maxpool2d_bwd_nhwc(gy.data_ptr(), arg.data_ptr(), gx.data_ptr(), n, h, w, c, *k, stride, *pad, wide, 0, F._stream()), "bwd")
        results.append((y, arg, gx))
    for a, b in zip(*results):
        assert torch.equal(a, b)
    assert torch.equal(results[0][0].permute(0, 3, 1, 2).float(), tF.max_pool2d(x.permute(0, 3, 1, 2).float(), k, stride, pad))
