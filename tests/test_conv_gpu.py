"""Convolution on this library's GEMM kernels against torch's conv2d in fp32: the three native
paths (1 x 1 as GEMM, shifted-row k x k with stride 1 / 2, im2col for the stem), forward and all
gradients; the older gather-based kernel; a ResNet-50 training step with no library convolution."""
import pytest
import torch
import torch.nn.functional as tF

pytestmark = pytest.mark.gpu

CL = torch.channels_last


def _case(cin, cout, k, n, hw, seed=0):
    torch.manual_seed(seed)
    x = torch.randn(n, cin, *hw, device="cuda", dtype=torch.bfloat16).contiguous(memory_format=CL)
    w = (torch.randn(cout, cin, k, k, device="cuda") / (cin * k * k) ** 0.5).to(torch.bfloat16)
    b = torch.randn(cout, device="cuda", dtype=torch.bfloat16)
    return x, w, b


def _rel(got, want):
    return float((got.float() - want).abs().max() / (want.abs().max() + 1e-6))


@pytest.mark.parametrize("cin,cout,k,stride,pad,dil,n,hw,path", [
    (64, 64, 1, 1, 0, 1, 4, (56, 56), "pointwise"), (512, 2048, 1, 1, 0, 1, 2, (7, 7), "pointwise"),
    (256, 512, 1, 2, 0, 1, 3, (28, 28), "pointwise"),
    (64, 64, 3, 1, 1, 1, 4, (56, 56), "shift"), (128, 128, 3, 2, 1, 1, 2, (56, 56), "shift"),
    (256, 320, 3, 1, 2, 2, 1, (15, 17), "shift"), (512, 512, 3, 1, 1, 1, 5, (7, 7), "shift"),
    (64, 192, 5, 2, 2, 1, 2, (13, 11), "shift"), (64, 128, 3, 1, 0, 1, 3, (9, 5), "shift"),
    (3, 64, 7, 2, 3, 1, 2, (64, 64), "im2col"), (16, 24, 3, 1, 1, 1, 2, (10, 9), "im2col"),
])
def test_forward_and_gradients_match_torch(cin, cout, k, stride, pad, dil, n, hw, path):
    from ferrotorch_b200 import _native
    from ferrotorch_b200.ops import conv as C

    x, w, b = _case(cin, cout, k, n, hw)
    assert C.native_conv_enabled() and C.native_path(x, w, stride, pad, dil) == path
    xr, wr, br = x.float().requires_grad_(), w.float().requires_grad_(), b.float().requires_grad_()
    ref = tF.conv2d(xr, wr, br, stride, pad, dil)
    gy = torch.randn_like(ref)
    ref.backward(gy)
    xn, wn, bn = x.clone().requires_grad_(), w.clone().requires_grad_(), b.clone().requires_grad_()
    before = _native.launch_count()
    y = C.conv2d(xn, wn, bn, stride, pad, dil)
    y.backward(gy.to(torch.bfloat16))
    torch.cuda.synchronize()
    assert _native.launch_count() > before and _native.device_status(0) == 0
    assert y.is_contiguous(memory_format=CL) and y.dtype == torch.bfloat16
    assert _rel(y, ref.detach()) < 2e-2
    assert _rel(xn.grad, xr.grad) < 2e-2
    assert _rel(wn.grad, wr.grad) < 2e-2
    assert _rel(bn.grad, br.grad) < 2e-2


def test_fused_epilogue_and_fp32_weights():
    from ferrotorch_b200.ops import conv as C

    x, w, b = _case(128, 128, 3, 2, (14, 14), seed=3)
    ref = tF.conv2d(x.float(), w.float(), b.float(), 1, 1)
    res = torch.randn_like(ref).to(torch.bfloat16).contiguous(memory_format=CL)
    z = C.conv2d(x, w.float(), b.float(), 1, 1, residual=res, relu=True)   # fp32 parameters (autocast-style)
    assert _rel(z, torch.relu(ref + res.float())) < 2e-2
    r = C.conv2d(x, w, None, 1, 1, relu=True)
    assert _rel(r, torch.relu(tF.conv2d(x.float(), w.float(), None, 1, 1))) < 2e-2


def test_relu_backward():
    from ferrotorch_b200.ops import conv as C

    x, w, _ = _case(64, 128, 3, 2, (14, 14), seed=1)
    xr, wr = x.float().requires_grad_(), w.float().requires_grad_()
    torch.relu(tF.conv2d(xr, wr, None, 1, 1)).square().sum().backward()
    xn, wn = x.clone().requires_grad_(), w.clone().requires_grad_()
    C.conv2d(xn, wn, None, 1, 1, relu=True).float().square().sum().backward()
    assert _rel(xn.grad, xr.grad) < 5e-2 and _rel(wn.grad, wr.grad) < 5e-2


@pytest.mark.parametrize("cin,cout,k,stride,pad,dil,n,hw", [
    (64, 64, 3, 1, 1, 1, 4, (56, 56)), (128, 128, 3, 2, 1, 1, 2, (28, 28)), (256, 72, 3, 1, 2, 2, 1, (15, 17)),
])
def test_gather_kernel_forward(cin, cout, k, stride, pad, dil, n, hw):
    from ferrotorch_b200.ops import conv as C

    x, w, b = _case(cin, cout, k, n, hw)
    ref = tF.conv2d(x.float(), w.float(), b.float(), stride, pad, dil)
    y = C.conv2d_gather(x, w, b, stride, pad, dil)
    res = torch.randn_like(y)
    z = C.conv2d_gather(x, w, b, stride, pad, dil, residual=res, relu=True)
    torch.testing.assert_close(y.float(), ref, rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(z.float(), torch.relu(ref + res.float()), rtol=2e-2, atol=3e-2)


def _loss_and_grads(m, x, fn):
    m.zero_grad(set_to_none=True)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = fn(m(x))
    loss.backward()
    return float(loss), {n: p.grad.detach().float().clone() for n, p in m.named_parameters()}


def _cos(a, b):
    a, b = a.flatten(), b.flatten()
    return float(torch.dot(a, b) / (a.norm() * b.norm() + 1e-12))


def test_bottleneck_block_gradients_match_the_library_path():
    # one strided bottleneck (1x1, 3x3 stride 2, 1x1, projection shortcut; batch norm in training
    # mode) with fp32 parameters under autocast: every gradient against the cuDNN path
    from ferrotorch_b200.models import resnet as R
    from ferrotorch_b200.ops import conv as C

    torch.manual_seed(4)
    down = torch.nn.Sequential(torch.nn.Conv2d(256, 512, 1, 2, bias=False), torch.nn.BatchNorm2d(512))
    blk = R.Bottleneck(256, 128, 2, down).cuda().to(memory_format=CL)
    C.convert_convs(blk)
    x = torch.randn(32, 256, 28, 28, device="cuda", dtype=torch.bfloat16).contiguous(memory_format=CL)
    tgt = torch.randn(32, 512, 14, 14, device="cuda")
    fn = lambda y: (y.float() - tgt).square().mean()  # noqa: E731
    l_native, g_native = _loss_and_grads(blk, x, fn)
    prev = C.use_native_conv(False)
    try:
        l_lib, g_lib = _loss_and_grads(blk, x, fn)
    finally:
        C.use_native_conv(prev)
    assert abs(l_native - l_lib) < 2e-2 * abs(l_lib)
    for name in g_lib:
        assert _cos(g_native[name], g_lib[name]) > 0.99, "%s: cosine %.4f" % (name, _cos(g_native[name], g_lib[name]))


def test_resnet50_training_step_runs_no_library_convolution():
    from ferrotorch_b200.models import resnet as R
    from ferrotorch_b200.ops import conv as C

    torch.manual_seed(2)
    m = R.resnet50(num_classes=10).cuda().to(memory_format=CL)
    x = torch.randn(16, 3, 96, 96, device="cuda", dtype=torch.bfloat16).contiguous(memory_format=CL)
    t = torch.randint(0, 10, (16,), device="cuda")
    for k in C.stats:
        C.stats[k] = 0
    fn = lambda logits: tF.cross_entropy(logits.float(), t)  # noqa: E731
    l_native, g_native = _loss_and_grads(m, x, fn)
    assert C.stats["library"] == 0 and C.stats["shift"] == 16 and C.stats["pointwise"] == 36 and C.stats["im2col"] == 1
    assert all(torch.isfinite(g).all() for g in g_native.values())
    prev = C.use_native_conv(False)
    try:
        l_lib, g_lib = _loss_and_grads(m, x, fn)
    finally:
        C.use_native_conv(prev)
    assert abs(l_native - l_lib) < 0.05 * max(1.0, abs(l_lib))
    # 53 layers of bf16 activations and small-batch batch norm amplify rounding differences on the
    # way back, so only the classifier's gradient is compared here; the block test above and the
    # per-layer tests compare every gradient of every path
    assert _cos(g_native["fc.weight"], g_lib["fc.weight"]) > 0.9


def test_folded_resnet_matches_eval_model():
    from ferrotorch_b200.models import resnet as R

    torch.manual_seed(2)
    m = R.resnet50(num_classes=10).cuda().bfloat16().to(memory_format=CL).eval()
    x = torch.randn(4, 3, 64, 64, device="cuda", dtype=torch.bfloat16).contiguous(memory_format=CL)
    fused = R.fuse_for_inference(m).cuda()
    with torch.no_grad():
        ref = m(x).float()
        out = fused(x).float()
    assert torch.isfinite(out).all()
    torch.testing.assert_close(out, ref, rtol=0.1, atol=0.1 * float(ref.abs().max()))


@pytest.mark.parametrize("cin,cout,k,stride,pad,dil,n,hw", [
    (64, 64, 3, 1, (1, 1), 1, 1, (1, 1)), (64, 128, 3, 2, (1, 1), 1, 1, (5, 7)), (128, 64, 1, 2, (0, 0), 1, 2, (9, 8)),
    (64, 64, 3, 2, (1, 1), 1, 3, (97, 97)), (192, 320, 3, 1, (1, 1), 1, 2, (16, 8)), (64, 256, 2, 2, (0, 0), 1, 2, (8, 10)),
    (64, 64, (5, 3), 1, (2, 0), 1, 2, (11, 6)), (64, 64, 3, 1, (4, 4), 4, 1, (20, 20)), (64, 64, 3, 2, (0, 0), 1, 2, (8, 8)),
    (64, 64, 3, 1, (130, 130), 130, 1, (5, 4)), (64, 64, 3, 2, (130, 2), 1, 1, (7, 6)),     # outside a tensor map's range: the padded copy
])
@pytest.mark.parametrize("channels_last_filter", [False, True])
def test_walks_against_torch(cin, cout, k, stride, pad, dil, n, hw, channels_last_filter):
    # edges of the 256-pixel tiles and of the images, odd sizes, pixels that no tap reaches; filters in either memory format
    from ferrotorch_b200 import _native
    from ferrotorch_b200.ops import conv as C

    torch.manual_seed(cin + cout + hw[0])
    kh, kw = (k, k) if isinstance(k, int) else k
    x = torch.randn(n, cin, *hw, device="cuda", dtype=torch.bfloat16).contiguous(memory_format=CL)
    w = (torch.randn(cout, cin, kh, kw, device="cuda") / (cin * kh * kw) ** 0.5).to(torch.bfloat16)
    w = w.contiguous(memory_format=CL) if channels_last_filter else w
    xr, wr = x.double().cpu().requires_grad_(), w.double().cpu().requires_grad_()
    ref = tF.conv2d(xr, wr, None, stride, pad, dil)
    gy = torch.randn(ref.shape, device="cuda", dtype=torch.bfloat16)
    ref.backward(gy.double().cpu())
    xn, wn = x.clone(memory_format=torch.preserve_format).requires_grad_(), w.clone(memory_format=torch.preserve_format).requires_grad_()
    y = C.conv2d(xn, wn, None, stride, pad, dil)
    y.backward(gy)
    # one rounding to bf16 (2^-9 relative) of fp32 sums; the filter gradient sums up to n * Ho * Wo products
    for got, want in ((y, ref), (xn.grad, xr.grad), (wn.grad, wr.grad)):
        want = want.detach().cuda()
        assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -14 * want.abs().max()).all())
    assert y.is_contiguous(memory_format=CL) and wn.grad.stride() == wn.stride() and _native.device_status(0) == 0
    # a trainer's gradient arena, bf16 and fp32: the gradient is added to what is there
    for dt in (torch.bfloat16, torch.float32):
        wa = w.clone(memory_format=torch.contiguous_format).requires_grad_()
        wa.main_grad = torch.ones(w.shape, device="cuda", dtype=dt)
        C.conv2d(x, wa, None, stride, pad, dil).backward(gy)
        want = wr.grad.cuda() + 1
        assert wa.grad is None and bool(((wa.main_grad.double() - want).abs() <= 2.0 ** -7 * want.abs() + 2.0 ** -7).all())


@pytest.mark.parametrize("n,hw,k,stride,pad,dil", [(2, (17, 35), (7, 7), 2, (3, 3), 1), (1, (9, 16), (3, 2), 1, (0, 1), 2), (3, (40, 33), (9, 9), 3, (4, 4), 1),
                                                   (1, (5, 5), (5, 5), 1, (0, 0), 1)])
def test_patch_rows_of_four_channels(n, hw, k, stride, pad, dil):
    # runs of sixteen pixels that end with a line, rows of up to 41 vectors, taps and columns behind the filter's
    from ferrotorch_b200.ops import conv as C

    torch.manual_seed(hw[0])
    x = torch.randn(n, 4, *hw, device="cuda", dtype=torch.bfloat16)
    ho, wo = (C.out_size(hw[i], k[i], stride, pad[i], dil) for i in range(2))
    kpad = (k[0] * k[1] * 4 + 15) // 8 * 8
    got = C._im2col(x.contiguous(memory_format=CL).permute(0, 2, 3, 1).contiguous().permute(0, 3, 1, 2), *k, stride, pad, dil, ho, wo, kpad)
    want = tF.unfold(x.float(), k, dil, pad, stride).view(n, 4, k[0] * k[1], ho * wo).permute(0, 3, 2, 1).reshape(n * ho * wo, -1)
    assert torch.equal(got[:, :want.shape[1]].float(), want) and not bool(got[:, want.shape[1]:].any())


@pytest.mark.parametrize("k,stride,pad,relu", [(3, 1, 1, False), (3, 2, 1, True), (2, 1, 0, False)])
def test_the_input_may_change_in_place_before_the_backward_pass(k, stride, pad, relu):
    from ferrotorch_b200.ops import conv as C

    x, w, b = _case(64, 64, k, 2, (9, 10), seed=k)
    grads = []
    for change in (False, True):
        wn, h = w.clone().requires_grad_(), x.clone(memory_format=torch.preserve_format)
        leaf = torch.zeros((), device="cuda", dtype=torch.bfloat16, requires_grad=True)
        h = h + leaf                                    # an activation that records gradients
        y = C.conv2d(h, wn, b, stride, pad, relu=relu)
        if change:
            h.mul_(-3).add_(1)
        y.float().pow(2).sum().backward()
        grads.append((y.detach(), wn.grad, leaf.grad))
    for got, want in zip(grads[1], grads[0]):
        assert torch.equal(got, want)
