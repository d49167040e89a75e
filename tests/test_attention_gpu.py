"""Flash-attention kernels against the fp32 PyTorch attention of ops.reference."""
import pytest
import torch

from ferrotorch_b200 import _native
from ferrotorch_b200.ops import functional as F
from ferrotorch_b200.ops import reference as R

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device=DEV) * scale).to(torch.bfloat16)


def _close(got, want, atol, rtol, what):
    err = (got.float() - want.float()).abs()
    tol = atol + rtol * want.float().abs()
    assert not (err > tol).any(), "%s: max err %.4g" % (what, float(err.max()))


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,D,causal", [
    (1, 128, 128, 2, 2, 128, True),
    (2, 256, 256, 4, 2, 128, True),
    (1, 384, 384, 4, 1, 128, False),
    (2, 200, 200, 4, 2, 128, True),     # ragged: tile tails in q and kv
    (1, 100, 333, 2, 1, 128, True),     # query block is the tail of a longer key sequence
    (1, 1024, 1024, 8, 2, 128, True),
    (2, 256, 256, 4, 4, 64, True),
    (1, 130, 190, 2, 2, 64, False),
    (1, 2048, 2048, 4, 2, 128, True),   # many key blocks per CTA: lazy rescale, ring wrap-arounds
    (1, 640, 640, 2, 1, 128, True),     # odd number of query tiles: the last CTA has one tile only
    (2, 513, 513, 4, 2, 128, True),
    (1, 300, 700, 2, 2, 64, True),
    (1, 1024, 1024, 2, 2, 64, False),
])
def test_flash_fwd(B, Sq, Sk, Hq, Hkv, D, causal):
    torch.manual_seed(Sq + Sk + Hq)
    q, k, v = _rand(B, Sq, Hq, D), _rand(B, Sk, Hkv, D), _rand(B, Sk, Hkv, D)
    out, lse = F.flash_attn_fwd(q, k, v, causal)
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    want, lse_w = R.attention(q, k, v, causal)
    _close(out, want, 2e-2, 2e-2, "attention out")
    _close(lse, lse_w, 2e-2, 1e-3, "attention lse")


def test_flash_fwd_large_scores_lazy_rescale():
    # row maxima that keep growing along the keys (by more and by less than the lazy-rescale
    # threshold) exercise both the rescale of O in TMEM and the stale-reference path
    torch.manual_seed(5)
    B, S, H, D = 1, 1024, 2, 128
    q, k, v = _rand(B, S, H, D), _rand(B, S, H, D), _rand(B, S, H, D)
    ramp = torch.linspace(0.2, 3.0, S, device=DEV).view(1, S, 1, 1)
    k = (k.float() * ramp).to(torch.bfloat16)
    out, lse = F.flash_attn_fwd(q, k, v, False)
    want, lse_w = R.attention(q, k, v, False)
    _close(out, want, 2e-2, 2e-2, "attention out (growing maxima)")
    _close(lse, lse_w, 2e-2, 1e-3, "attention lse (growing maxima)")
    assert _native.device_status(0) == 0


def test_flash_fwd_packed_qkv():
    torch.manual_seed(0)
    B, S, Hq, Hkv, D = 2, 256, 8, 2, 128
    qkv = _rand(B, S, Hq + 2 * Hkv, D)
    q, k, v = qkv[:, :, :Hq], qkv[:, :, Hq:Hq + Hkv], qkv[:, :, Hq + Hkv:]
    out, _ = F.flash_attn_fwd(q, k, v, True)
    want, _ = R.attention(q, k, v, True)
    _close(out, want, 2e-2, 2e-2, "packed qkv")
    assert _native.device_status(0) == 0


@pytest.mark.parametrize("B,Sq,Sk,Hq,Hkv,D,causal", [
    (1, 128, 128, 2, 2, 128, True),
    (2, 256, 256, 4, 2, 128, True),
    (1, 320, 320, 4, 1, 128, False),
    (2, 200, 200, 4, 2, 128, True),
    (1, 100, 333, 2, 1, 128, True),
    (1, 1024, 1024, 8, 2, 128, True),
    (2, 256, 256, 4, 4, 64, True),
    (1, 130, 190, 2, 2, 64, False),
    (1, 2048, 2048, 8, 2, 128, True),    # many steps per CTA: ring and double-buffer wrap-arounds, GQA group of 4
    (2, 700, 700, 4, 4, 128, True),
    (1, 448, 448, 2, 1, 128, False),
])
@pytest.mark.parametrize("two_pass", [False, True])
def test_flash_bwd(B, Sq, Sk, Hq, Hkv, D, causal, two_pass):
    from ferrotorch_b200.ops import attention as A
    from ferrotorch_b200.ops.attention import flash_attention

    if two_pass and D != 128:
        pytest.skip("head_dim 64 always runs the two-pass kernels")
    prev = A.deterministic(two_pass)
    try:
        _flash_bwd_case(flash_attention, B, Sq, Sk, Hq, Hkv, D, causal)
    finally:
        A.deterministic(prev)


def _flash_bwd_case(flash_attention, B, Sq, Sk, Hq, Hkv, D, causal):

    torch.manual_seed(Sq * 3 + Sk + Hq)
    q, k, v = (_rand(B, Sq, Hq, D).requires_grad_(), _rand(B, Sk, Hkv, D).requires_grad_(),
               _rand(B, Sk, Hkv, D).requires_grad_())
    do = _rand(B, Sq, Hq, D, scale=0.5)
    out = flash_attention(q, k, v, causal=causal)
    out.backward(do)
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    want, _ = R.attention(qr, kr, vr, causal)
    want.backward(do.float())
    _close(q.grad, qr.grad, 3e-2, 3e-2, "dq")
    _close(k.grad, kr.grad, 3e-2, 3e-2, "dk")
    _close(v.grad, vr.grad, 3e-2, 3e-2, "dv")


def test_flash_bwd_packed_qkv_grad_layout():
    from ferrotorch_b200.ops.attention import flash_attention

    torch.manual_seed(2)
    B, S, Hq, Hkv, D = 1, 256, 8, 2, 128
    qkv = _rand(B, S, Hq + 2 * Hkv, D).requires_grad_()
    q, k, v = qkv[:, :, :Hq], qkv[:, :, Hq:Hq + Hkv], qkv[:, :, Hq + Hkv:]
    do = _rand(B, S, Hq, D, scale=0.5)
    flash_attention(q, k, v, causal=True).backward(do)
    ref_in = qkv.detach().float().requires_grad_()
    qr, kr, vr = ref_in[:, :, :Hq], ref_in[:, :, Hq:Hq + Hkv], ref_in[:, :, Hq + Hkv:]
    R.attention(qr, kr, vr, True)[0].backward(do.float())
    _close(qkv.grad, ref_in.grad, 3e-2, 3e-2, "packed dqkv")


@pytest.mark.parametrize("D,offset", [(128, 0), (128, 4), (64, 0), (64, 4)])
@pytest.mark.parametrize("Sq", [1, 63, 130])
def test_flash_bwd_with_an_output_at_any_place(D, offset, Sq):
    # an output eight bytes into its buffer cannot be read 16 bytes at a time by the row sums of O * dO
    from ferrotorch_b200.ops.attention import attention_block_backward

    torch.manual_seed(D + Sq)
    B, H = 2, 3
    q, k, v, do = _rand(B, Sq, H, D), _rand(B, Sq, H, D), _rand(B, Sq, H, D), _rand(B, Sq, H, D, scale=0.5)
    out, lse = F.flash_attn_fwd(q, k, v, False)
    buf = torch.empty(out.numel() + offset, device=DEV, dtype=out.dtype)
    moved = buf[offset:].view(out.shape)
    moved.copy_(out)
    want = attention_block_backward(q, k, v, out, lse, do, False)
    got = attention_block_backward(q, k, v, moved, lse, do, False)
    # the sums of D products differ in their order only: 2^-20 of them, then gradients rounded to bf16
    for g, w, what in zip(got, want, ("dq", "dk", "dv")):
        _close(g, w, 2.0 ** -8, 2.0 ** -7, what)
    qr, kr, vr = (t.float().requires_grad_() for t in (q, k, v))
    R.attention(qr, kr, vr, False)[0].backward(do.float())
    for g, w, what in zip(got, (qr.grad, kr.grad, vr.grad), ("dq", "dk", "dv")):
        _close(g, w, 3e-2, 3e-2, what)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("B,Sq,H", [(2, 1031, 3), (1, 6145, 1), (3, 257, 8)])
def test_row_sums_keep_their_bits_whatever_the_loads(D, B, Sq, H):
    # wide loads (from 6144 rows on) add in the order of the narrow ones: the two-pass kernels give the same gradients for an output at an
    # odd place, which takes the narrow loads
    from ferrotorch_b200.ops.attention import attention_block_backward, deterministic

    torch.manual_seed(D)
    q, k, v, do = _rand(B, Sq, H, D), _rand(B, Sq, H, D), _rand(B, Sq, H, D), _rand(B, Sq, H, D)
    out, lse = F.flash_attn_fwd(q, k, v, True)
    moved = torch.empty(out.numel() + 4, device=DEV, dtype=out.dtype)[4:].view(out.shape).copy_(out)
    old = deterministic(True)
    try:
        want = attention_block_backward(q, k, v, moved, lse, do, True)
        got = attention_block_backward(q, k, v, out, lse, do, True)
    finally:
        deterministic(old)
    for g, w in zip(got, want):
        assert torch.equal(g, w)


@pytest.mark.parametrize("Sq,Sk,causal", [(1, 128, False), (15, 130, False), (16, 16, True), (17, 200, True), (49, 49, True), (65, 300, False), (128, 129, True),
                                          (193, 193, True)])
@pytest.mark.parametrize("Hq,Hkv", [(1, 1), (6, 2)])
def test_flash_bwd_ragged_parts_of_a_query_tile(Sq, Sk, causal, Hq, Hkv):
    # one to twelve steps through the three stages; dQ is added sixteen queries at a time, the last of them past Sq or cut by it.
    # Gradients lie in the middle of a larger buffer's rows' worth of scratch only if nothing is written past Sq: the next batch would show it
    from ferrotorch_b200.ops.attention import flash_attention

    _flash_bwd_case(flash_attention, 2, Sq, Sk, Hq, Hkv, 128, causal)


@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("B,S,Hq,Hkv,D", [(3, 700, 6, 2, 128), (2, 129, 3, 3, 64), (1, 1153, 5, 1, 128), (5, 64, 2, 1, 64)])
def test_every_block_of_every_head_is_taken_once(B, S, Hq, Hkv, D, causal):
    # the order of the work depends on the mask; numbers of blocks, heads and sequences that do not divide each other
    from ferrotorch_b200.ops.attention import flash_attention

    _flash_bwd_case(flash_attention, B, S, S, Hq, Hkv, D, causal)
    q, k, v = _rand(B, S, Hq, D), _rand(B, S, Hkv, D), _rand(B, S, Hkv, D)
    _close(F.flash_attn_fwd(q, k, v, causal)[0], R.attention(q, k, v, causal)[0], 2e-2, 2e-2, "out")
