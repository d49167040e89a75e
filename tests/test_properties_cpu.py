"""Property-based checks (hypothesis) of host-side code: invariants that must hold for every input
of a family, not only for hand-picked cases."""
import numpy as np
import pytest
import torch

hypothesis = pytest.importorskip("hypothesis")
from hypothesis import example, given, settings  # noqa: E402
from hypothesis import strategies as st  # noqa: E402

FAST = settings(max_examples=40, deadline=None)


@FAST
@given(st.integers(1, 400), st.floats(0.05, 0.95), st.integers(0, 2 ** 31 - 1))
def test_nms_keeps_an_independent_dominating_set(n, thr, seed):
    # (1) kept boxes do not overlap each other above the threshold; (2) every dropped box overlaps a kept
    # box of a higher score above it; (3) native sweep and torch formulation agree
    from ferrotorch_b200.ops import det_ops as D

    g = torch.Generator().manual_seed(seed)
    xy, wh = torch.rand(n, 2, generator=g) * 60, torch.rand(n, 2, generator=g) * 40 + 0.5
    boxes, scores = torch.cat([xy, xy + wh], 1), torch.rand(n, generator=g)
    keep = D.nms(boxes, scores, thr)
    assert torch.equal(keep, D.nms_torch(boxes, scores, thr))
    assert (scores[keep][:-1] >= scores[keep][1:]).all()
    iou = D.box_iou(boxes, boxes)
    kk = iou[keep][:, keep].clone()
    kk.fill_diagonal_(0)
    assert (kk <= thr).all()
    dropped = torch.ones(n, dtype=torch.bool)
    dropped[keep] = False
    for i in torch.where(dropped)[0].tolist():
        better = keep[scores[keep] >= scores[i]]
        assert (iou[i, better] > thr).any()


@FAST
@example(1, 7, 16454)               # the top code beside a scale that lost 3.7e-4 of itself to fp16
@given(st.integers(1, 6), st.integers(1, 8), st.integers(0, 2 ** 31 - 1))
def test_q4_0_round_trip_error_and_fixed_point(rows, blocks, seed):
    # |x - dq(q(x))| <= |d| / 2 except at the clamped top code (<= |d|); quantising the result again changes nothing
    from ferrotorch_b200.ops.quant import dequant_q4_0_planes, quantize_q4_0_planes

    g = torch.Generator().manual_seed(seed)
    x = torch.randn(rows, 32 * blocks, generator=g) * torch.rand(1, generator=g) * 10
    nib, sc = quantize_q4_0_planes(x)
    y = dequant_q4_0_planes(nib, sc)
    d = sc.float().abs().repeat_interleave(32, dim=1)
    # |x| <= 8 |d| before d is rounded to fp16 (by 2^-11 of it at most): at the top code |x| - 7 |d| <= |d| (1 + 8 * 2^-11)
    assert ((x - y).abs() <= d * (1 + 2.0 ** -8) + 1e-6).all()
    inner = (x - y).abs() <= d * 0.5 * 1.01 + 1e-3 * d + 1e-6          # fp16 scale rounding leaves a little slack
    assert inner.float().mean() > 0.9
    nib2, sc2 = quantize_q4_0_planes(y)
    y2 = dequant_q4_0_planes(nib2, sc2)
    nib3, sc3 = quantize_q4_0_planes(y2)
    assert torch.equal(nib2, nib3) and torch.equal(sc2, sc3)


@FAST
@given(st.integers(0, 2 ** 40), st.integers(0, 2 ** 63 - 1), st.lists(st.integers(0, 37), min_size=1, max_size=6))
def test_philox_stream_is_continuous_over_arbitrary_splits(counter, seed, cuts):
    # drawing n words at once equals drawing them in pieces: the generator's (counter, offset) state carries over
    from ferrotorch_b200.utils.philox import PhiloxGenerator, PhiloxState

    total = sum(cuts)
    a = PhiloxGenerator(seed)
    a.set_state(PhiloxState.from_parts(counter, seed, 0))
    whole = a.words(total)
    b = PhiloxGenerator(seed)
    b.set_state(PhiloxState.from_parts(counter, seed, 0))
    pieces = np.concatenate([b.words(c) for c in cuts]) if total else np.zeros(0, dtype=whole.dtype)
    assert np.array_equal(whole, pieces)
    assert a.get_state() == b.get_state()


@FAST
@given(st.integers(2, 5), st.integers(1, 3), st.integers(0, 2 ** 31 - 1), st.booleans())
def test_attention_over_key_blocks_merges_exactly(parts, heads_kv, seed, causal_first):
    # attention over the whole key set = merge of attention over any partition of the keys
    from ferrotorch_b200.ops import reference as R
    from ferrotorch_b200.parallel.context_parallel import merge_attention

    g = torch.Generator().manual_seed(seed)
    S, D = 4 * parts + 3, 8
    q = torch.randn(1, 6, 2 * heads_kv, D, generator=g)
    k, v = torch.randn(1, S, heads_kv, D, generator=g), torch.randn(1, S, heads_kv, D, generator=g)
    want, want_lse = R.attention(q, k, v, causal=False)
    cuts = sorted(set(torch.randint(1, S, (parts - 1,), generator=g).tolist()))
    bounds = [0] + cuts + [S]
    out = lse = None
    for lo, hi in zip(bounds[:-1], bounds[1:]):
        o, l = R.attention(q, k[:, lo:hi], v[:, lo:hi], causal=False)
        out, lse = (o, l) if out is None else merge_attention(out, lse, o, l)
    assert torch.allclose(out, want, atol=1e-5) and torch.allclose(lse, want_lse, atol=1e-5)


@FAST
@given(st.lists(st.tuples(st.sampled_from(["float32", "float16", "bfloat16", "int64", "int32", "uint8", "bool"]),
                          st.lists(st.integers(0, 5), min_size=0, max_size=3)), min_size=1, max_size=5),
       st.integers(0, 2 ** 31 - 1))
def test_safetensors_round_trip_of_any_dtype_and_shape(specs, seed):
    import os
    import tempfile

    from ferrotorch_b200.serialize.state import load_safetensors, save_safetensors

    g = torch.Generator().manual_seed(seed)
    state = {}
    for i, (dt, shape) in enumerate(specs):
        dtype = getattr(torch, dt)
        if dtype.is_floating_point:
            t = torch.randn(shape, generator=g).to(dtype)
        elif dtype == torch.bool:
            t = torch.rand(shape, generator=g) > 0.5
        else:
            t = torch.randint(0, 100, shape, generator=g).to(dtype)
        state["t%d.weight" % i] = t
    with tempfile.TemporaryDirectory() as d:
        path = os.path.join(d, "x.safetensors")
        save_safetensors(state, path, metadata={"format": "pt"})
        back = load_safetensors(path)
        assert set(back) == set(state)
        for k, t in state.items():
            assert back[k].dtype == t.dtype and back[k].shape == t.shape and torch.equal(back[k], t)


@FAST
@given(st.integers(1, 4), st.integers(2, 40), st.integers(2, 40), st.integers(1, 9), st.integers(0, 2 ** 31 - 1))
def test_roi_align_of_a_constant_map_is_that_constant_inside_the_map(c, h, w, k, seed):
    # bilinear samples of a constant are the constant; boxes that stay inside the map never touch the zero border
    from ferrotorch_b200.ops import det_ops as D

    g = torch.Generator().manual_seed(seed)
    val = torch.rand(c, generator=g) + 0.5
    feat = val.view(1, c, 1, 1).expand(1, c, h, w).contiguous()
    x1, y1 = torch.rand(k, generator=g) * (w - 1) * 0.5, torch.rand(k, generator=g) * (h - 1) * 0.5
    x2, y2 = x1 + torch.rand(k, generator=g) * (w - 1) * 0.5, y1 + torch.rand(k, generator=g) * (h - 1) * 0.5
    rois = torch.stack([torch.zeros(k), x1, y1, x2, y2], 1)
    for fn in (D.roi_align, D.roi_align_torch):
        out = fn(feat, rois, 3, 1.0, 2, True)
        assert torch.allclose(out, val.view(1, c, 1, 1).expand_as(out), atol=1e-5)


def test_gated_products_take_the_faster_kernel_of_what_was_measured():
    from ferrotorch_b200.ops import functional as F

    # rows, features, contraction, us as two kernels, us as one (weights from HBM, launches back to back)
    for rows, features, _k, two, one in [
            (129, 512, 2048, 15.3, 22.0), (214, 4096, 2048, 20.1, 23.5), (256, 4736, 2048, 21.3, 23.7), (129, 5504, 2048, 30.1, 23.9),
            (214, 8192, 2048, 31.3, 26.1), (257, 3584, 3072, 39.2, 28.8), (512, 4096, 2048, 31.5, 24.5), (257, 4736, 2048, 22.2, 24.4),
            (257, 5504, 2048, 31.8, 34.5), (320, 8192, 3072, 45.5, 46.7), (257, 11008, 4096, 73.9, 76.2), (1024, 4096, 2048, 34.9, 34.6),
            (640, 8192, 3072, 64.9, 62.8), (1024, 14336, 4096, 183.1, 171.2), (1500, 5504, 2048, 61.6, 56.1)]:
        if abs(two - one) > 0.02 * one:
            assert F._gates_in_gemm(rows, 2 * features) == (one < two), (rows, features)


def test_divided_sums_are_taken_where_they_were_measured_to_be_faster():
    from ferrotorch_b200.ops import functional as F

    # rows, columns, contraction, us of the CTA pairs, us of the clusters
    for m, n, k, pairs, clusters in [
            (129, 4096, 2048, 15.4, 13.5), (224, 4096, 2048, 15.4, 16.5), (256, 3072, 3072, 20.0, 18.4), (129, 6144, 4096, 26.1, 24.0),
            (192, 6144, 4096, 26.1, 26.6), (224, 6144, 4096, 26.6, 30.6), (256, 6144, 6144, 36.5, 39.4), (256, 2048, 2048, 15.1, 15.5),
            (288, 4096, 4096, 25.7, 26.3), (512, 4096, 4096, 26.2, 35.0), (400, 4096, 14336, 77.4, 56.0), (400, 6144, 4096, 45.1, 36.7),
            (400, 2048, 4096, 24.6, 19.0), (524, 4096, 4096, 44.5, 31.8), (640, 2048, 4096, 24.7, 29.1), (640, 2048, 8192, 43.8, 37.9),
            (640, 1024, 4096, 24.4, 18.3), (640, 6144, 4096, 46.4, 39.8), (192, 2048, 1024, 8.5, 11.4), (400, 3072, 2048, 15.6, 23.0),
            (640, 16384, 2048, 39.8, 76.2), (768, 3072, 2048, 16.1, 20.4)]:
        assert F._streams(m, n, k) == (clusters < pairs), (m, n, k)
