"""Paged KV cache kernels and the inference engine."""
import os
import subprocess
import sys

import pytest
import torch

from ferrotorch_b200 import _native
from ferrotorch_b200.nn.paged import OutOfPages, PagedAttentionManager, PagedKVCache
from ferrotorch_b200.ops import reference as R

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
@pytest.mark.parametrize("D,Hq,Hkv,splits", [(128, 8, 2, 1), (128, 8, 2, 3), (64, 4, 4, 2), (128, 4, 1, 0)])
def test_paged_decode_matches_reference(D, Hq, Hkv, splits):
    torch.manual_seed(D + Hq + splits)
    B, bs = 5, 16
    lens = [1, 17, 64, 100, 333]
    cache = PagedKVCache(1, Hkv, D, num_blocks=64, max_seqs=B, max_seq_len=512, block_size=bs)
    mgr = PagedAttentionManager(cache)
    ks, vs = [], []
    for b, n in enumerate(lens):
        assert mgr.add_sequence(n) == b
        k = torch.randn(n, Hkv, D, device="cuda").to(torch.bfloat16)
        v = torch.randn(n, Hkv, D, device="cuda").to(torch.bfloat16)
        ks.append(k), vs.append(v)
        pos = torch.arange(n, device="cuda", dtype=torch.int32)
        sid = torch.full((n,), b, device="cuda", dtype=torch.int32)
        cache.append(0, k, v, pos, sid)
    q = torch.randn(B, Hq, D, device="cuda").to(torch.bfloat16)
    out = cache.decode(0, q, torch.tensor(lens, device="cuda", dtype=torch.int32), n_splits=splits)
    torch.cuda.synchronize()
    for b, n in enumerate(lens):
        gk, gv = cache.gather(0, b, n)
        assert torch.equal(gk, ks[b]) and torch.equal(gv, vs[b])
        want, _ = R.attention(q[b][None, None], ks[b][None], vs[b][None], causal=False)
        err = (out[b].float() - want[0, 0].float()).abs().max().item()
        assert err < 2e-2, "seq %d len %d err %g" % (b, n, err)


@pytest.mark.gpu
@pytest.mark.parametrize("Hq,Hkv,splits,bs", [(8, 8, 2, 16), (8, 4, 1, 32), (16, 2, 4, 16), (32, 8, 0, 8), (8, 2, 2, 128)])
def test_paged_decode_tensor_core_kernel_long_contexts(Hq, Hkv, splits, bs):
    # head_dim 128 with a page size dividing 128 takes the tcgen05 kernel: group sizes 1 / 2 / 4 / 8,
    # contexts long enough to wrap its three-stage ring several times, growing score maxima
    # (lazy rescale of the accumulator), tails that end inside a page and inside a tile
    torch.manual_seed(Hq + Hkv + splits + bs)
    D = 128
    lens = [1, 127, 129, 700, 1531]
    B = len(lens)
    cache = PagedKVCache(1, Hkv, D, num_blocks=sum((n + bs - 1) // bs for n in lens) + 4, max_seqs=B,
                         max_seq_len=2048, block_size=bs)
    mgr = PagedAttentionManager(cache)
    ks, vs = [], []
    for b, n in enumerate(lens):
        assert mgr.add_sequence(n) == b
        ramp = torch.linspace(0.3, 2.5, n, device="cuda").view(n, 1, 1)
        k = (torch.randn(n, Hkv, D, device="cuda") * ramp).to(torch.bfloat16)
        v = torch.randn(n, Hkv, D, device="cuda").to(torch.bfloat16)
        ks.append(k), vs.append(v)
        cache.append(0, k, v, torch.arange(n, device="cuda", dtype=torch.int32),
                     torch.full((n,), b, device="cuda", dtype=torch.int32))
    q = torch.randn(B, Hq, D, device="cuda").to(torch.bfloat16)
    out = cache.decode(0, q, torch.tensor(lens, device="cuda", dtype=torch.int32), n_splits=splits)
    torch.cuda.synchronize()
    assert _native.device_status(0) == 0
    for b, n in enumerate(lens):
        want, _ = R.attention(q[b][None, None], ks[b][None], vs[b][None], causal=False)
        err = (out[b].float() - want[0, 0].float()).abs().max().item()
        assert err < 3e-2, "seq %d len %d err %g" % (b, n, err)


def test_page_pool_bookkeeping():
    cache = PagedKVCache(1, 1, 8, num_blocks=4, max_seqs=2, max_seq_len=64, block_size=16, device="cpu",
                         dtype=torch.float32)
    mgr = PagedAttentionManager(cache)
    a = mgr.add_sequence(20)            # 2 pages
    assert mgr.free_pages == 2
    b = mgr.add_sequence(16)            # 1 page
    mgr.extend(b, 1)                    # 17 tokens -> 2 pages
    assert mgr.free_pages == 0
    with pytest.raises(OutOfPages):
        mgr.extend(a, 20)
    assert mgr.num_sequences() == 2 and mgr.pool_utilization() == 1.0 and mgr.pool().num_used == 4 == mgr.pool().num_total
    mgr.remove_sequence(a)
    assert mgr.free_pages == 2 and a not in mgr.active and mgr.pool_utilization() == 0.5
    k = torch.arange(17 * 8, dtype=torch.float32).view(17, 1, 8)
    cache.append(0, k, -k, torch.arange(17, dtype=torch.int32), torch.full((17,), b, dtype=torch.int32))
    gk, gv = cache.gather(0, b, 17)
    assert torch.equal(gk, k) and torch.equal(gv, -k)
    out = cache.decode(0, torch.ones(2, 1, 8), torch.tensor([0, 17], dtype=torch.int32))
    assert out.shape == (2, 1, 8)


def _run(nproc, port, graph=False, weights="bf16"):
    env = dict(os.environ, NCCL_NVLS_ENABLE="0", MASTER_ADDR="127.0.0.1", FT_TEST_GRAPH="1" if graph else "0",
               FT_COMM_TIMEOUT_MS="5000", FT_TEST_WEIGHTS=weights)
    script = os.path.join(HERE, "engine_worker.py")
    cmd = [sys.executable, script] if nproc == 1 else [
        sys.executable, "-m", "torch.distributed.run", "--nnodes=1", "--nproc-per-node", str(nproc),
        "--master-addr", "127.0.0.1", "--master-port", str(port), script]
    proc = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=240)
    assert proc.returncode == 0, proc.stdout[-3000:] + proc.stderr[-3000:]
    assert "ok" in proc.stdout


@pytest.mark.gpu
def test_engine_single_gpu():
    _run(1, 0)


@pytest.mark.gpu
@pytest.mark.multigpu
def test_engine_tensor_parallel_2():
    _run(2, 29551)


@pytest.mark.gpu
def test_engine_single_gpu_cuda_graph():
    _run(1, 0, graph=True)


@pytest.mark.gpu
@pytest.mark.multigpu
def test_engine_tensor_parallel_2_cuda_graph():
    _run(2, 29552, graph=True)


@pytest.mark.gpu
@pytest.mark.multigpu
def test_engine_tensor_parallel_all_gpus_cuda_graph():
    n = torch.cuda.device_count()
    n = 8 if n >= 8 else 4 if n >= 4 else 2
    if n == 2:
        pytest.skip("covered by the two-GPU test")
    _run(n, 29553, graph=True)


# The Q4_0 weight format of the engine is a composition of kernels that each have their own test
# (gather, dequant-GEMM); these two check the composition.


@pytest.mark.gpu
def test_engine_q4_0_single_gpu():
    _run(1, 0, weights="q4_0")


@pytest.mark.gpu
@pytest.mark.multigpu
def test_engine_q4_0_tensor_parallel_2():
    _run(2, 29553, weights="q4_0")


@pytest.mark.gpu
@pytest.mark.parametrize("D,Hq,Hkv", [(64, 4, 4), (128, 8, 2), (16, 1, 1), (96, 6, 2)])
def test_rotation_into_the_pages_is_rotation_then_append(D, Hq, Hkv):
    # rows of several sequences at positions within, at the edge of and past a page, and a padding row of no sequence
    from ferrotorch_b200.nn.layers import RotaryPositionEmbedding
    from ferrotorch_b200.nn.paged import RaggedBatch

    torch.manual_seed(D + Hq)
    rope = RotaryPositionEmbedding(D, 256)
    with torch.no_grad():
        results = []
        packed = torch.randn(1 + 1 + 40, Hq + 2 * Hkv, D, device="cuda").to(torch.bfloat16)
        for fused in (True, False):
            cache = PagedKVCache(2, Hkv, D, num_blocks=16, max_seqs=3, max_seq_len=256, block_size=16)
            mgr = PagedAttentionManager(cache)
            for n in (17, 60, 40):
                mgr.add_sequence(n)
            batch = RaggedBatch([(0, [1], 16, [0]), (cache.pad_slot, [1], 0, [0]), (1, list(range(40)), 15, [39])], "cuda")
            x = packed.clone()
            if fused:
                cache.append_rotated(1, x, rope, batch, Hq)
            else:
                x = rope(x[None], positions=batch.positions, n_rot_heads=Hq + Hkv)[0]
                cache.append(1, x[:, Hq:Hq + Hkv], x[:, Hq + Hkv:], batch.positions, batch.slots)
            results.append((x[:, :Hq].clone(), cache.k[1], cache.v[1], cache.k[0]))
    for a, b in zip(*results):
        assert torch.equal(a, b)
    assert bool(results[0][1].any()) and not bool(results[0][3].any())


@pytest.mark.gpu
@pytest.mark.parametrize("bs,D,Dv", [(16, 128, 128), (8, 128, 64), (24, 96, 128), (48, 112, 80), (256, 64, 128), (20, 128, 128), (16, 48, 64)])
@pytest.mark.parametrize("splits,window", [(1, 0), (3, 0), (1, 150)])
def test_paged_decode_reads_nothing_past_the_context(bs, D, Dv, splits, window):
    # boxes of 8 to 128 tokens and rows that are copied (pages of 20, heads of 48); contexts that end on a tile, one key past it and inside
    # a page; what the pages hold behind the context is not finite
    torch.manual_seed(bs + D)
    Hkv, G, lens = 2, 4, [1, 128, 129, 256, 700, 1031]
    cache = PagedKVCache(1, Hkv, D, num_blocks=sum((n + bs - 1) // bs for n in lens) + 2, max_seqs=len(lens), max_seq_len=1056, block_size=bs, v_head_dim=Dv)
    cache.k[0].fill_(float("nan")), cache.v[0].fill_(float("nan"))
    mgr = PagedAttentionManager(cache)
    ks, vs = [], []
    for b, n in enumerate(lens):
        assert mgr.add_sequence(n) == b
        ks.append(torch.randn(n, Hkv, D, device="cuda").to(torch.bfloat16)), vs.append(torch.randn(n, Hkv, Dv, device="cuda").to(torch.bfloat16))
        cache.append(0, ks[b], vs[b], torch.arange(n, device="cuda", dtype=torch.int32), torch.full((n,), b, device="cuda", dtype=torch.int32))
    q = torch.randn(len(lens), Hkv * G, D, device="cuda").to(torch.bfloat16)
    out = cache.decode(0, q, torch.tensor(lens, device="cuda", dtype=torch.int32), n_splits=splits, window=window)
    for b, n in enumerate(lens):
        k, v = (t[b][max(0, n - window) if window else 0:].float().repeat_interleave(G, 1) for t in (ks, vs))
        p = torch.softmax(torch.einsum("hd,thd->ht", q[b].float(), k) * D ** -0.5, -1)
        want = torch.einsum("ht,thd->hd", p, v)
        # P and the result are rounded to bf16
        assert bool(((out[b].float() - want).abs() <= 2.0 ** -7 * (1 + want.abs())).all()), "sequence of %d" % n


@pytest.mark.gpu
@pytest.mark.parametrize("change", ["subclass", "forward", "hook", "global hook"])
def test_rotations_and_projections_that_are_not_plain_are_called(change):
    from torch import nn

    from ferrotorch_b200.nn.layers import Linear, RotaryPositionEmbedding, SwiGLU
    from ferrotorch_b200.nn.paged import RaggedBatch
    from ferrotorch_b200.ops import functional as F

    def altered(cls, factor, *args):
        """A module of cls whose result is ``factor`` times what it would be."""
        def scaled(m, x, **kwargs):
            return cls.forward(m, x, **kwargs) * factor

        handle = None
        if change == "subclass":
            m = type("Scaled", (cls,), {"forward": scaled})(*args)
        else:
            m = cls(*args)
            if change == "forward":
                m.forward = lambda x, **kwargs: scaled(m, x, **kwargs)
            elif change == "hook":
                m.register_forward_hook(lambda mod, args, out: out * factor)
            else:
                handle = nn.modules.module.register_module_forward_hook(lambda mod, args, out: out * factor if mod is m else None)
        return m, handle

    torch.manual_seed(0)
    D, Hq, Hkv, T = 64, 4, 2, 5
    packed = torch.randn(T, Hq + 2 * Hkv, D, device="cuda").to(torch.bfloat16)
    rope, handle = altered(RotaryPositionEmbedding, 2, D, 64)
    try:
        cache = PagedKVCache(1, Hkv, D, num_blocks=8, max_seqs=2, max_seq_len=64, block_size=16)
        PagedAttentionManager(cache).add_sequence(T)
        batch = RaggedBatch([(0, list(range(T)), 0, [T - 1])], "cuda")
        with torch.no_grad():
            want = RotaryPositionEmbedding(D, 64)(packed.clone()[None], positions=batch.positions, n_rot_heads=Hq + Hkv)[0] * 2
            q = cache.append_rotated(0, packed.clone(), rope, batch, Hq)
        k, v = cache.gather(0, 0, T)
        assert torch.equal(q, want[:, :Hq]) and torch.equal(k, want[:, Hq:Hq + Hkv]) and torch.equal(v, want[:, Hq + Hkv:])
    finally:
        handle and handle.remove()

    mlp = SwiGLU(512, 1024).to("cuda", torch.bfloat16)
    x = torch.randn(3, 512, device="cuda").to(torch.bfloat16)
    up, handle = altered(Linear, 2, 512, 2048, False)
    up = up.to("cuda", torch.bfloat16)
    up.weight = mlp.gate_up_proj.weight
    try:
        with torch.no_grad():
            want = mlp.down_proj(F.swiglu(F.linear(x, up.weight) * 2))
            mlp.gate_up_proj = up
            assert torch.equal(F.serving(mlp)(x), want)
    finally:
        handle and handle.remove()
    # a bias keeps the projection as well
    mlp = SwiGLU(512, 1024, bias=True).to("cuda", torch.bfloat16)
    with torch.no_grad():
        assert torch.equal(F.serving(mlp)(x), mlp(x))


@pytest.mark.gpu
@pytest.mark.parametrize("bs,D", [(16, 128), (20, 128), (64, 64), (16, 96)])
@pytest.mark.parametrize("Hkv,G", [(8, 1), (4, 2), (4, 4), (4, 8)])
def test_paged_decode_of_more_ctas_than_sms(bs, D, Hkv, G):
    # a loaded server: one CTA for each sequence and key head, two to an SM (a ring of three tiles that wraps many times) up to groups of
    # four heads; boxes, and pages of 20 tokens that are copied; what the pages hold behind the context is not finite
    torch.manual_seed(bs + D + G)
    lens = [1, 128, 129, 700, 1900, 256, 383, 1031] * 5
    B = len(lens)
    assert B * Hkv > torch.cuda.get_device_properties(0).multi_processor_count
    cache = PagedKVCache(1, Hkv, D, num_blocks=sum((n + bs - 1) // bs for n in lens) + 2, max_seqs=B, max_seq_len=1920, block_size=bs)
    cache.k[0].fill_(float("nan")), cache.v[0].fill_(float("nan"))
    mgr = PagedAttentionManager(cache)
    for b, n in enumerate(lens):
        assert mgr.add_sequence(n) == b
    T = sum(lens)
    k, v = (torch.randn(T, Hkv, D, device="cuda").to(torch.bfloat16) for _ in range(2))
    pos = torch.cat([torch.arange(n, dtype=torch.int32) for n in lens]).cuda()
    cache.append(0, k, v, pos, torch.repeat_interleave(torch.arange(B, dtype=torch.int32), torch.tensor(lens)).cuda())
    q = torch.randn(B, Hkv * G, D, device="cuda").to(torch.bfloat16)
    out = cache.decode(0, q, torch.tensor(lens, device="cuda", dtype=torch.int32), n_splits=1)
    at = 0
    for b, n in enumerate(lens):
        kb, vb = (t[at:at + n].float().repeat_interleave(G, 1) for t in (k, v))
        at += n
        want = torch.einsum("ht,thd->hd", torch.softmax(torch.einsum("hd,thd->ht", q[b].float(), kb) * D ** -0.5, -1), vb)
        # P and the result are rounded to bf16
        assert bool(((out[b].float() - want).abs() <= 2.0 ** -7 * (1 + want.abs())).all()), "sequence of %d" % n
    assert _native.device_status(0) == 0
