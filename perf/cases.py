"""The workloads by which the speed of this package is judged, through its public entry points.

Five kinds of work, each over the whole range in which it is used:

* ``train``     one optimizer step of a Llama-shaped decoder on :class:`FlatTrainer` (forward, backward, update);
* ``serve``     one step of the serving engine (:class:`PagedStepper`): single tokens of running sequences, portions of prompts, or both;
* ``resnet``    one training step of a ResNet (convolutions, batch norms, momentum SGD);
* ``attention`` flash attention by itself, forward and backward;
* ``q4``        a linear layer over Q4_0 blocks.

``listed`` gives the cases that are looked at by name, ``draw`` others of the same ranges; ``exact`` restates every kind with plain
torch in 64 bits.  Weights and data are random; shapes are those of the package's presets, tests and benchmarks, or generic.
"""
import math
import random

import torch
import torch.nn.functional as tF

DEV = "cuda"
PAGE = 16
TINY = dict(hidden=512, heads=4, kv=2, dim=128, ffn=1408, vocab=2048)            # the smallest decoder that is trained and served here
LLM_1B = dict(hidden=2048, heads=32, kv=8, dim=64, ffn=8192, vocab=128256)
LLM_3B = dict(hidden=3072, heads=24, kv=8, dim=128, ffn=8192, vocab=128256)
LLM_8B = dict(hidden=4096, heads=32, kv=8, dim=128, ffn=14336, vocab=128256)
MHA_7B = dict(hidden=4096, heads=32, kv=32, dim=128, ffn=11008, vocab=32000)


def listed():
    return [
        # a first run or a unit test of a training script: every launch counts
        dict(name="train_tiny", kind="train", **TINY, layers=2, batch=2, seq=256, micro=1, clip=0.0),
        # fine-tuning a 1B-shaped model on texts of no round length, with gradient clipping
        dict(name="train_ragged", kind="train", **dict(LLM_1B, vocab=32000), layers=2, batch=3, seq=1001, micro=1, clip=1.0),
        # the shape of 8B pre-training: full rows, gradients of several micro-batches summed in fp32, the large vocabulary
        dict(name="train_8b", kind="train", **LLM_8B, layers=2, batch=4, seq=4096, micro=4, clip=0.0),
        # one user's chat: a token at a time
        dict(name="decode_one", kind="serve", **LLM_8B, layers=4, singles=1, ctx=700, portions=0, tokens=0, past=0, graph=True),
        # a loaded server: a token each of many sequences with long contexts
        dict(name="decode_batch", kind="serve", **LLM_8B, layers=4, singles=64, ctx=2048, portions=0, tokens=0, past=0, graph=True),
        # short questions arriving together
        dict(name="prefill_short", kind="serve", **LLM_1B, layers=4, singles=0, ctx=0, portions=3, tokens=77, past=0, graph=False),
        # long prompts
        dict(name="prefill_batch", kind="serve", **LLM_8B, layers=4, singles=0, ctx=0, portions=4, tokens=2048, past=0, graph=False),
        # a step of continuous batching: running sequences beside a portion of a long prompt whose beginning is cached
        dict(name="mixed_step", kind="serve", **LLM_3B, layers=4, singles=24, ctx=900, portions=1, tokens=500, past=1024, graph=False),
        # images of an odd size in a small batch
        dict(name="resnet18_small", kind="resnet", depth=18, batch=8, side=193, classes=1000),
        # the usual image-classification training step
        dict(name="resnet50_train", kind="resnet", depth=50, batch=256, side=224, classes=1000),
        # attention over a long document, forward and backward
        dict(name="attention_long", kind="attention", batch=1, q_len=8192, k_len=8192, heads=32, kv=8, dim=128, causal=True),
        # a decode-sized batch through the gate/up projection of a quantised 70B-shaped model
        dict(name="q4_decode", kind="q4", rows=32, n=28672, k=8192),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["train", "train", "serve", "serve", "serve", "resnet", "attention", "q4"])
    if kind == "train":
        arch = dict(rng.choice([TINY, LLM_1B, LLM_3B, LLM_8B, MHA_7B]))
        arch["vocab"] = rng.choice([2048, 32000, 128256])
        micro = rng.choice([1, 1, 2, 4])
        seq = _log(rng, 64, 4096)
        batch = micro * rng.randint(1, max(1, min(4, 8192 // (seq * micro))))
        return dict(kind=kind, **arch, layers=rng.randint(1, 2), batch=batch, seq=seq, micro=micro, clip=rng.choice([0.0, 1.0]))
    if kind == "serve":
        arch = rng.choice([TINY, LLM_1B, LLM_3B, LLM_8B, MHA_7B])
        mode = rng.choice(["decode", "decode", "prefill", "mixed"])
        tokens = _log(rng, 2, 2048)
        return dict(kind=kind, **arch, layers=rng.randint(1, 4), singles=_log(rng, 1, 64) if mode != "prefill" else 0, ctx=_log(rng, 16, 4000),
                    portions=0 if mode == "decode" else rng.randint(1, max(1, min(8, 4096 // tokens))), tokens=tokens if mode != "decode" else 0,
                    past=rng.choice([0, 0, _log(rng, 16, 2000)]) if mode != "decode" else 0, graph=mode == "decode")
    if kind == "resnet":
        depth, side = rng.choice([18, 34, 50]), rng.randint(96, 256)
        return dict(kind=kind, depth=depth, batch=_log(rng, 2, 256 * 200 * 200 // (side * side)), side=side, classes=rng.choice([10, 1000]))
    if kind == "attention":
        q = _log(rng, 64, 8192)
        dim = rng.choice([64, 128])
        kv = rng.choice([1, 4, 8])
        causal = rng.random() < 0.7
        same = rng.random() < 0.7
        return dict(kind=kind, batch=rng.randint(1, max(1, min(4, 8192 // q))), q_len=q, k_len=q if same else q + _log(rng, 16, 2048), heads=kv * rng.choice([1, 2, 4]),
                    kv=kv, dim=dim, causal=causal)
    return dict(kind=kind, rows=_log(rng, 1, 2048), n=8 * _log(rng, 128, 3584), k=64 * _log(rng, 16, 224))


# --------------------------------------------------------------------------- decoders
def _config(case, positions):
    from ferrotorch_b200.models.llama import LlamaConfig

    return LlamaConfig(vocab_size=case["vocab"], hidden_size=case["hidden"], intermediate_size=case["ffn"], num_hidden_layers=case["layers"],
                       num_attention_heads=case["heads"], num_key_value_heads=case["kv"], head_dim=case["dim"], max_position_embeddings=positions)


def _decoder(case, positions, gen):
    from ferrotorch_b200.models.llama import LlamaForCausalLM

    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device(DEV):
            model = LlamaForCausalLM(_config(case, positions))
    finally:
        torch.set_default_dtype(old)
    with torch.no_grad():
        for p in model.parameters():                      # projections ~ N(0, 0.02), norms near 1, as after some training
            p.normal_(0.0, 0.02, generator=gen) if p.dim() > 1 else p.uniform_(0.9, 1.1, generator=gen)
    return model


def _llama_params(case):
    h, d, f = case["hidden"], case["dim"], case["ffn"]
    layer = h * d * (2 * case["heads"] + 2 * case["kv"]) + 3 * h * f + 2 * h
    return layer * case["layers"] + h, case["vocab"] * h


def _contexts(case):
    """Cached tokens of every single-token sequence: ragged, the longest ``ctx``."""
    return [case["ctx"] - (i * 37) % (case["ctx"] // 4 + 1) for i in range(case["singles"])]


def _portions(case):
    """Tokens of every prompt portion: ragged, the first the longest."""
    return [max(2, case["tokens"] - (i * 29) % (case["tokens"] // 8 + 1)) for i in range(case["portions"])]


def _prepare_train(case, gen, seed):
    from ferrotorch_b200.train.engine import FlatTrainer

    model = _decoder(case, case["seq"], gen)
    tr = FlatTrainer(model, lr=3e-4, betas=(0.9, 0.95), weight_decay=0.1, max_grad_norm=case["clip"] or None, micro_batches=case["micro"])
    ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), device=DEV, generator=gen)
    return dict(kind="train", trainer=tr, x=ids[:, :-1].contiguous(), y=ids[:, 1:].contiguous())


def _prepare_serve(case, gen, seed):
    from ferrotorch_b200.models.serving import PagedStepper

    ctx, por = _contexts(case), _portions(case)
    spans = [(c, 1) for c in ctx] + [(case["past"], n) for n in por]
    top = max(a + b for a, b in spans)
    model = _decoder(case, top, gen).eval()
    pages = sum((a + b + PAGE - 1) // PAGE for a, b in spans)
    st = PagedStepper(model, pages, PAGE, len(spans), top, cuda_graph=case["graph"])
    for t in [*st.cache.k, *st.cache.v]:                  # what earlier tokens left: rotated keys and values of a normed hidden state
        t.normal_(0.0, 0.02 * math.sqrt(case["hidden"]), generator=gen)
    rng, entries = random.Random(seed), []
    for start, n in spans:
        slot = st.admit()
        st.reserve(slot, start + n)
        entries.append((slot, [rng.randrange(case["vocab"]) for _ in range(n)], start, [n - 1]))
    return dict(kind="serve", stepper=st, entries=entries)


def _rms(x, w):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * w


def _rotate(x, pos, theta=500000.0):
    """Halves of a head rotated: ``x [T, heads, dim]``."""
    d = x.shape[-1]
    # the angles are tables of the model, held in 32 bits
    inv = 1.0 / (theta ** (torch.arange(0, d, 2, device=x.device, dtype=torch.float32) / d))
    ang = pos.float()[:, None] * inv
    cos, sin = ang.cos().double()[:, None], ang.sin().double()[:, None]
    a, b = x[..., :d // 2], x[..., d // 2:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(q, k, v, causal, offset):
    """``q [Sq, Hq, D]``, ``k / v [Sk, Hkv, D]`` -> ``[Sq, Hq, D]``, a group of heads at a time."""
    g, out = q.shape[1] // k.shape[1], []
    dead = None
    if causal:
        dead = torch.arange(k.shape[0], device=q.device)[None] > torch.arange(q.shape[0], device=q.device)[:, None] + offset
    for h in range(k.shape[1]):
        s = torch.einsum("qhd,kd->hqk", q[:, h * g:(h + 1) * g], k[:, h]) * q.shape[-1] ** -0.5
        if dead is not None:
            s = s.masked_fill(dead, float("-inf"))
        out.append(torch.einsum("hqk,kd->qhd", s.softmax(-1), v[:, h]))
    return torch.cat(out, 1)


def _layer_exact(case, p, i, x, attention):
    n = "model.layers.%d." % i
    h = _rms(x, p[n + "input_layernorm.weight"])
    qkv = (h @ p[n + "self_attn.qkv_proj.weight"].t()).unflatten(-1, (-1, case["dim"]))
    x = x + attention(i, qkv).flatten(-2) @ p[n + "self_attn.o_proj.weight"].t()
    h = _rms(x, p[n + "post_attention_layernorm.weight"])
    gate, up = (h @ p[n + "mlp.gate_up_proj.weight"].t()).chunk(2, -1)
    return x + (tF.silu(gate) * up) @ p[n + "mlp.down_proj.weight"].t()


def _exact_train(case, state):
    tr, B, S = state["trainer"], case["batch"], case["seq"]
    p = {n: q.detach().double().requires_grad_() for n, q in tr.model.named_parameters()}
    hq, hkv = case["heads"], case["kv"]
    pos = torch.arange(S, device=DEV)
    total = 0.0

    def attention(_, qkv):
        rot = _rotate(qkv[:, :hq + hkv], pos)
        return _attend(rot[:, :hq], rot[:, hq:], qkv[:, hq + hkv:], True, 0)

    for b in range(B):
        x = p["model.embed_tokens.weight"][state["x"][b]]
        for i in range(case["layers"]):
            x = _layer_exact(case, p, i, x, attention)
        z = _rms(x, p["model.norm.weight"]) @ p["lm_head.weight"].t()
        loss = tF.cross_entropy(z, state["y"][b], reduction="sum") / (B * S)
        loss.backward()
        total += loss.detach()
    return [total, *_updated(tr, p, case["clip"])]


def _updated(tr, p, clip):
    """Gradients and updated weights after the first step, in the trainer's flat layout."""
    a = tr.arena
    grads = torch.zeros(a.numel, device=DEV, dtype=torch.float64)
    params = torch.zeros_like(grads)
    scale = 1.0
    if clip:
        scale = min(1.0, clip / (float(sum(q.grad.square().sum() for q in p.values())) ** 0.5 + 1e-6))
    for n, q, off, num in a.slots:
        w = p[n].detach().reshape(-1)
        g = p[n].grad.reshape(-1)
        grads[off:off + num] = g
        g = g * scale
        if tr.kind == "sgd":
            params[off:off + num] = w - tr.lr * (g + tr.weight_decay * w)
        else:
            decay = tr.weight_decay if q.dim() >= 2 else 0.0
            params[off:off + num] = w * (1 - tr.lr * decay) - tr.lr * g / (g.abs() + tr.eps)      # the first step: m^ = g, v^ = g^2
    return grads, params


def _exact_serve(case, state):
    st, entries = state["stepper"], state["entries"]
    cache, hq, hkv = st.cache, case["heads"], case["kv"]
    p = {n: q.detach().double() for n, q in st.model.named_parameters()}
    ks, vs = [t.double() for t in cache.k], [t.double() for t in cache.v]
    starts = [e[2] for e in entries]
    lens = [len(e[1]) for e in entries]
    rows = [sum(lens[:i]) for i in range(len(lens))]
    pos = torch.tensor([s + j for s, n in zip(starts, lens) for j in range(n)], device=DEV)
    pages = [torch.tensor(cache.pages_of(e[0]), device=DEV) for e in entries]

    def attention(i, qkv):
        rot = _rotate(qkv[:, :hq + hkv], pos)
        out = []
        for s, n, r, pg in zip(starts, lens, rows, pages):
            at = torch.arange(s, s + n, device=DEV)
            ks[i][pg[at // PAGE], at % PAGE] = rot[r:r + n, hq:]
            vs[i][pg[at // PAGE], at % PAGE] = qkv[r:r + n, hq + hkv:]
            k, v = ks[i][pg].flatten(0, 1)[:s + n], vs[i][pg].flatten(0, 1)[:s + n]
            out.append(_attend(rot[r:r + n, :hq], k, v, True, s))
        return torch.cat(out)

    x = p["model.embed_tokens.weight"][torch.tensor([t for e in entries for t in e[1]], device=DEV)]
    for i in range(case["layers"]):
        x = _layer_exact(case, p, i, x, attention)
    x = x[torch.tensor([r + n - 1 for r, n in zip(rows, lens)], device=DEV)]
    return [_rms(x, p["model.norm.weight"]) @ p["lm_head.weight"].t(), *ks, *vs]


# --------------------------------------------------------------------------- ResNets
def _resnet_loss(model, x, y):
    return tF.cross_entropy(model(x).float(), y)


def _prepare_resnet(case, gen, seed):
    from ferrotorch_b200.models import resnet
    from ferrotorch_b200.train.engine import FlatTrainer

    with torch.device(DEV):
        model = getattr(resnet, "resnet%d" % case["depth"])(num_classes=case["classes"])
    model = model.to(memory_format=torch.channels_last)
    with torch.no_grad():
        for n, p in model.named_parameters():
            if p.dim() == 4:                              # fan-out initialisation
                p.normal_(0.0, math.sqrt(2.0 / (p.shape[0] * p.shape[2] * p.shape[3])), generator=gen)
            elif p.dim() == 2:
                p.normal_(0.0, 0.01, generator=gen)
            elif n.endswith("weight"):                    # the last norm of a block starts small, as training recipes have it
                last = n.endswith("bn3.weight") or (case["depth"] < 50 and n.endswith("bn2.weight"))
                p.fill_(0.2 if last else 1.0)
            else:
                p.zero_()
    tr = FlatTrainer(model.to(torch.bfloat16), optimizer="sgd", lr=0.1, momentum=0.9, weight_decay=1e-4, loss_fn=_resnet_loss, no_decay=lambda n, p: False)
    x = torch.randn((case["batch"], 3, case["side"], case["side"]), device=DEV, generator=gen).to(torch.bfloat16)
    y = torch.randint(0, case["classes"], (case["batch"],), device=DEV, generator=gen)
    return dict(kind="resnet", trainer=tr, x=x.contiguous(memory_format=torch.channels_last), y=y)


def _resnet_blocks(depth):
    """``(name, input channels, channels, stride, bottleneck)`` of every block."""
    counts = {18: (2, 2, 2, 2), 34: (3, 4, 6, 3), 50: (3, 4, 6, 3)}[depth]
    grow, cin, out = (4 if depth == 50 else 1), 64, []
    for s, (n, c) in enumerate(zip(counts, (64, 128, 256, 512))):
        for b in range(n):
            out.append(("layer%d.%d." % (s + 1, b), cin, c, 2 if s and not b else 1, grow == 4))
            cin = c * grow
    return out


def _exact_resnet(case, state):
    if case["batch"] * case["side"] ** 2 * (2 if case["depth"] == 50 else 1) > 64 * 224 * 224 * 2:
        return None                                       # too slow in 64 bits
    tr = state["trainer"]
    p = {n: q.detach().double().contiguous().requires_grad_() for n, q in tr.model.named_parameters()}

    def bn(x, n):
        return tF.batch_norm(x, None, None, p[n + ".weight"], p[n + ".bias"], True, 0.0, 1e-5)

    x = state["x"].double().contiguous()
    x = tF.max_pool2d(tF.relu(bn(tF.conv2d(x, p["conv1.weight"], stride=2, padding=3), "bn1")), 3, 2, 1)
    for n, cin, c, stride, bottle in _resnet_blocks(case["depth"]):
        idt = x if n + "downsample.0.weight" not in p else bn(tF.conv2d(x, p[n + "downsample.0.weight"], stride=stride), n + "downsample.1")
        if bottle:
            o = tF.relu(bn(tF.conv2d(x, p[n + "conv1.weight"]), n + "bn1"))
            o = tF.relu(bn(tF.conv2d(o, p[n + "conv2.weight"], stride=stride, padding=1), n + "bn2"))
            o = bn(tF.conv2d(o, p[n + "conv3.weight"]), n + "bn3")
        else:
            o = tF.relu(bn(tF.conv2d(x, p[n + "conv1.weight"], stride=stride, padding=1), n + "bn1"))
            o = bn(tF.conv2d(o, p[n + "conv2.weight"], padding=1), n + "bn2")
        x = tF.relu(o + idt)
    z = x.mean((2, 3)) @ p["fc.weight"].t() + p["fc.bias"]
    loss = tF.cross_entropy(z, state["y"])
    loss.backward()
    return [loss.detach(), *_updated(tr, p, 0.0)]


def _resnet_work(case):
    """Parameters and multiply-adds of an image's forward pass."""
    half = lambda n: (n - 1) // 2 + 1                     # noqa: E731
    side = half(case["side"])
    macs, params = side * side * 64 * 147, 64 * 147 + 128
    side = half(side)
    for n, cin, c, stride, bottle in _resnet_blocks(case["depth"]):
        out = half(side) if stride == 2 else side
        wide = c * (4 if bottle else 1)
        convs = [(side, cin * c), (out, 9 * c * c), (out, c * wide)] if bottle else [(out, 9 * cin * c), (out, 9 * c * c)]
        if stride == 2 or cin != wide:
            convs.append((out, cin * wide))
        macs += sum(s * s * w for s, w in convs)
        params += sum(w for _, w in convs) + 2 * (2 * c + wide)
        side = out
    return params + (512 * (4 if case["depth"] == 50 else 1) + 1) * case["classes"], macs


# --------------------------------------------------------------------------- attention, quantised layers
def _prepare_attention(case, gen, seed):
    def t(n, h):
        return torch.randn((case["batch"], n, h, case["dim"]), device=DEV, generator=gen).to(torch.bfloat16)

    q, k, v = t(case["q_len"], case["heads"]), t(case["k_len"], case["kv"]), t(case["k_len"], case["kv"])
    return dict(kind="attention", q=q.requires_grad_(), k=k.requires_grad_(), v=v.requires_grad_(), d=t(case["q_len"], case["heads"]), causal=case["causal"])


def _exact_attention(case, state):
    outs = []
    g = case["heads"] // case["kv"]
    for b in range(case["batch"]):
        parts = []
        for h in range(case["kv"]):                       # a key head and its queries at a time
            q = state["q"][b, :, h * g:(h + 1) * g].detach().double().requires_grad_()
            k, v = (state[n][b, :, h:h + 1].detach().double().requires_grad_() for n in "kv")
            o = _attend(q, k, v, case["causal"], case["k_len"] - case["q_len"])
            parts.append([o.detach(), *torch.autograd.grad(o, (q, k, v), state["d"][b, :, h * g:(h + 1) * g].double())])
        outs.append([torch.cat(x, 1) for x in zip(*parts)])
    return [torch.stack(x) for x in zip(*outs)]


def _prepare_q4(case, gen, seed):
    from ferrotorch_b200.ops.quant import Q4Linear, quantize_q4_0_planes

    w = torch.randn((case["n"], case["k"]), device=DEV, generator=gen) * 0.02
    return dict(kind="q4", layer=Q4Linear(*quantize_q4_0_planes(w)), x=torch.randn((case["rows"], case["k"]), device=DEV, generator=gen).to(torch.bfloat16))


def _exact_q4(case, state):
    nib, sc = state["layer"].nibbles, state["layer"].scales
    x, out = state["x"].double(), []
    for r in range(0, case["n"], 4096):
        b = nib[r:r + 4096].view(-1, case["k"] // 32, 16)
        w = (torch.cat([b & 15, b >> 4], -1).double() - 8.0) * sc[r:r + 4096].double()[..., None]
        out.append(x @ w.flatten(1).t())
    return [torch.cat(out, 1)]


# --------------------------------------------------------------------------- what is asked for
def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    make = dict(train=_prepare_train, serve=_prepare_serve, resnet=_prepare_resnet, attention=_prepare_attention, q4=_prepare_q4)
    return make[case["kind"]](case, gen, seed)


def run(state):
    kind = state["kind"]
    if kind in ("train", "resnet"):
        tr = state["trainer"]
        loss = tr.step(state["x"], state["y"])
        return [loss, tr.arena.grads, tr.arena.params]
    if kind == "serve":
        st = state["stepper"]
        return [st.step(state["entries"]), *st.cache.k, *st.cache.v]
    if kind == "attention":
        from ferrotorch_b200.ops.attention import flash_attention

        q, k, v = state["q"], state["k"], state["v"]
        out = flash_attention(q, k, v, causal=state["causal"])
        return [out.detach(), *torch.autograd.grad(out, (q, k, v), state["d"])]
    return [state["layer"](state["x"])]


def work(case):
    kind = case["kind"]
    if kind == "train":
        body, table = _llama_params(case)
        rows, grad = case["batch"] * case["seq"], 4 if case["micro"] > 2 else 2
        att = 6 * case["seq"] * rows * case["heads"] * case["dim"] * case["layers"]              # causal: half of the scores
        # weights read and written, gradients written, fp32 weights and two moments read and written
        return dict(bytes=(body + 2 * table) * (4 + grad + 24) + rows * 16, flops=6 * (body + table) * rows + att)
    if kind == "serve":
        body, table = _llama_params(case)
        spans = [(c, 1) for c in _contexts(case)] + [(case["past"], n) for n in _portions(case)]
        rows, seqs = sum(n for _, n in spans), len(spans)
        seen = sum(n * a + n * (n + 1) // 2 for a, n in spans)                                   # query-key pairs
        kv = 2 * 2 * case["kv"] * case["dim"] * case["layers"]
        nbytes = 2 * (body + table + rows * case["hidden"] + seqs * case["vocab"]) + kv * (sum(a for a, _ in spans) + rows)
        return dict(bytes=nbytes, flops=2 * (body * rows + table * seqs) + 4 * seen * case["heads"] * case["dim"] * case["layers"])
    if kind == "resnet":
        params, macs = _resnet_work(case)
        # weights read and written, gradients written, fp32 weights and momentum read and written, images read
        return dict(bytes=params * (4 + 2 + 16) + case["batch"] * case["side"] ** 2 * 6, flops=6 * macs * case["batch"])
    if kind == "attention":
        b, sq, sk, h, kv, d = (case[n] for n in ("batch", "q_len", "k_len", "heads", "kv", "dim"))
        pairs = sq * (sk - sq) + sq * (sq + 1) // 2 if case["causal"] else sq * sk
        return dict(bytes=2 * b * d * (4 * sq * h + 4 * sk * kv), flops=12 * b * h * d * pairs)
    return dict(bytes=case["n"] * case["k"] * 9 / 16 + 2 * case["rows"] * (case["n"] + case["k"]), flops=2.0 * case["rows"] * case["n"] * case["k"])


def tolerance(case):
    """About four times what the paths show against :func:`exact`; weights, activations and results are bf16."""
    return dict(rel={"train": 0.07, "serve": 0.07, "resnet": 0.2, "attention": 0.01, "q4": 0.01}[case["kind"]])


def exact(case, seed):
    state = prepare(case, seed)
    fn = dict(train=_exact_train, serve=_exact_serve, resnet=_exact_resnet, attention=_exact_attention, q4=_exact_q4)[case["kind"]]
    if case["kind"] in ("train", "resnet", "attention"):
        return fn(case, state)
    with torch.no_grad():
        return fn(case, state)
