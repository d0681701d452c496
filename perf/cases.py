"""The work that is timed: what a program built on this framework has it do, over the range it is used in.

A case names a kind of call and its sizes:

  layer   `SparseMoe.forward` on device tensors, through a stack of layers that rotate (so that the weights come
          from memory, as they do in a model): GGUF Q4_K experts with f16 activations, or bf16 / f16 / f32 banks
  host    the same call on host arrays: the copies in and out and the wait are inside the call
  decode  one greedy decode step of the whole OLMoE-shaped decoder, replayed from the graph a serving loop keeps
  prompt  `OlmoeDecoder.forward` on a prompt, the way a sequence enters the cache

Shapes are the repository's own: OLMoE (hidden 2048, intermediate 1024, 64 experts, top-8), the 128-expert
shape (intermediate 768, renormalised weights), and a small 16-expert layer.  Weights are N(0, 0.02), activations
N(0, 1), as in the benchmark; everything is drawn on the device from the seed.
"""
from __future__ import annotations

import math

import torch

from mummu_b200 import _lib as L
from mummu_b200 import moe, synth
from mummu_b200.olmoe import OlmoeConfig, OlmoeDecoder, bucket

ACT = {"q4_k": L.F16, "f16": L.F16, "bf16": L.BF16, "f32": L.F32}
WEIGHT = {"q4_k": L.Q4_K, "f16": L.F16, "bf16": L.BF16, "f32": L.F32}
TORCH = {"q4_k": torch.float16, "f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
WEIGHT_BYTES = {"q4_k": 144 / 256, "f16": 2, "bf16": 2, "f32": 4}

OLMOE = dict(hidden=2048, inter=1024, experts=64, top_k=8, norm=False)
WIDE = dict(hidden=2048, inter=768, experts=128, top_k=8, norm=True)
SMALL = dict(hidden=1024, inter=512, experts=16, top_k=2, norm=False)


def listed():
    return [
        # one sequence being decoded: a token through the experts of layer after layer
        dict(name="q4k_token", kind="layer", dtype="q4_k", tokens=1, layers=4, skew=0.0, **OLMOE),
        # the benchmark's batch of sequences in decode
        dict(name="q4k_batch64", kind="layer", dtype="q4_k", tokens=64, layers=4, skew=0.0, **OLMOE),
        # a large decode batch of ragged size: several tiles of rows per expert
        dict(name="q4k_batch201", kind="layer", dtype="q4_k", tokens=201, layers=4, skew=0.0, **OLMOE),
        # a prompt on the same packed weights
        dict(name="q4k_prompt777", kind="layer", dtype="q4_k", tokens=777, layers=2, skew=0.0, **OLMOE),
        # a host program without device tensors: a decode batch in pinned host arrays, in and out
        dict(name="q4k_host32", kind="host", dtype="q4_k", tokens=32, layers=4, skew=0.0, **OLMOE),
        # decode on an unquantised checkpoint
        dict(name="bf16_batch47", kind="layer", dtype="bf16", tokens=47, layers=1, skew=0.0, **OLMOE),
        # prefill with a skewed router: the hottest expert serves about eight times the mean load
        dict(name="bf16_prefill4096", kind="layer", dtype="bf16", tokens=4096, layers=1, skew=1.0, **OLMOE),
        # the largest: a full step of the 128-expert shape
        dict(name="bf16_wide16384", kind="layer", dtype="bf16", tokens=16384, layers=1, skew=0.0, **WIDE),
        # the reference's own precision: the layer its parity is stated on
        dict(name="f32_batch16", kind="layer", dtype="f32", tokens=16, layers=1, skew=0.0, **OLMOE),
        # the whole model, one sequence and a serving batch, half a thousand keys in the cache
        dict(name="model_decode1", kind="decode", batch=1, keys=517),
        dict(name="model_decode32", kind="decode", batch=32, keys=517),
        # prompts entering the cache, as many tokens as the benchmark feeds at a time
        dict(name="model_prompt4x512", kind="prompt", batch=4, length=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["q4k", "q4k", "q4k", "host", "half", "half", "f32", "decode", "prompt"])
    if kind == "decode":
        return dict(kind="decode", batch=_log(rng, 1, 32), keys=_log(rng, 40, 600))
    if kind == "prompt":
        batch = _log(rng, 1, 8)
        return dict(kind="prompt", batch=batch, length=_log(rng, 33, 2048 // batch))
    shape = rng.choice([OLMOE, OLMOE, WIDE, SMALL])
    skew = rng.choice([0.0, 0.0, 1.0])
    if kind == "q4k":
        tokens = _log(rng, 1, 2048)
        return dict(kind="layer", dtype="q4_k", tokens=tokens, layers=4 if tokens <= 256 else 2, skew=skew, **shape)
    if kind == "host":
        return dict(kind="host", dtype="q4_k", tokens=_log(rng, 1, 256), layers=4, skew=skew, **shape)
    if kind == "f32":
        return dict(kind="layer", dtype="f32", tokens=_log(rng, 1, 128), layers=1, skew=skew, **shape)
    return dict(kind="layer", dtype=rng.choice(["bf16", "f16"]), tokens=_log(rng, 1, 12000), layers=1, skew=skew, **shape)


class _Case:
    """What the program holds before the call; run() fills `out` anew each time."""


def _layers(case, gen):
    H, I, E, K = case["hidden"], case["inter"], case["experts"], case["top_k"]
    dtype = case["dtype"]
    cfg = moe.SparseMoeConfig(H, I, E, K)
    bias = synth.zipf_router_bias(E, case["skew"]) if case["skew"] else None
    stack = []
    for l in range(case["layers"]):
        m = cfg.init(device=0, act_dtype=ACT[dtype], weight_dtype=WEIGHT[dtype], max_tokens=case["tokens"] if l == 0 else 0)
        if l:
            m.adopt_scratch(stack[0])
        m.set_router((torch.randn(H, E, generator=gen, device="cuda") * 0.02).cpu().numpy(), bias=bias)
        for which, shape in ((L.BANK_GATE, (E, I, H)), (L.BANK_UP, (E, I, H)), (L.BANK_DOWN, (E, H, I))):
            w = torch.randn(shape, generator=gen, device="cuda").mul_(0.02)
            m.set_bank(which, moe.q4k_quantize_device(w) if dtype == "q4_k" else w.to(TORCH[dtype]))
            del w
        stack.append(m)
    return stack


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = _Case()
    s.kind = case["kind"]
    if s.kind in ("layer", "host"):
        s.top_k, s.norm = case["top_k"], case["norm"]
        s.layers = _layers(case, gen)
        xs = [torch.randn(case["tokens"], case["hidden"], generator=gen, device="cuda").to(TORCH[case["dtype"]])
              for _ in s.layers]
        if s.kind == "host":
            s.pinned = [(x.cpu().pin_memory(), torch.empty(x.shape, dtype=x.dtype).pin_memory()) for x in xs]
            s.xs = [(x.numpy(), y.numpy()) for x, y in s.pinned]
        else:
            s.xs = xs
        return s
    cfg = OlmoeConfig()
    B = case["batch"]
    keys = case["keys"] if s.kind == "decode" else case["length"]
    max_ctx = 640 if s.kind == "decode" else keys
    s.dec = OlmoeDecoder(cfg, device=0, expert_dtype=L.Q4_K, max_batch=B, max_ctx=max_ctx,
                         max_tokens=B if s.kind == "decode" else B * keys)
    s.dec.random_init(seed=seed)
    s.dec.embed.mul_(50.0)         # a trained checkpoint's residual stream: unit scale beside what one layer adds to it
    s.ids = torch.randint(0, cfg.vocab_size, (B, keys), generator=gen, device="cuda")
    if s.kind == "prompt":
        s.batch, s.length = B, keys
        return s
    # sequences of different lengths: `keys` cached positions for the longest
    lengths = [keys - (7 * b) % (keys // 4 + 1) for b in range(B)]
    s.state = s.dec.static_state(B, max_ctx)
    s.dec.k_cache.normal_(generator=gen)
    s.dec.v_cache.normal_(generator=gen).mul_(0.9)
    for b in range(B):
        s.dec.seed_static(s.state, b, lengths[b])
    s.state.tokens[:, 0] = s.ids[:, -1].to(torch.int32)
    s.state.positions.copy_(torch.tensor(lengths, dtype=torch.int32))
    s.graph = s.dec.make_decode_graph(s.state, B, bucket(keys + 1, max_ctx))
    return s


def run(s):
    if s.kind == "layer":
        return [m.forward(x, s.top_k, s.norm) for m, x in zip(s.layers, s.xs)]
    if s.kind == "host":
        return [m.forward(x, s.top_k, s.norm, out=y) for m, (x, y) in zip(s.layers, s.xs)]
    if s.kind == "decode":
        s.graph.replay()
        return s.state.logits
    logits = s.dec.forward(s.ids, 0)
    return logits, s.dec.k_cache[:, :s.batch, :, :s.length], s.dec.v_cache[:, :s.batch, :, :s.length]


def _experts_hit(experts, top_k, tokens):
    return experts * (1.0 - (1.0 - top_k / experts) ** tokens)


def work(case):
    if case["kind"] in ("layer", "host"):
        H, I, E, K, T = case["hidden"], case["inter"], case["experts"], case["top_k"], case["tokens"]
        act = 4 if case["dtype"] == "f32" else 2
        hit = _experts_hit(E, K, T)
        per_layer = hit * 3 * H * I * WEIGHT_BYTES[case["dtype"]] + H * E * 4 + 2 * T * H * act
        return {"bytes": case["layers"] * per_layer, "flops": case["layers"] * (T * K * 6.0 * H * I + 2.0 * T * H * E)}
    c = OlmoeConfig()
    H, I, E, K, V, NL = (c.hidden_size, c.intermediate_size, c.num_experts, c.num_experts_per_tok, c.vocab_size,
                         c.num_hidden_layers)
    B = case["batch"]
    if case["kind"] == "decode":
        T, pairs = B, sum(case["keys"] - (7 * b) % (case["keys"] // 4 + 1) + 1 for b in range(B))
        kv = 2 * pairs * H * 2
    else:
        T, pairs = B * case["length"], B * case["length"] * (case["length"] + 1) / 2
        kv = 2 * T * H * 2
    layer_bytes = _experts_hit(E, K, T) * 3 * H * I * 144 / 256 + H * E * 4 + 4 * H * H * 2 + kv
    layer_flops = T * K * 6.0 * H * I + 2.0 * T * H * E + 8.0 * T * H * H + 4.0 * pairs * H
    return {"bytes": NL * layer_bytes + V * H * 2 + T * H * 2 + B * V * 4, "flops": NL * layer_flops + 2.0 * B * V * H}


def _unpack_q4k(raw, shape):
    """Q4_K bytes -> the values they stand for, f64: d*scale*q - dmin*min, (scale, min) six bits each."""
    blk = raw.view(-1, 144)
    d, dmin = blk[:, 0:4].contiguous().view(torch.float16).double().split(1, 1)
    lo, mid, hi = blk[:, 4:8].int(), blk[:, 8:12].int(), blk[:, 12:16].int()
    sc = torch.cat([lo & 63, (hi & 15) | ((lo >> 6) << 4)], 1).double()
    mn = torch.cat([mid & 63, (hi >> 4) | ((mid >> 6) << 4)], 1).double()
    q = blk[:, 16:].view(-1, 4, 32)
    q = torch.stack([q & 15, q >> 4], 2).view(-1, 8, 32).double()
    return ((d * sc)[:, :, None] * q - (dmin * mn)[:, :, None]).view(shape)


def _moe64(x, router, bias, banks, shapes, top_k, norm):
    """The layer in 64 bits from the values its weights stand for; banks as given to the handle, one expert at a time."""
    p = torch.softmax(x @ router + bias, -1)
    w, ids = p.topk(top_k, -1)
    if norm:
        w = w / w.sum(-1, keepdim=True)
    y = torch.zeros_like(x)

    def weight(b, e):
        if banks[b].dtype == torch.uint8:
            return _unpack_q4k(banks[b].view(shapes[b][0], -1)[e], shapes[b][1:])
        return banks[b][e].double()
    for e in range(shapes[0][0]):
        t, k = (ids == e).nonzero(as_tuple=True)
        if t.numel():
            h = torch.nn.functional.silu(x[t] @ weight(0, e).T) * (x[t] @ weight(1, e).T)
            y[t] += (h @ weight(2, e).T) * w[t, k][:, None]
    return y


def _exact_layers(case, gen):
    H, I, E = case["hidden"], case["inter"], case["experts"]
    shapes = [(E, I, H), (E, I, H), (E, H, I)]
    bias = synth.zipf_router_bias(E, case["skew"]) if case["skew"] else [0.0] * E
    bias = torch.tensor(bias, dtype=torch.float64, device="cuda")
    layers = []
    for _ in range(case["layers"]):
        router = (torch.randn(H, E, generator=gen, device="cuda") * 0.02).double()
        banks = []
        for shape in shapes:
            w = torch.randn(shape, generator=gen, device="cuda").mul_(0.02)
            banks.append(moe.q4k_quantize_device(w) if case["dtype"] == "q4_k" else w.to(TORCH[case["dtype"]]))
        layers.append((router, banks))
    xs = [torch.randn(case["tokens"], H, generator=gen, device="cuda").to(TORCH[case["dtype"]]).double() for _ in layers]
    return [_moe64(x, r, bias, b, shapes, case["top_k"], case["norm"]) for x, (r, b) in zip(xs, layers)]


def _exact_model(case, gen, seed):
    """The decoder in 64 bits from the 16-bit and packed weights: new tokens against a cache (decode) or against each
    other (prompt).  The weights are drawn as `OlmoeDecoder.random_init` draws them."""
    c = OlmoeConfig()
    H, E, I, V, NL, nh, hd = (c.hidden_size, c.num_experts, c.intermediate_size, c.vocab_size, c.num_hidden_layers,
                              c.num_attention_heads, c.head_dim)
    B = case["batch"]
    decode = case["kind"] == "decode"
    keys = case["keys"] if decode else case["length"]
    ids = torch.randint(0, V, (B, keys), generator=gen, device="cuda")
    lengths = [0] * B
    if decode:
        kc, vc = (torch.empty(NL, B, nh, 640, hd, dtype=torch.float16, device="cuda") for _ in range(2))
        kc.normal_(generator=gen)
        vc.normal_(generator=gen).mul_(0.9)
        lengths = [keys - (7 * b) % (keys // 4 + 1) for b in range(B)]
        ids = ids[:, -1:]
    T = ids.shape[1]
    wgen = torch.Generator(device="cuda")
    wgen.manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=wgen, device="cuda") * 0.02
    embed, lm_head = rnd(V, H).to(torch.float16).mul_(50.0), rnd(V, H).to(torch.float16)
    shapes = [(E, I, H), (E, I, H), (E, H, I)]
    rms = lambda v: v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + c.rms_norm_eps)
    pos = torch.tensor(lengths, device="cuda")[:, None] + torch.arange(T, device="cuda")
    half = torch.arange(hd // 2, device="cuda", dtype=torch.float64)
    ang = (pos[..., None] * c.rope_theta ** (-2.0 * half / hd))[:, None]                 # [B, 1, T, hd / 2]
    cos, sin = torch.cat([ang.cos()] * 2, -1), torch.cat([ang.sin()] * 2, -1)
    rope = lambda v: v * cos + torch.cat([-v[..., hd // 2:], v[..., :hd // 2]], -1) * sin
    heads = lambda v: v.view(B, T, nh, hd).transpose(1, 2)
    x = embed[ids].double()
    ks, vs = [], []
    for l in range(NL):
        wq, wk, wv, wo = (rnd(H, H).to(torch.float16).double() for _ in range(4))
        router = rnd(H, E).double()
        banks = [moe.q4k_quantize_device(rnd(*shape)) for shape in shapes]
        h = rms(x)
        q, k, v = rope(heads(rms(h @ wq.T))), rope(heads(rms(h @ wk.T))), heads(h @ wv.T)
        out = torch.empty_like(q)
        for b in range(B):
            kb, vb = k[b], v[b]
            if decode:
                kb = torch.cat([kc[l, b, :, :lengths[b]].double(), kb], 1)
                vb = torch.cat([vc[l, b, :, :lengths[b]].double(), vb], 1)
            score = q[b] @ kb.transpose(1, 2) / math.sqrt(hd)
            late = torch.arange(kb.shape[1], device="cuda")[None, :] > pos[b][:, None]
            out[b] = torch.softmax(score.masked_fill(late, -math.inf), -1) @ vb
        x = x + out.transpose(1, 2).reshape(B, T, H) @ wo.T
        moe_in = rms(x).reshape(B * T, H)
        x = x + _moe64(moe_in, router, 0.0, banks, shapes, c.num_experts_per_tok, c.norm_topk_prob).view(B, T, H)
        if not decode:
            ks.append(k.float())
            vs.append(v.float())
    logits = rms(x[:, -1]) @ lm_head.double().T
    return logits if decode else (logits, torch.stack(ks), torch.stack(vs))


def exact(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["kind"] in ("layer", "host"):
        ys = _exact_layers(case, gen)
        return [y.cpu().numpy() for y in ys] if case["kind"] == "host" else ys
    return _exact_model(case, gen, seed)


def tolerance(case):
    # About four times what was measured (relative 2-norm).  Layers against the same layer in 64 bits from the
    # dequantised weights: 8.5e-4 for packed experts (16-bit intermediate and sub-block sums), 5e-4 for f16, 2.9e-3
    # for bf16, 1.4e-6 for f32.  The decode step against the library trunk: 9.7e-4.  A prompt fed in two pieces
    # instead of one: 3.2e-3 on the logits, where roundings move a few near-tied expert choices.
    if case["kind"] in ("layer", "host"):
        return {"rel": {"q4_k": 3e-3, "f16": 3e-3, "bf16": 1.2e-2, "f32": 6e-6}[case["dtype"]]}
    return {"rel": 4e-3 if case["kind"] == "decode" else 1.2e-2}
