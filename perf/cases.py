"""What is timed: the work that users of this package have it do, through its public entry points.

Kinds of case (`kind`):

* ``stack``      one decode token through a stack of MoE blocks, replayed from a CUDA graph (`DecodeStackGraph`): the
                 decode loop at concurrency one, at the full width and at the width that one of several
                 tensor-parallel ranks holds;
* ``block``      one MoE block (`FusedMoE.forward`), eager: router, routed and shared experts, from a single token over a
                 small decode batch to a whole prompt;
* ``experts``    the routed experts alone (`ResidentExperts.forward`), eager, for engines that keep their own router and
                 shared experts: packed NVFP4 banks or unquantised BF16 ones;
* ``attention``  the decode attention core with the cache update (`kernels.decode_attention`), eager: a sliding window or
                 a long full cache;
* ``layer``      one decoder layer (`DecodeLayer`) at decode, replayed from a CUDA graph;
* ``model``      a decode step of a whole small model (`DecodeModel`), token ids to logits, replayed from a CUDA graph.

Weights are random bytes and normals of the values that quantised normal weights have: E2M1 codes about uniform over
their sixteen values, E4M3 block scales where a block's largest of sixteen normals puts them. Which experts a token
takes is decided by a clear margin, as a trained router decides it: with random logits the last chosen and the first
rejected score often share a BF16 value, and then another order of the sums, equally right, picks another expert.
"""
import math
from types import SimpleNamespace

import torch

import inkling_b200 as ib

BF16 = torch.bfloat16
TAPS = 4          # taps of the short convolutions
D_REL = 16        # channels of the relative states
ROUTE_SCALE = 8.0


def listed():
    full = dict(hidden=4096, width=2048, experts=256, shared=2, top_k=6)
    return [
        # the decode loop at concurrency one: eight of the model's blocks at full width
        dict(name="stack_8_full", kind="stack", layers=8, **full),
        # the same loop on one of eight tensor-parallel ranks: all forty blocks, an eighth of their width
        dict(name="stack_40_eighth", kind="stack", layers=40, **dict(full, width=256)),
        # the smallest call: one token through one small block
        dict(name="block_small_1", kind="block", tokens=1, hidden=1024, width=512, experts=32, shared=2, top_k=4),
        # a decode batch of four sequences through one block
        dict(name="block_4", kind="block", tokens=4, **full),
        # a long prompt through one block, of a ragged length
        dict(name="block_prompt_1999", kind="block", tokens=1999, **full),
        # a decode batch of 61 sequences on the routed experts, popularity of the experts skewed as in served traffic
        dict(name="experts_61", kind="experts", tokens=61, quantized=True, skew=1.1, **full),
        # a prompt on the routed experts
        dict(name="experts_prompt_1024", kind="experts", tokens=1024, quantized=True, skew=0.6, **full),
        # a layer whose experts were left unquantised, five sequences
        dict(name="experts_bf16_5", kind="experts", tokens=5, quantized=False, skew=1.1, **full),
        # one token against a full sliding window
        dict(name="attention_window", kind="attention", batch=1, heads=64, kv_heads=16, head_dim=128, slots=512, window=512,
             extent=512, position=5000, padded=False),
        # eight sequences deep into a long context, padded on the left to different lengths
        dict(name="attention_long", kind="attention", batch=8, heads=64, kv_heads=8, head_dim=128, slots=32768, window=0,
             extent=1024, position=30001, padded=True),
        # a sparse full-attention layer for seven sequences
        dict(name="layer_7", kind="layer", batch=7, heads=64, kv_heads=8, head_dim=128, slots=4096, window=0, extent=1024,
             position=3000, **full),
        # one token through a model of six layers: a dense one, four sliding sparse ones, a full-attention sparse one
        dict(name="model_1", kind="model", layers=6, heads=64, kv_heads=8, head_dim=128, slots=4096, position=3000, dense=8192,
             vocab=32768, **full),
    ]


def _log_uniform(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(("stack", "block", "block", "experts", "experts", "attention", "attention", "layer", "model"))
    if kind == "stack":
        hidden, width = rng.choice(((4096, 2048), (4096, 1024), (4096, 512), (4096, 256), (2048, 256), (1024, 512)))
        most = min(40, 8 * 2048 * 4096 // (width * hidden))
        return dict(kind=kind, layers=_log_uniform(rng, 1, most), hidden=hidden, width=width, experts=rng.choice((64, 128, 256)),
                    shared=rng.choice((1, 2)), top_k=rng.choice((4, 6, 8)))
    if kind == "block":
        hidden, width = rng.choice(((4096, 2048), (4096, 1024), (4096, 512), (2048, 1024), (1024, 512)))
        return dict(kind=kind, tokens=_log_uniform(rng, 1, 1999), hidden=hidden, width=width, experts=rng.choice((64, 128, 256)),
                    shared=2, top_k=rng.choice((4, 6)))
    if kind == "experts":
        quantized = rng.random() < 0.7
        hidden, width = rng.choice(((4096, 2048), (4096, 1024), (2048, 1024), (1024, 512)))
        return dict(kind=kind, tokens=_log_uniform(rng, 1, 1999 if quantized else 64), quantized=quantized,
                    skew=round(rng.uniform(0.0, 1.5), 2), hidden=hidden, width=width, experts=rng.choice((64, 128, 256)),
                    shared=0, top_k=rng.choice((4, 6, 8)))
    if kind == "attention":
        heads = rng.choice((16, 32, 64))
        window = rng.choice((0, 0, 128, 512))
        batch = _log_uniform(rng, 1, 8)
        slots = window or _log_uniform(rng, 300, 32768)
        return dict(kind=kind, batch=batch, heads=heads, kv_heads=heads // rng.choice((1, 4, 8)) if slots <= 4096 else heads // 8,
                    head_dim=rng.choice((64, 128, 128, 256)) if slots <= 8192 else 128, slots=slots, window=window,
                    extent=window or min(slots, 1024), position=rng.randrange(window or slots // 2, 20000 if window else slots),
                    padded=rng.random() < 0.5)
    window = rng.choice((0, 512))
    slots = window or rng.choice((1024, 4096))
    shape = dict(hidden=4096, width=rng.choice((2048, 1024, 512)), experts=rng.choice((64, 128)), shared=2, top_k=6)
    if kind == "layer":
        return dict(kind=kind, batch=rng.randint(1, 8), heads=64, kv_heads=16 if window else 8, head_dim=128, slots=slots, window=window,
                    extent=window or 1024, position=rng.randrange(512, 20000 if window else slots), **shape)
    return dict(kind=kind, layers=rng.randint(2, 5), heads=64, kv_heads=8, head_dim=128, slots=4096, position=rng.randrange(512, 4096),
                dense=rng.choice((4096, 8192)), vocab=rng.choice((8192, 16384, 32768)), **shape)


# ------------------------------------------------------------------ weights


class _Source:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.device = torch.device("cuda", 0)
        self.gen = torch.Generator(device=self.device).manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=BF16):
        return torch.empty(*shape, dtype=dtype, device=self.device).normal_(0.0, std, generator=self.gen)

    def uniform(self, *shape, low=0.0, high=1.0):
        return torch.empty(*shape, dtype=torch.float32, device=self.device).uniform_(low, high, generator=self.gen)

    def bytes(self, out, low, high):
        out.random_(low, high, generator=self.gen)


def _nvfp4_banks(src, case):
    """Every expert's packed banks, one allocation per kind."""
    banks = ib.ExpertBanks(case["experts"], case["hidden"], case["width"], src.device)
    for codes in (banks.gate_up_proj, banks.down_proj):
        src.bytes(codes, 0, 256)
    for scales in (banks.gate_up_proj_scale, banks.down_proj_scale):
        src.bytes(scales, 0x6A, 0x77)   # E4M3 80 .. 224
    for scale2 in (banks.gate_up_proj_scale2, banks.down_proj_scale2):
        scale2.copy_(src.uniform(case["experts"], low=3.5e-5, high=4.5e-5))
    return banks


def _experts(src, case, quantized=True):
    if quantized:
        weights = _nvfp4_banks(src, case).weights
    else:
        gate_up = src.normal(case["experts"], 2 * case["width"], case["hidden"], std=0.02)
        down = src.normal(case["experts"], case["hidden"], case["width"], std=0.02)
        weights = {e: dict(gate_up_proj=gate_up[e], down_proj=down[e]) for e in range(case["experts"])}
    return ib.ResidentExperts(case["hidden"], case["width"], None, weights, quantized)


def _moe(src, case, favoured):
    """A block and the direction that all its router's rows share. `favoured`: the correction bias decides for the same
    experts at every token (in a stack, where no token is made for each block); else the tokens decide (`_routed_tokens`)."""
    d, f, experts, shared = case["hidden"], case["width"], case["experts"], case["shared"]
    router = src.normal(experts + shared, d, std=1.28 / math.sqrt(d), dtype=torch.float32)
    common = src.normal(d, dtype=torch.float32)
    common /= common.norm()
    router[:experts] -= 4.0 / math.sqrt(d) * 4.0 * common   # most experts score low on most tokens
    bias = src.normal(experts, std=0.01, dtype=torch.float32)
    if favoured:
        bias[torch.randperm(experts, generator=src.gen, device=src.device)[: case["top_k"]]] += 1.0
    block = ib.FusedMoE(router.to(BF16), bias, torch.ones(1, dtype=BF16, device=src.device), ROUTE_SCALE, case["top_k"],
                        src.normal(shared, f, d, std=0.02), src.normal(shared, f, d, std=0.02), src.normal(shared, d, f, std=0.02),
                        _experts(src, case))
    return block, common


def _routed_tokens(src, block, common, tokens, case):
    """Normal activations that lean towards the router rows of `top_k` experts each, as hidden states that were trained
    with their router do."""
    chosen = _choices(src, tokens, case, skew=0.6)
    rows = block.router_weight.float()[: case["experts"]]
    own = rows + 16.0 / math.sqrt(case["hidden"]) * common
    x = src.normal(tokens, case["hidden"], dtype=torch.float32) + 0.25 * math.sqrt(case["hidden"]) * common
    return (x + 5.0 * own[chosen].sum(1)).to(BF16)


def _choices(src, tokens, case, skew):
    """`top_k` different experts per token, popularity falling as rank ** -skew over a random order of the experts."""
    rank = torch.randperm(case["experts"], generator=src.gen, device=src.device) + 1
    p = rank.float() ** -skew
    return torch.multinomial(p.expand(tokens, -1), case["top_k"], replacement=False, generator=src.gen)


def _attention(src, case, index, window, extent, full):
    h, hk, c, d = case["heads"], case["kv_heads"], case["head_dim"], case["hidden"]
    return ib.DecodeAttention(src.normal((h + 2 * hk) * c + h * D_REL, d, std=1 / math.sqrt(d)), src.normal(d, h * c, std=1 / math.sqrt(h * c)),
                              1 + src.normal(c, std=0.1), 1 + src.normal(c, std=0.1), src.normal(hk * c, 1, TAPS, std=0.2, dtype=torch.float32),
                              src.normal(hk * c, 1, TAPS, std=0.2, dtype=torch.float32), src.normal(D_REL, extent, std=0.3),
                              layer_idx=index, heads=h, kv_heads=hk, head_dim=c, d_rel=D_REL, window=window,
                              log_scaling_n_floor=1024 if full else None)


def _layer(src, case, index, block, window, extent, full):
    d = case["hidden"]
    ones = torch.ones(d, dtype=BF16, device=src.device)
    return ib.DecodeLayer(_attention(src, case, index, window, extent, full), block, ones, ones, src.normal(d, 1, TAPS, std=0.1, dtype=torch.float32),
                          src.normal(d, 1, TAPS, std=0.1, dtype=torch.float32))


def _layer_cache(src, case, batch, slots):
    hk, c, d = case["kv_heads"], case["head_dim"], case["hidden"]
    return SimpleNamespace(k_cache=src.normal(batch, hk, slots, c), v_cache=src.normal(batch, hk, slots, c),
                           conv_caches=[SimpleNamespace(cache=src.normal(batch, n, TAPS, dtype=torch.float32)) for n in (hk * c, hk * c, d, d)])


def _pads(src, batch, position, padded):
    """Tokens of left padding per sequence: none, or up to a quarter of the context."""
    if not padded:
        return torch.zeros(batch, dtype=torch.int64, device=src.device)
    return (src.uniform(batch) * 0.25 * position).to(torch.int64)


def _captured(step):
    """A step as an engine captures it: three warm-up passes on a side stream, then one graph."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side), torch.inference_mode():
        for _ in range(3):
            step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side), torch.inference_mode():
        out = step()
    torch.cuda.synchronize()
    return graph, out


# ------------------------------------------------------------------ the contract


def prepare(case, seed):
    src = _Source(seed)
    s = SimpleNamespace(kind=case["kind"])
    with torch.no_grad():
        _PREPARE[case["kind"]](s, src, case)
    return s


def _prepare_stack(s, src, case):
    stack = ib.MoEStack([_moe(src, case, favoured=True)[0] for _ in range(case["layers"])], case["hidden"])
    s.runner = ib.DecodeStackGraph(stack, src.normal(1, case["hidden"]))
    s.token = src.normal(1, case["hidden"])


def _prepare_block(s, src, case):
    s.block, common = _moe(src, case, favoured=False)
    s.x = _routed_tokens(src, s.block, common, case["tokens"], case).unsqueeze(0)
    s.block(s.x)   # a serving program warms its blocks up before the first request


def _prepare_experts(s, src, case):
    s.experts = _experts(src, case, case["quantized"])
    s.x = src.normal(case["tokens"], case["hidden"])
    s.indices = _choices(src, case["tokens"], case, case["skew"])
    s.weights = (src.uniform(case["tokens"], case["top_k"], low=0.2, high=1.8)).to(BF16)
    s.experts(s.x, s.indices, s.weights)


def _prepare_attention(s, src, case):
    b, h, hk, c = case["batch"], case["heads"], case["kv_heads"], case["head_dim"]
    s.q, s.r = src.normal(b, h, 1, c), src.normal(b, 1, h, D_REL)
    s.proj = src.normal(D_REL, case["extent"], std=0.3)
    s.k, s.v = src.normal(b, hk, case["slots"], c), src.normal(b, hk, case["slots"], c)
    s.new_k, s.new_v = src.normal(b, hk, 1, c), src.normal(b, hk, 1, c)
    s.position = torch.tensor(case["position"], dtype=torch.int64, device=src.device)
    s.pads = _pads(src, b, case["position"], case["padded"])
    s.options = dict(window=case["window"], log_scaling_n_floor=None if case["window"] else 1024, scale=1.0 / math.sqrt(c))


def _prepare_layer(s, src, case):
    batch = case["batch"]
    block, common = _moe(src, case, favoured=False)
    layer = _layer(src, case, 0, block, case["window"], case["extent"], not case["window"])
    hidden = _routed_tokens(src, block, common, batch, case).unsqueeze(1)
    s.caches = [_layer_cache(src, case, batch, case["slots"])]
    cache = SimpleNamespace(layers=s.caches, position=torch.tensor(case["position"], dtype=torch.int64, device=src.device),
                            pad_counts=_pads(src, batch, case["position"], True))
    s.keep = (layer, hidden, cache)
    s.graph, s.out = _captured(lambda: layer(hidden, cache))


def _prepare_model(s, src, case):
    """The last layer is a full-attention one, the others slide; the first is dense, the others sparse."""
    d, layers, window = case["hidden"], [], 512
    s.caches = []
    for i in range(case["layers"]):
        full = i == case["layers"] - 1
        if i == 0:
            f = case["dense"]
            block = ib.DenseMLP(src.normal(f, d, std=0.02), src.normal(f, d, std=0.02), src.normal(d, f, std=0.02), torch.ones(1, dtype=BF16, device=src.device))
        else:
            block = _moe(src, case, favoured=True)[0]
        layers.append(_layer(src, case, i, block, 0 if full else window, 1024 if full else window, full))
        s.caches.append(_layer_cache(src, case, 1, case["slots"] if full else window))
    ones = torch.ones(d, dtype=BF16, device=src.device)
    model = ib.DecodeModel(src.normal(case["vocab"], d), ones, layers, ones, src.normal(case["vocab"], d, std=0.02), 4.0)
    ids = torch.randint(case["vocab"], (1, 1), generator=src.gen, device=src.device)
    s.start = torch.tensor(case["position"], dtype=torch.int64, device=src.device)
    s.position = s.start.clone()
    cache = SimpleNamespace(layers=s.caches, position=s.position, pad_counts=torch.zeros(1, dtype=torch.int64, device=src.device))
    s.keep = (model, ids, cache)

    def step():
        s.position.copy_(s.start)   # every pass decodes the same position: the caches of a long run would fill up
        return model(ids, cache)

    s.graph, s.out = _captured(step)


_PREPARE = dict(stack=_prepare_stack, block=_prepare_block, experts=_prepare_experts, attention=_prepare_attention,
                layer=_prepare_layer, model=_prepare_model)


def _updated(caches):
    return [[c.k_cache, c.v_cache] + [h.cache for h in c.conv_caches] for c in caches]


def run(state):
    s = state
    with torch.no_grad():
        if s.kind == "stack":
            s.runner.token_in.copy_(s.token)
            return s.runner.replay()
        if s.kind == "block":
            return s.block(s.x)
        if s.kind == "experts":
            return s.experts(s.x, s.indices, s.weights)
        if s.kind == "attention":
            out = ib.kernels.decode_attention(s.q, s.r, s.proj, s.k, s.v, s.position, s.pads, new_key=s.new_k, new_value=s.new_v, **s.options)
            return [out, s.k, s.v]
        s.graph.replay()
        return [s.out, _updated(s.caches)]


def _distinct(case, tokens, skew):
    """Expected number of different experts among the tokens' choices."""
    p = [(i + 1.0) ** -skew for i in range(case["experts"])]
    total = sum(p)
    return sum(1.0 - (1.0 - min(1.0, case["top_k"] * v / total)) ** tokens for v in p)


def _work_experts(case, tokens, skew, quantized=True):
    d, f = case["hidden"], case["width"]
    per_expert = 3 * d * f * (0.5 + 1 / 16 if quantized else 2.0)
    return _distinct(case, tokens, skew) * per_expert + 2 * 2 * tokens * d, 6.0 * tokens * case["top_k"] * d * f


def _work_block(case, tokens, skew):
    d, f = case["hidden"], case["width"]
    nbytes, flops = _work_experts(case, tokens, skew)
    rows = case["experts"] + case["shared"]
    return nbytes + 2 * rows * d + 2 * 3 * case["shared"] * d * f, flops + 6.0 * tokens * case["shared"] * d * f + 2.0 * tokens * rows * d


def _work_attention(batch, heads, kv_heads, head_dim, used, extent):
    nbytes = batch * (2 * 2 * kv_heads * head_dim * used + 2 * 2 * heads * head_dim) + 2 * D_REL * min(extent, used)
    return nbytes, batch * heads * (4.0 * head_dim * used + 2.0 * D_REL * min(extent, used))


def _work_layer(case, batch, window, extent, pad_share):
    h, hk, c, d = case["heads"], case["kv_heads"], case["head_dim"], case["hidden"]
    used = min(window or case["slots"], case["position"] + 1) if window else (case["position"] + 1) * (1 - pad_share)
    nbytes, flops = _work_attention(batch, h, hk, c, used, extent)
    weights = d * ((h + 2 * hk) * c + h * D_REL) + d * h * c
    history = batch * TAPS * (2 * hk * c + 2 * d) * 4 * 2
    return nbytes + 2 * weights + history + 4 * TAPS * (2 * hk * c + 2 * d), flops + 2.0 * batch * weights


def work(case):
    kind = case["kind"]
    if kind == "stack":
        nbytes, flops = (v * case["layers"] for v in _work_block(case, 1, 0.0))
    elif kind == "block":
        nbytes, flops = _work_block(case, case["tokens"], 0.6)
    elif kind == "experts":
        nbytes, flops = _work_experts(case, case["tokens"], case["skew"], case["quantized"])
    elif kind == "attention":
        used = case["window"] or (case["position"] + 1) * (1 - (0.125 if case["padded"] else 0))
        nbytes, flops = _work_attention(case["batch"], case["heads"], case["kv_heads"], case["head_dim"], used, case["extent"])
    elif kind == "layer":
        a = _work_layer(case, case["batch"], case["window"], case["extent"], 0.125)
        b = _work_block(case, case["batch"], 0.6)
        nbytes, flops = a[0] + b[0], a[1] + b[1]
    else:
        d = case["hidden"]
        nbytes, flops = 2.0 * d * case["vocab"] + 2.0 * 3 * d * case["dense"], 2.0 * d * case["vocab"] + 6.0 * d * case["dense"]
        for i in range(case["layers"]):
            full = i == case["layers"] - 1
            a = _work_layer(case, 1, 0 if full else 512, 1024 if full else 512, 0.0)
            b = _work_block(case, 1, 0.0) if i else (0, 0)
            nbytes, flops = nbytes + a[0] + b[0], flops + a[1] + b[1]
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """BF16 inputs, intermediates and results; products of four-bit weights summed in FP16 and FP32."""
    return {"rel": 1e-2}
