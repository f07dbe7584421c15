"""Several tokens at once: the grouped kernel behind FusedMoE and ResidentExperts, the router and the plan, at the sizes where
their tiles end."""
import pytest
import torch

import cases
from helpers import BF16, layer_on_device, max_rel
from oracle import moe as oracle_moe

pytestmark = pytest.mark.gpu
TOL = 2e-2   # of the largest magnitude, the bar of the other expert kernels: FP16 / digit operands, BF16 intermediates


@pytest.fixture(scope="module")
def ib():
    import inkling_b200

    return inkling_b200


@pytest.fixture(scope="module")
def device():
    return torch.device("cuda", 0)


def one_allocation_per_kind(banks, device):
    """Banks the way a loader lays them out: one tensor per kind, the experts views into it."""
    stacked = {n: torch.stack([banks[e][n].reshape(1).float() if n.endswith("scale2") else banks[e][n] for e in sorted(banks)]).to(device)
               for n in banks[0]}
    return {e: {n: t[e] for n, t in stacked.items()} for e in banks}


@pytest.mark.parametrize("d,f,experts,tokens", [
    (1024, 512, 32, 2), (1024, 512, 32, 15), (1024, 512, 32, 17), (1024, 512, 32, 65),   # tiles of 16 and 64 tokens
    (512, 256, 16, 70), (512, 768, 4, 31),                                                # of 32 and 128; an odd number of chunks
    (512, 256, 4, 33), (512, 256, 4, 129), (512, 256, 4, 300),                            # of 64 and 256: one or both accumulators
    (256, 256, 16, 9),                                                                    # a single chunk
])
def test_a_block_of_several_tokens(ib, device, d, f, experts, tokens):
    p, banks, x = cases.make_layer(d, f, experts, 2, 3, tokens, seed=tokens, bias="randn")
    dp = layer_on_device(p, device)
    module = ib.ResidentExperts(d, f, None, one_allocation_per_kind(banks, device))
    assert module.bank_maps is not None
    layer = ib.FusedMoE(dp["router_weight"], dp["router_bias"], dp["global_scale"], p["route_scale"], p["top_k"],
                        dp["shared_gate"], dp["shared_up"], dp["shared_down"], module, None)
    for _ in range(2):
        got = layer(x.to(device).unsqueeze(0))[0].float().cpu()
    module.check_status()
    idx, w, gam = layer.topk_indices[:tokens].cpu(), layer.topk_weights[:tokens].cpu(), layer.gammas[:tokens].cpu()
    assert max_rel(got, oracle_moe.moe_layer_fp32(x, p, banks, idx, w, gam)) <= TOL
    alone = module(x.to(device), idx.to(device), w.to(device)).float().cpu()
    assert max_rel(alone, oracle_moe.routed_experts_fp32(x, idx, w, banks)) <= TOL


@pytest.mark.parametrize("d,f,experts,tokens", [(256, 128, 8, 2), (256, 128, 8, 70), (384, 128, 2, 131), (256, 128, 2, 300), (512, 256, 5, 17)])
def test_unquantised_banks_of_several_tokens(ib, device, d, f, experts, tokens):
    gen = torch.Generator().manual_seed(tokens)
    banks = {e: dict(gate_up_proj=(torch.randn(2 * f, d, generator=gen) * 0.05).to(BF16), down_proj=(torch.randn(d, f, generator=gen) * 0.05).to(BF16))
             for e in range(experts)}
    x = torch.randn(tokens, d, generator=gen).to(BF16)
    idx = torch.stack([torch.randperm(experts, generator=gen)[:2] for _ in range(tokens)])
    w = torch.rand(tokens, 2, generator=gen).to(BF16)
    module = ib.ResidentExperts(d, f, None, one_allocation_per_kind(banks, device), quantized=False)
    assert module.bank_maps is not None
    got = module(x.to(device), idx.to(device), w.to(device)).float().cpu()
    module.check_status()
    assert max_rel(got, oracle_moe.routed_experts_bf16_fp32(x, idx, w, banks)) <= TOL


@pytest.mark.parametrize("d,f,experts,tokens", [
    (256, 2048, 100, 100), (256, 2048, 100, 500),   # one ring stage an item, more deals than blocks, more items a deal than the queue holds
    (512, 1024, 60, 290),                            # deals that end inside an expert; gate/up and down of different lengths
    (4096, 128, 3, 5), (256, 256, 1, 2),             # one item a deal; fewer items than blocks
    (1024, 512, 40, 13), (1024, 512, 40, 60), (512, 512, 64, 700),   # first deals of one, of some and of most items; later ones of one and of several
])
def test_every_item_is_dealt_whatever_their_number(ib, device, d, f, experts, tokens):
    if f % 256:   # (packed banks need a multiple of 256 columns: BF16 ones)
        gen = torch.Generator().manual_seed(tokens)
        banks = {e: dict(gate_up_proj=(torch.randn(2 * f, d, generator=gen) * 0.05).to(BF16), down_proj=(torch.randn(d, f, generator=gen) * 0.05).to(BF16))
                 for e in range(experts)}
        x = torch.randn(tokens, d, generator=gen).to(BF16)
        want = oracle_moe.routed_experts_bf16_fp32
    else:
        _, banks, x = cases.make_layer(d, f, experts, 1, 1, tokens, seed=tokens, bias="randn")
        gen, want = torch.Generator().manual_seed(tokens), oracle_moe.routed_experts_fp32
    k = min(3, experts)
    idx = torch.stack([torch.randperm(experts, generator=gen)[:k] for _ in range(tokens)])
    w = torch.rand(tokens, k, generator=gen).to(BF16)
    module = ib.ResidentExperts(d, f, None, one_allocation_per_kind(banks, device), quantized=f % 256 == 0)
    assert module.bank_maps is not None
    for _ in range(2):   # (the counter starts over)
        got = module(x.to(device), idx.to(device), w.to(device)).float().cpu()
        module.check_status()
        assert max_rel(got, want(x, idx, w, banks)) <= TOL


def test_experts_that_are_not_there_are_skipped_and_reported(ib, device):
    """A rank that holds the experts 2..5 of 8: routes to the others add nothing; an id beyond the table sets the status."""
    d, f, tokens = 512, 256, 20
    p, banks, x = cases.make_layer(d, f, 8, 2, 3, tokens, seed=6, bias="randn")
    mine = {e: b for e, b in one_allocation_per_kind(banks, device).items() if 2 <= e <= 5}
    module = ib.ResidentExperts(d, f, None, mine)
    gen = torch.Generator().manual_seed(1)
    idx = torch.stack([torch.randperm(6, generator=gen)[:3] for _ in range(tokens)])
    w = torch.rand(tokens, 3, generator=gen).to(BF16)
    got = module(x.to(device), idx.to(device), w.to(device)).float().cpu()
    module.check_status()
    assert max_rel(got, oracle_moe.routed_experts_fp32(x, idx, w, {e: banks[e] for e in mine})) <= TOL
    idx[3, 1] = 7
    module(x.to(device), idx.to(device), w.to(device))
    with pytest.raises(RuntimeError, match="outside"):
        module.check_status()


@pytest.mark.parametrize("hidden,routed,shared,top_k,tokens", [(4096, 256, 2, 6, 17), (1024, 61, 1, 4, 33), (264, 300, 0, 8, 9), (8, 8, 2, 8, 100),
                                                               (2056, 256, 2, 6, 333), (4096, 256, 2, 6, 1999), (520, 40, 1, 4, 5000)])   # several tiles a block
def test_a_token_is_routed_the_same_in_any_company(ib, device, hidden, routed, shared, top_k, tokens):
    """Bit-exact: the many-token router against the one-launch router on the same tokens in groups of at most eight."""
    gen = torch.Generator().manual_seed(hidden)
    weight = (torch.randn(routed + shared, hidden, generator=gen) * 1.3 / hidden ** 0.5).to(BF16).to(device)
    bias = (torch.randn(routed, generator=gen) * 0.05).to(device)
    scale = torch.full((1,), 1.25).to(BF16).to(device)
    x = torch.randn(tokens, hidden, generator=gen).to(BF16).to(device)

    def route(x):
        t = x.shape[0]
        out = (torch.empty(t, top_k, dtype=BF16, device=device), torch.empty(t, top_k, dtype=torch.int64, device=device),
               torch.empty(t, shared, dtype=BF16, device=device))
        logits = torch.empty(t, routed, dtype=BF16, device=device)
        ib.kernels.router_forward(x, weight, bias, scale, 8.0, top_k, shared, *out, ib.kernels.router_workspace(t, routed + shared, device),
                                  routed_logits=logits)
        return (*out, logits)

    whole = route(x)
    parts = [route(x[i:i + 8]) for i in range(0, tokens, 8)]
    for i, got in enumerate(whole):
        assert torch.equal(got, torch.cat([p[i] for p in parts]))


@pytest.mark.parametrize("local,start,routes", [(256, 0, 1), (3, 5, 31), (256, 0, 33), (40, 100, 1025), (257, 3, 5000), (2000, 0, 20000)])
def test_the_plan_is_a_stable_sort_at_any_size(ib, device, local, start, routes):
    gen = torch.Generator().manual_seed(routes)
    idx = torch.randint(0, start + local + 2, (routes,), generator=gen)   # some on other ranks
    sources = torch.randint(1, 1 << 40, (local, 2), generator=gen)
    i32 = dict(dtype=torch.int32, device=device)
    pointers = torch.zeros((start + local) * 2, dtype=torch.int64, device=device)
    experts, counts, rows = torch.empty(local, **i32), torch.empty(local, **i32), torch.full((local, routes), -1, **i32)
    ib.kernels.expert_plan[(1,)](idx.to(device), sources.to(device), None, None, None, None, None, torch.empty(0, **i32), pointers, experts,
                                 counts, rows, start, local, 0, 2, routes, routes)
    want = oracle_moe.expert_plan(idx.view(-1, 1), sources, start, local, 2, routes)
    for got, name in ((experts, "experts"), (counts, "counts"), (rows, "rows")):
        assert torch.equal(got.cpu(), torch.as_tensor(want[name]).to(torch.int32)), name
    assert torch.equal(pointers.cpu(), torch.as_tensor(want["pointers"]))


def _block(ib, device, tokens, seed=5, d=256, f=256, experts=8):
    p, banks, x = cases.make_layer(d, f, experts, 2, 3, tokens, seed=seed, bias="randn")
    dp = layer_on_device(p, device)
    return ib.FusedMoE(dp["router_weight"], dp["router_bias"], dp["global_scale"], p["route_scale"], p["top_k"], dp["shared_gate"],
                       dp["shared_up"], dp["shared_down"], ib.ResidentExperts(d, f, None, one_allocation_per_kind(banks, device)), None), x.to(device)


def test_more_tokens_than_are_planned_at_a_time(ib, device):
    """A call of 32 768 tokens and a rest: the rest comes out as in a call of its own. Tokens do not mix, so only the order
    of FP32 sums could differ, if at all: one rounding of the BF16 result."""
    layer, x = _block(ib, device, 64)
    many = x.repeat(32768 // 64 + 1, 1)[:32768 + 37].contiguous()
    whole = layer(many)
    idx, w = layer.topk_indices[:len(many)].clone(), layer.topk_weights[:len(many)].clone()
    rest = layer(many[32768:])
    assert max_rel(whole[32768:].float().cpu(), rest.float().cpu()) <= 2 ** -8
    assert max_rel(whole[:64].float().cpu(), layer(x).float().cpu()) <= 2 ** -8
    routed = layer.experts(many, idx, w)
    assert max_rel(routed[32768:].float().cpu(), layer.experts(many[32768:], idx[32768:], w[32768:]).float().cpu()) <= 2 ** -8
    layer.experts.check_status()


@pytest.mark.parametrize("tokens", [1, 9])
def test_a_block_sees_weights_exchanged_underneath(ib, device, tokens):
    """`tensor.data = ...` keeps the tensor and changes its storage; a copy of the module makes its own record."""
    import copy

    d, f = (1024, 512)
    layer, x = _block(ib, device, tokens, d=d, f=f, experts=32)
    other, _ = _block(ib, device, tokens, seed=8, d=d, f=f, experts=32)
    first = layer(x).clone()
    other.experts = layer.experts
    want = other(x).clone()
    old = [getattr(layer, n).clone() for n in ("router_weight", "router_bias", "shared_gate", "shared_up", "shared_down")]
    keep = [getattr(layer, n).data for n in ("router_weight", "router_bias", "shared_gate", "shared_up", "shared_down")]
    twin = copy.deepcopy(layer)
    for n in ("router_weight", "router_bias", "shared_gate", "shared_up", "shared_down"):
        getattr(layer, n).data = getattr(other, n).clone()
    assert torch.equal(layer(x), want) and not torch.equal(first, want)
    assert torch.equal(twin(x), first)
    del old, keep


@pytest.mark.parametrize("tokens", [2, 12])
def test_a_first_call_may_be_one_under_capture(ib, device, tokens):
    layer, x = _block(ib, device, tokens)
    twin, _ = _block(ib, device, tokens)
    want = twin(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = layer(x)
    graph.replay()
    assert torch.equal(out, want)


@pytest.mark.parametrize("tokens", [2, 9, 70])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), -float("inf"), 2.0 ** 126])
def test_a_token_that_is_not_finite_stays_its_own(ib, device, tokens, value):
    """A NaN or an infinity in one token (or, with 2^126, in its gate/up result only) reaches all of its outputs: every row of
    the second projection has a non-zero weight for a non-finite input. The others keep their bits."""
    d, f = 512, 256
    p, banks, x = cases.make_layer(d, f, 8, 2, 3, tokens, seed=4, bias="randn")
    module = ib.ResidentExperts(d, f, None, one_allocation_per_kind(banks, device))
    gen = torch.Generator().manual_seed(2)
    idx = torch.stack([torch.randperm(8, generator=gen)[:3] for _ in range(tokens)]).to(device)
    w = (0.5 + torch.rand(tokens, 3, generator=gen)).to(BF16).to(device)
    x = x.to(device)
    clean = module(x, idx, w)
    bad = tokens // 2
    x[bad, 100:200:50] = value
    got = module(x, idx, w)
    assert not torch.isfinite(got[bad]).any()
    rest = [t for t in range(tokens) if t != bad]
    assert torch.equal(got[rest], clean[rest])
    block = ib.FusedMoE(p["router_weight"][:8].to(device).contiguous(), p["router_bias"].to(device), p["global_scale"].to(device), p["route_scale"], 3,
                        *(torch.empty(0, *s, dtype=BF16, device=device) for s in ((f, d), (f, d), (d, f))), module, None)
    assert not torch.isfinite(block(x)[bad]).any()


@pytest.mark.parametrize("tokens", [1, 2, 9])
@pytest.mark.parametrize("name,change", [
    ("router_weight", lambda t: t.float()), ("router_weight", lambda t: t.view(torch.float16)), ("router_weight", lambda t: t.t()),
    ("global_scale", lambda t: t.float()), ("shared_down", lambda t: t.transpose(1, 2)), ("shared_up", lambda t: t.view(torch.float16)),
])
def test_a_tensor_changed_underneath_is_checked_again(ib, device, tokens, name, change):
    """Another type, layout or storage after the first call, also at the same address: refused, and right again when taken back."""
    layer, x = _block(ib, device, tokens, d=1024, f=512, experts=8)
    want = layer(x).clone()
    was = getattr(layer, name).data
    getattr(layer, name).data = change(was)
    with pytest.raises(AssertionError):
        layer(x)
    getattr(layer, name).data = was
    assert torch.equal(layer(x), want)


def _fill_what_is_free(device):
    """Tensors that take whatever the allocator has got back, so that a write to it, or a read of what was there, shows."""
    return [torch.full((512 << k,), 127, dtype=torch.uint8, device=device) for k in range(15) for _ in range(24)]


def _capture(step):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        out = step()
    return graph, out


@pytest.mark.parametrize("tokens", [1, 4, 12])
def test_a_graph_outlives_a_larger_call(ib, device, tokens):
    """A step captured after an eager one; then a prompt through the same modules replaces their buffers."""
    layer, x = _block(ib, device, tokens, d=1024, f=512, experts=8)
    stack = ib.MoEStack([_block(ib, device, 1, seed=s, d=1024, f=512, experts=8)[0] for s in (6, 7)], 1024)
    decode = ib.DecodeStackGraph(stack, x[:1])
    alone = decode.replay().clone()
    idx, w = torch.arange(tokens * 3, device=device).view(tokens, 3) % 8, torch.ones(tokens, 3, dtype=BF16, device=device)

    def step():
        return layer(x), layer.experts(x, idx, w), layer.forward_partial(x)

    want = [t.clone() for t in step()]
    graph, out = _capture(step)
    prompt = x.repeat(-(-700 // tokens), 1)
    layer(prompt), layer.experts(prompt, idx.repeat(len(prompt) // tokens, 1), w.repeat(len(prompt) // tokens, 1))
    stack(prompt), stack.layers[-1](prompt)
    fill = _fill_what_is_free(device)
    for t in out:
        t.zero_()
    graph.replay()
    assert all(torch.equal(got, t) for got, t in zip(out, want))
    decode.out.zero_()
    assert torch.equal(decode.replay(), alone)
    assert all(bool((t == 127).all()) for t in fill)


@pytest.mark.parametrize("tokens", [2, 8, 12])
def test_buffers_made_under_capture_are_the_graphs_alone(ib, device, tokens):
    """First calls under capture; then an eager call and the second graph, both before the first graph's first replay (which is
    what clears the router's counters in its buffers)."""
    layer, x = _block(ib, device, tokens)
    want = _block(ib, device, tokens)[0](x)
    fill = _fill_what_is_free(device)
    del fill
    graphs = [_capture(lambda: (layer(x), layer(x))) for _ in range(2)]
    assert torch.equal(layer(x), want)
    for graph, out in reversed(graphs):
        graph.replay()
        assert torch.equal(out[0], want) and torch.equal(out[1], want)
    assert torch.equal(layer(x), want)


@pytest.mark.parametrize("kind", ["heads", "rows"])
def test_the_zeros_of_a_norm_under_capture(ib, device, kind):
    """The norm's zero rows, used by a graph and replaced by a larger call; first made under capture, then needed eagerly."""
    draw = lambda *shape: torch.randn(*shape, device=device).to(BF16)  # noqa: E731
    taps = torch.zeros(128, 1, 4, device=device)

    def make():
        attention = ib.DecodeAttention(draw(640, 128), draw(128, 256), draw(64), draw(64), taps, taps, draw(16, 8), layer_idx=0, heads=4, kv_heads=2,
                                       head_dim=64, d_rel=32)
        return attention if kind == "heads" else ib.DecodeLayer(attention, None, draw(64), draw(64), taps, taps)

    x, weight = draw(5, 64), draw(64)
    want = make()._norm(x.clone(), weight)
    module = make()
    module._norm(x.clone(), weight)
    graph, out = _capture(lambda: module._norm(x, weight))
    module._norm(draw(3000, 64), weight)
    fill = _fill_what_is_free(device)
    graph.replay()
    assert torch.equal(out, want)
    del fill
    module = make()
    graph, out = _capture(lambda: module._norm(x, weight))
    assert torch.equal(module._norm(x.clone(), weight), want)
    graph.replay()
    assert torch.equal(out, want)


def test_experts_put_in_place_of_others_get_the_room_they_need(ib, device):
    """A block that has seen 40 tokens is given experts that have seen two (room for eight routes)."""
    layer, x = _block(ib, device, 40)
    want = layer(x).clone()
    fresh = _block(ib, device, 2)[0].experts
    fresh(x[:2], layer.topk_indices[:2], layer.topk_weights[:2])
    assert fresh.capacity == 8
    layer.experts = fresh
    assert torch.equal(layer(x), want)


@pytest.mark.parametrize("tokens", [1, 9])
def test_errors_of_the_native_calls_keep_their_types(ib, device, tokens):
    layer, x = _block(ib, device, tokens, d=1024, f=512, experts=8)
    idx, w = torch.zeros(tokens, 3, dtype=torch.int64, device=device), torch.ones(tokens, 3, dtype=BF16, device=device)
    for wrong in (x.float(), x[:, :-8], x.cpu().float()):
        with pytest.raises(AssertionError):
            layer(wrong)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        layer(x.cpu())
    if tokens > 1:
        for args in ((x, idx.int(), w), (x, idx, w.float()), (x, idx, w[:, :-1])):
            with pytest.raises(AssertionError):
                layer.experts(*args)


def test_out_of_memory_in_a_native_call_is_torchs_error(ib, device):
    """The scratch of a call finds no room: the allocator's limit is set to what is reserved, and the
    scratch of the next call comes on top."""
    layer, x = _block(ib, device, 64)
    prompt = x.repeat(64, 1)
    want = layer(prompt).clone()   # (buffers of the module, and the scratch, which goes back)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(device).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved(device) + (1 << 20)) / total, device)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            layer(prompt)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, device)
    assert torch.equal(layer(prompt), want)


def test_other_threads_run_while_a_call_waits_for_its_stream(ib, device):
    """More launches than a stream's queue holds, behind 0.5 s of other work: the call that finds the queue full waits, but not
    with the interpreter."""
    import threading
    import time

    layer, x = _block(ib, device, 9)
    layer(x)
    torch.cuda.synchronize()
    stop, gaps = threading.Event(), []

    def ticks():
        last = time.monotonic()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.monotonic()
            gaps.append(now - last)
            last = now

    thread = threading.Thread(target=ticks)
    thread.start()
    torch.cuda._sleep(int(0.5 * 1.9e9))
    start = time.monotonic()
    for _ in range(600):
        layer(x)
    waited = time.monotonic() - start
    stop.set()
    thread.join()
    torch.cuda.synchronize()
    assert waited > 0.25, "the queue took everything: the call never waited"
    assert max(gaps) < waited / 2   # (nearly all of it with the interpreter's lock held, a millisecond on an idle host)


def test_calls_of_several_threads_do_not_mix(ib, device):
    """One module on one stream from four threads: a call's launches follow one another."""
    import threading

    layer, x = _block(ib, device, 48)
    inputs = [x[12 * i:12 * i + 12].contiguous() for i in range(4)]
    want = [layer(t).clone() for t in inputs]
    torch.cuda.synchronize()
    wrong = []

    def run(i):
        for n in range(150):
            if not torch.equal(layer(inputs[i]), want[i]):
                wrong.append((i, n))

    threads = [threading.Thread(target=run, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


def test_descriptors_are_there_for_every_stream(ib, device):
    """Made on a stream that has other work in front; a stream that does not wait for it finds them whole."""
    gate, up, down = torch.zeros(2, 256, 512, dtype=BF16, device=device), torch.zeros(2, 256, 512, dtype=BF16, device=device), torch.zeros(2, 512, 256, dtype=BF16, device=device)
    want = ib.kernels.encode_shared_maps(gate, up, down).cpu()
    torch.cuda.synchronize()
    busy, other = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(busy):
        used = torch.full((1 << 14,), 127, dtype=torch.uint8, device=device)   # (what the allocator may hand out next)
        del used
        torch.cuda._sleep(int(0.1 * 1.9e9))
        maps = ib.kernels.encode_shared_maps(gate, up, down)
    with torch.cuda.stream(other):
        assert torch.equal(maps.cpu(), want)
    torch.cuda.synchronize()


def test_a_router_call_of_more_tokens_than_a_grid_is_high(ib, device):
    """65 535 tiles of sixteen tokens and a few more: the last tokens as in a call of their own."""
    tokens, hidden, routed, top_k = 65535 * 16 + 21, 8, 4, 2
    gen = torch.Generator(device).manual_seed(1)
    draw = lambda *s: torch.randn(*s, generator=gen, device=device)  # noqa: E731
    x, weight, bias, scale = draw(tokens, hidden).to(BF16), draw(routed, hidden).to(BF16), draw(routed) * 0.1, torch.ones(1, dtype=BF16, device=device)

    def route(x):
        t = x.shape[0]
        out = (torch.empty(t, top_k, dtype=BF16, device=device), torch.empty(t, top_k, dtype=torch.int64, device=device), torch.empty(t, 0, dtype=BF16, device=device))
        ib.kernels.router_forward(x, weight, bias, scale, 8.0, top_k, 0, *out, ib.kernels.router_workspace(t, routed, device))
        return out

    whole, last = route(x), route(x[-40:].contiguous())
    assert all(torch.equal(a[-40:], b) for a, b in zip(whole, last))


def test_a_token_comes_out_the_same_in_any_larger_company(ib, device):
    """From two tokens on, tiles of 16, 32 and 64 tokens: a token is a column of its own, its sums run in the same order."""
    layer, x = _block(ib, device, 300, d=512, f=256, experts=8)
    whole = layer(x)
    for tokens in (2, 9, 17, 40, 70, 131):   # means of 0.75 to 49 routes an expert (whole: 113)
        assert torch.equal(layer(x[:tokens].contiguous()), whole[:tokens]), tokens


def test_a_copy_of_a_stack_is_its_own(ib, device):
    """The copy's launch reads the copy's tensors, and takes nothing over that was kept for the original's graphs."""
    import copy

    stack = ib.MoEStack([_block(ib, device, 1, seed=s, d=1024, f=512, experts=8)[0] for s in (6, 7)], 1024)
    x = _block(ib, device, 1, d=1024, f=512, experts=8)[1]
    decode = ib.DecodeStackGraph(stack, x)
    stack.layers[0](x.repeat(40, 1))   # (replaces buffers that the graph has)
    want = stack(x).clone()
    twin = copy.deepcopy(stack)
    assert not twin._kept and not twin.layers[0]._kept and stack.layers[0]._kept
    for block in stack.layers:
        for t in (block.router_weight, block.shared_down, block.shared_gate):
            t.zero_()
    assert not torch.equal(stack(x), want)
    assert torch.equal(twin(x), want)
    del decode
