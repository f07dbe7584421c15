"""GPU parity of what sits either side of the MoE block and of the unquantised expert
layer: residual add + RMS norm, the short convolution (mlp_sconv) with the decoder
residual, the BF16-bank GEMV (the reference's QUANT=0 build), against the CPU oracle and
against fixtures written by the reference's own modules and kernels."""
import pytest
import torch

import cases
from helpers import BF16, bf16_ulps, max_rel
from oracle import moe as oracle_moe

pytestmark = pytest.mark.gpu
TOL = 2e-2


@pytest.fixture(scope="module")
def ib():
    import inkling_b200

    return inkling_b200


@pytest.fixture(scope="module")
def device():
    return torch.device("cuda", 0)


def g(golden, key, dtype=None):
    t = torch.from_numpy(golden[key])
    return t.to(dtype) if dtype is not None else t


def test_add_rmsnorm_against_oracle_and_reference_module(ib, device, golden):
    gen = torch.Generator().manual_seed(cases.GLUE_SEED)
    x, w = cases.glue_inputs(gen)
    # residual = 0, partial = x: the norm of bf16(x) is the reference module's fixture
    residual = torch.zeros_like(x).to(device)
    normed = torch.empty_like(residual)
    ib.kernels.add_rmsnorm(x.float().to(device), residual, w.to(device), cases.EPS, normed)
    torch.cuda.synchronize()
    assert torch.equal(residual.cpu(), x)
    want = g(golden, "glue/norm_bf16", BF16)
    ulps = bf16_ulps(normed, want)
    assert int(ulps.max()) <= 1 and float((ulps > 0).float().mean()) < 0.01   # rsqrt and summation order: last bit
    # a real residual and an FP32 partial that does not fit BF16: both roundings of the add
    gen = torch.Generator().manual_seed(5)
    partial = torch.randn(4, 4096, generator=gen) * 0.3
    res = torch.randn(4, 4096, generator=gen).to(BF16)
    weight = (1.0 + 0.1 * torch.randn(4096, generator=gen)).to(BF16)
    want_res, want_norm = oracle_moe.add_rms_norm_reference(partial, res, weight, cases.EPS)
    res_d, norm_d = res.to(device), torch.empty(4, 4096, dtype=BF16, device=device)
    ib.kernels.add_rmsnorm(partial.to(device), res_d, weight.to(device), cases.EPS, norm_d)
    torch.cuda.synchronize()
    assert torch.equal(res_d.cpu(), want_res)                       # the BF16 add is exact arithmetic + one rounding
    ulps = bf16_ulps(norm_d, want_norm)
    assert int(ulps.max()) <= 1 and float((ulps > 0).float().mean()) < 0.01


def test_short_conv_against_oracle_and_reference(ib, device, golden):
    gen = torch.Generator().manual_seed(cases.GLUE_SEED)
    cases.glue_inputs(gen)
    seq, taps, res = cases.sconv_inputs(gen)
    k = taps.shape[-1]
    history = torch.zeros(seq.shape[0], seq.shape[-1], k)
    history[..., 1:] = seq[:, : k - 1].float().transpose(1, 2)
    want, want_history = oracle_moe.short_conv_reference(seq[:, -1], taps, history, res[:, -1])
    weight = taps.unsqueeze(1).contiguous().to(device)
    h_d = history.to(device)
    y = ib.kernels.short_conv(seq[:, -1:].contiguous().to(device), weight, h_d, res[:, -1:].contiguous().to(device))
    torch.cuda.synchronize()
    assert torch.equal(y[:, 0].cpu(), want)                         # same FP32 operations in the same order
    assert torch.equal(h_d.cpu(), want_history)
    ulps = bf16_ulps(y[:, 0], g(golden, "glue/sconv_module_bf16", BF16))
    assert int(ulps.max()) <= 1 and float((ulps > 0).float().mean()) < 0.02   # the module's conv1d sums in another order
    # without the decoder residual
    h_d = history.to(device)
    y = ib.kernels.short_conv(seq[:, -1:].contiguous().to(device), weight, h_d, None)
    want0, _ = oracle_moe.short_conv_reference(seq[:, -1], taps, history, None)
    assert torch.equal(y[:, 0].cpu(), want0)
    # FP32 input (the block's all-reduced output): rounded to BF16 first
    h_d = history.to(device)
    x32 = seq[:, -1:].float() * 1.001
    y = ib.kernels.short_conv(x32.contiguous().to(device), weight, h_d, res[:, -1:].contiguous().to(device))
    want32, want_h32 = oracle_moe.short_conv_reference(x32[:, 0].to(BF16), taps, history, res[:, -1])
    torch.cuda.synchronize()
    assert torch.equal(y[:, 0].cpu(), want32) and torch.equal(h_d.cpu(), want_h32)
    # four decode steps in a row: the history carries
    h_d, h_cpu = history.to(device), history.clone()
    for step in range(4):
        xs = torch.randn(seq.shape[0], 1, seq.shape[-1], generator=gen).to(BF16)
        y = ib.kernels.short_conv(xs.to(device), weight, h_d, None)
        want_y, h_cpu = oracle_moe.short_conv_reference(xs[:, 0], taps, h_cpu, None)
        assert torch.equal(y[:, 0].cpu(), want_y)
    assert torch.equal(h_d.cpu(), h_cpu)


def _bf16_table(dev_banks, device):
    n = max(dev_banks) + 1
    table = torch.zeros(n, 2, dtype=torch.int64)
    for e, b in dev_banks.items():
        table[e] = torch.tensor([b["gate_up_proj"].data_ptr(), b["down_proj"].data_ptr()])
    return table.reshape(-1).to(device)


@pytest.mark.parametrize("name", ["tiny", "small", "mid"])
def test_bf16_bank_gemv_against_oracle_and_reference_cuda_file(ib, device, golden, name):
    c = cases.LAYER_CASES[name]
    p, banks, x = cases.make_layer(**c)
    bf = cases.bf16_banks(banks)
    if f"{name}/bf16_gemv_out" in golden:
        idx = g(golden, f"{name}/router_indices")
        w = g(golden, f"{name}/router_weights", BF16)
    else:
        gen = torch.Generator().manual_seed(3)
        idx = torch.stack([torch.randperm(c["experts"], generator=gen)[: c["top_k"]] for _ in range(x.shape[0])])
        w = torch.rand(x.shape[0], c["top_k"], generator=gen).to(BF16)
    dev = {e: {n: t.to(device).contiguous() for n, t in b.items()} for e, b in bf.items()}
    pointers = _bf16_table(dev, device)
    t, k = idx.shape
    activated = torch.zeros(t * k, c["f"], dtype=BF16, device=device)
    out = torch.full((t, c["d"]), float("nan"), dtype=torch.float32, device=device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    ib.kernels.routed_decode(x.to(device), idx.to(device), w.to(device), pointers, activated, out, c["experts"] - 1,
                             False, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    want_act, want_out = oracle_moe.routed_decode_bf16_reference(x, idx, w, bf)
    assert max_rel(activated.cpu().float(), want_act.float()) <= 8e-3
    assert max_rel(out.cpu(), want_out) <= 8e-3
    assert max_rel(out.cpu(), oracle_moe.routed_experts_bf16_fp32(x, idx, w, bf)) <= TOL
    if f"{name}/bf16_gemv_out" in golden:
        assert max_rel(activated.cpu().float(), g(golden, f"{name}/bf16_gemv_activated")) <= 8e-3
        assert max_rel(out.cpu(), g(golden, f"{name}/bf16_gemv_out")) <= 8e-3


def test_bf16_banks_skip_inactive_and_flag_out_of_range(ib, device):
    c = cases.LAYER_CASES["small"]
    p, banks, x = cases.make_layer(**c)
    bf = cases.bf16_banks(banks)
    dev = {e: {n: t.to(device).contiguous() for n, t in b.items()} for e, b in bf.items()}
    pointers = _bf16_table(dev, device)
    pointers.view(-1, 2)[3] = 0                                      # expert 3 is "not on this rank"
    idx = torch.tensor([[3, 1, 2, 4, 5, 6], [0, 1, 2, 3, 99, 5], [7, 8, 9, 10, 11, 12]])
    w = torch.full((3, 6), 0.25).to(BF16)
    activated = torch.zeros(18, c["f"], dtype=BF16, device=device)
    out = torch.empty(3, c["d"], dtype=torch.float32, device=device)
    status = torch.zeros(1, dtype=torch.int32, device=device)
    ib.kernels.routed_decode(x.to(device), idx.to(device), w.to(device), pointers, activated, out, c["experts"] - 1,
                             False, status=status)
    torch.cuda.synchronize()
    assert int(status.item()) & 1
    kept = {e: b for e, b in bf.items() if e != 3}
    _, want = oracle_moe.routed_decode_bf16_reference(x, idx, w, kept, max_expert=c["experts"] - 1)
    assert max_rel(out.cpu(), want) <= 8e-3


def test_resident_experts_over_bf16_banks(ib, device):
    """The unquantised expert layer through the drop-in module (stride-2 pointer table), at
    more tokens than one GEMV batch."""
    c = dict(cases.LAYER_CASES["small"], tokens=11)
    p, banks, x = cases.make_layer(**c)
    bf = cases.bf16_banks(banks)
    dev = {e: {n: t.to(device).contiguous() for n, t in b.items()} for e, b in bf.items()}
    experts = ib.ResidentExperts(c["d"], c["f"], None, dev, quantized=False)
    assert experts.stride == 2
    gen = torch.Generator().manual_seed(8)
    idx = torch.stack([torch.randperm(c["experts"], generator=gen)[: c["top_k"]] for _ in range(11)])
    w = torch.rand(11, c["top_k"], generator=gen).to(BF16)
    out = experts(x.to(device), idx.to(device), w.to(device))
    torch.cuda.synchronize()
    experts.check_status()
    assert out.dtype == BF16
    assert max_rel(out.float(), oracle_moe.routed_experts_bf16_fp32(x, idx, w, bf)) <= TOL


@pytest.mark.parametrize("hidden,rows", [(8, 3), (64, 5), (2048, 1), (2056, 2), (4096, 7), (16384, 2)])
def test_the_norm_alone_is_the_norm_of_the_sum_with_zeros(ib, device, hidden, rows):
    gen = torch.Generator().manual_seed(hidden)
    x, w = torch.randn(rows, hidden, generator=gen).to(BF16).to(device), torch.randn(hidden, generator=gen).to(BF16).to(device)
    x[0, :4] = 0
    kept, want = x.clone(), torch.empty_like(x)
    ib.kernels.add_rmsnorm(torch.zeros(rows, hidden, device=device), x.clone(), w, cases.EPS, want)
    assert torch.equal(ib.kernels.rmsnorm(x, w, cases.EPS), want) and torch.equal(x, kept)


def _conv(gen, device, batch, hidden, taps, at=0):
    """Taps and history, the latter `at` floats into its buffer."""
    buffer = torch.randn(batch * hidden * taps + at, generator=gen).to(device)
    return torch.randn(hidden, 1, taps, generator=gen).to(device) * 0.3, buffer[at:].view(batch, hidden, taps)


@pytest.mark.parametrize("batch,hidden,taps", [(1, 8, 4), (2, 256, 3), (3, 2040, 4), (1, 2056, 2), (7, 4096, 4), (2, 6152, 4), (1, 16384, 4)])
def test_convolution_residual_and_norm_in_one_launch(ib, device, batch, hidden, taps):
    """The same bits as short_conv and rmsnorm one after the other, twice (the history moves on)."""
    gen = torch.Generator().manual_seed(hidden)
    weight, history = _conv(gen, device, batch, hidden, taps)
    norm, again = torch.randn(hidden, generator=gen).to(BF16).to(device), history.clone()
    for _ in range(2):
        x, residual = (torch.randn(batch, 1, hidden, generator=gen).to(BF16).to(device) for _ in range(2))
        want = ib.kernels.short_conv(x, weight, again, residual)
        y, normed = ib.kernels.short_conv_norm(x, weight, history, residual, norm, cases.EPS)
        assert torch.equal(y, want) and torch.equal(history, again)
        assert torch.equal(normed, ib.kernels.rmsnorm(want.view(batch, hidden), norm, cases.EPS))


def test_a_convolution_history_may_start_anywhere(ib, device):
    gen = torch.Generator().manual_seed(1)
    weight, history = _conv(gen, device, 2, 300, 4, at=1)
    x, again = torch.randn(2, 1, 300, generator=gen).to(BF16).to(device), history.clone()
    assert torch.equal(ib.kernels.short_conv(x, weight, history), ib.kernels.short_conv(x, weight, again)) and torch.equal(history, again)


@pytest.mark.parametrize("batch,heads,kv_heads,head_dim,d_rel,taps", [(1, 64, 16, 128, 16, 4), (7, 64, 8, 128, 16, 4), (2, 3, 3, 64, 8, 3), (3, 4, 1, 256, 6, 4),
                                                                     (1, 2, 1, 8, 300, 2), (2, 1, 1, 40, 16, 4)])
def test_heads_between_projection_and_attention(ib, device, batch, heads, kv_heads, head_dim, d_rel, taps):
    """The same bits as the split, the norms, the convolutions and the copies one by one."""
    gen = torch.Generator().manual_seed(head_dim + heads)
    sizes = [heads * head_dim, kv_heads * head_dim, kv_heads * head_dim, heads * d_rel]
    qkvr = torch.randn(batch, sum(sizes), generator=gen).to(BF16).to(device)
    q_weight, k_weight = (torch.randn(head_dim, generator=gen).to(BF16).to(device) for _ in range(2))
    (k_taps, k_history), (v_taps, v_history) = (_conv(gen, device, batch, kv_heads * head_dim, taps) for _ in range(2))
    kh, vh = k_history.clone(), v_history.clone()
    got = ib.kernels.attention_heads(qkvr, q_weight, k_weight, k_taps, v_taps, k_history, v_history, cases.EPS, heads, kv_heads, head_dim, d_rel)
    q, k, v, r = qkvr.split(sizes, dim=-1)
    q = ib.kernels.rmsnorm(q.reshape(-1, head_dim).contiguous(), q_weight, cases.EPS).view(batch, heads, head_dim)
    k = ib.kernels.short_conv(k.unsqueeze(1).contiguous(), k_taps, kh)
    k = ib.kernels.rmsnorm(k.view(-1, head_dim), k_weight, cases.EPS).view(batch, kv_heads, head_dim)
    v = ib.kernels.short_conv(v.unsqueeze(1).contiguous(), v_taps, vh).view(batch, kv_heads, head_dim)
    for a, b in zip(got, (q, k, v, r.reshape(batch, heads, d_rel))):
        assert torch.equal(a, b)
    assert torch.equal(k_history, kh) and torch.equal(v_history, vh)


# rows fewer and more than blocks, at the edges of a consumer's sixteen, in one round and several; columns at the edges of a stage
@pytest.mark.parametrize("n,k", [(1, 32), (8, 256), (149, 288), (2377, 64), (17, 4096), (100, 4128), (33, 8192), (11841, 1024), (24000, 96)])
@pytest.mark.parametrize("tokens", [1, 2, 5, 8])
def test_a_projection_against_64_bits(ib, device, n, k, tokens):
    """Exact products; FP32 sums of k of them, each off by at most 2^-23 of the magnitudes so far, and one rounding to BF16 (two
    with the factor, of which the second is of a value that the first may have moved)."""
    gen = torch.Generator().manual_seed(n + k + tokens)
    x, w = torch.randn(tokens, k, generator=gen).to(BF16).to(device), (torch.randn(n, k, generator=gen) * 0.05).to(BF16).to(device)
    scale = torch.tensor([1.375]).to(BF16).to(device)
    exact, magnitude = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    for factor, got in ((1.0, ib.kernels.linear(x, w)), (1.375, ib.kernels.linear(x, w, scale))):
        bound = (1 if factor == 1.0 else 2.01) * 2.0 ** -8 * (exact * factor).abs() + factor * k * 2.0 ** -23 * magnitude
        assert got.shape == (tokens, n) and bool(((got.double() - exact * factor).abs() <= bound).all())


@pytest.mark.parametrize("n,k,tokens", [(4, 64, 1), (5, 512, 8), (1187, 96, 3), (6, 4128, 2), (3, 8192, 7), (5921, 288, 4), (13000, 32, 1)])
def test_a_gated_projection_rounds_as_the_tensor_operations_do(ib, device, n, k, tokens):
    """The two projections have the sums of `linear`, checked above; what follows has one outcome."""
    gen = torch.Generator().manual_seed(n * k)
    x = torch.randn(tokens, k, generator=gen).to(BF16).to(device)
    gate, up = ((torch.randn(n, k, generator=gen) * 1.5 / k ** 0.5).to(BF16).to(device) for _ in range(2))
    want = torch.nn.functional.silu(ib.kernels.linear(x, gate)) * ib.kernels.linear(x, up)
    assert torch.equal(ib.kernels.gated(x, gate, up), want)


def test_a_projection_in_a_chain_sees_what_the_kernel_in_front_wrote(ib, device):
    """Weights are asked for before the kernel in front has finished, the activations not: twenty in a row against one by one."""
    gen = torch.Generator().manual_seed(2)
    ws = [(torch.randn(2048, 2048, generator=gen) * 0.03).to(BF16).to(device) for _ in range(20)]
    x = torch.randn(3, 2048, generator=gen).to(BF16).to(device)
    one_by_one = x
    for w in ws:
        one_by_one = ib.kernels.linear(one_by_one, w)
        torch.cuda.synchronize()
    for _ in range(3):
        y = x
        for w in ws:
            y = ib.kernels.linear(y, w)
        assert torch.equal(y, one_by_one)


def _weights_normed(k, x, w0, norm):
    return k.linear(x, k.rmsnorm(w0, norm, cases.EPS))


def _weights_normed_one_further(k, x, w0, norm):
    w = k.rmsnorm(w0, norm, cases.EPS)
    return k.linear(k.rmsnorm(x, norm, cases.EPS), w)


def _weights_projected(k, x, w0, norm):
    return k.linear(x, k.linear(w0[:8], w0))


def _pair_projected(k, x, w0, norm):
    return k.gated(x, k.linear(w0[:8], w0), k.linear(w0[8:16], w0))


@pytest.mark.parametrize("rows,width,chain", [(16, 4096, _weights_normed), (16, 4096, _weights_normed_one_further), (32, 32, _weights_projected), (32, 32, _pair_projected)])
def test_a_projections_weights_may_be_what_the_kernels_in_front_wrote(ib, device, rows, width, chain):
    """A captured chain whose weights are other values at every replay, behind a kernel that takes long on a third of the SMs and lets
    the chain start beside it: what the weights' memory held before must not be read."""
    gen = torch.Generator(device=device).manual_seed(3)

    def values(*shape):
        return torch.randn(*shape, generator=gen, device=device).to(BF16)

    x, w0, norm = values(5, width), values(rows, 4096), torch.ones(4096, dtype=BF16, device=device)
    long_x, long_w = values(8, 8192), values(48, 8192)

    def step():
        ib.kernels.linear(long_x, long_w)
        return chain(ib.kernels, x, w0, norm)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = step()

    class OneByOne:
        def __getattr__(self, name):
            def call(*args):
                y = getattr(ib.kernels, name)(*args)
                torch.cuda.synchronize()
                return y
            return call

    for _ in range(4):
        x.copy_(values(5, width))
        w0.copy_(values(rows, 4096))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, chain(OneByOne(), x, w0, norm))


@pytest.mark.parametrize("n,k,tokens", [(300, 512, 8), (17, 96, 3), (24000, 288, 2), (4096, 4096, 7)])
def test_a_projections_sums_run_over_the_columns_in_order(ib, device, n, k, tokens):
    """Sixteen at a time into one accumulator: the same bits for a row and a token in any company, and with columns of zeros
    before or behind (a sum cut in parts would be cut elsewhere)."""
    gen = torch.Generator(device=device).manual_seed(n)
    x, w = torch.randn(tokens, k, generator=gen, device=device).to(BF16), torch.randn(n, k, generator=gen, device=device).to(BF16)
    y = ib.kernels.linear(x, w)
    for rows, some in ((slice(0, 1), slice(0, 1)), (slice(n // 3, n // 3 + 21), slice(1, 3)), (slice(n - 5, n), slice(0, tokens))):
        assert torch.equal(ib.kernels.linear(x[some].clone(), w[rows].clone()), y[some, rows])
    for before, behind in ((0, 8192 - k), (8192 - k, 0), (16, 1024 - 16)):
        if k + before + behind <= 8192:
            assert torch.equal(ib.kernels.linear(*(torch.nn.functional.pad(t, (before, behind)) for t in (x, w))), y)


@pytest.mark.skipif(not torch.__version__.startswith("2.11."), reason="what was seen with the library of torch 2.11: another may cut the sums elsewhere")
@pytest.mark.parametrize("n,k,tokens", [(11264, 4096, 1), (4096, 8192, 7), (8192, 4096, 3)])
def test_a_layers_projections_are_the_bits_of_a_plain_gemm(ib, device, n, k, tokens):
    gen = torch.Generator(device=device).manual_seed(n)
    x, w = torch.randn(tokens, k, generator=gen, device=device).to(BF16), (torch.randn(n, k, generator=gen, device=device) * 0.02).to(BF16)
    assert torch.equal(ib.kernels.linear(x, w), torch.nn.functional.linear(x, w))
