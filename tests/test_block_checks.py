"""What a block refuses before any address of its tensors reaches a kernel (no GPU: the checks come first)."""
from types import SimpleNamespace

import pytest
import torch
from torch import nn

D, F, ROUTED, SHARED = 256, 128, 8, 2


class _Experts(nn.Module):
    """What a FusedMoE needs of its experts to take its own tensors down."""

    quantized, bank_maps, generation, hidden_dim, intermediate_dim = True, None, 0, D, F

    def _reserve(self, routes):
        pass

    def _note_capture(self):
        pass


@pytest.fixture(autouse=True)
def nothing_is_captured(monkeypatch):
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)   # (the question needs a device)


def _block(**other):
    import inkling_b200 as ib

    bf = dict(dtype=torch.bfloat16)
    t = dict(router_weight=torch.zeros(ROUTED + SHARED, D, **bf), router_bias=torch.zeros(ROUTED), global_scale=torch.ones(1, **bf),
             shared_gate=torch.zeros(SHARED, F, D, **bf), shared_up=torch.zeros(SHARED, F, D, **bf), shared_down=torch.zeros(SHARED, D, F, **bf))
    t.update(other)
    block = ib.FusedMoE(t["router_weight"], t["router_bias"], t["global_scale"], 1.0, 2, t["shared_gate"], t["shared_up"], t["shared_down"], _Experts())
    block._reserve(4)
    return block


@pytest.mark.parametrize("name,change", [
    ("router_weight", lambda t: t.float()), ("router_weight", lambda t: t.half()), ("router_weight", lambda t: t[:, :-8].contiguous()),
    ("router_weight", lambda t: t.t().contiguous().t()), ("router_bias", lambda t: t[:-1]), ("router_bias", lambda t: t.repeat(2)),
    ("global_scale", lambda t: t.float()), ("shared_gate", lambda t: t.float()), ("shared_gate", lambda t: t.transpose(1, 2).contiguous()),
    ("shared_up", lambda t: t[:, :-16].contiguous()), ("shared_up", lambda t: t[:1]), ("shared_down", lambda t: t.transpose(1, 2)),
    ("shared_down", lambda t: t[:, :, :-16].contiguous()),
], ids=lambda v: v if isinstance(v, str) else "")
def test_a_tensor_the_kernels_would_misread_is_refused(name, change):
    block = _block(**{name: change(getattr(_block(), name))})
    with pytest.raises(AssertionError):
        block._record(False)
    with pytest.raises(AssertionError):
        block.block_descriptor()


def test_tensors_on_the_host_are_refused():
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        _block()._record(False)


def _out_of_memory_at(monkeypatch, nth):
    """torch.empty and torch.zeros as usual, the nth call of both together out of memory."""
    calls = []

    def wrap(make):
        def allocate(*args, **kwargs):
            calls.append(1)
            if len(calls) == nth:
                raise torch.OutOfMemoryError("planted")
            return make(*args, **kwargs)
        return allocate

    for name in ("empty", "zeros"):
        monkeypatch.setattr(torch, name, wrap(getattr(torch, name)))


@pytest.mark.parametrize("nth", range(1, 7))
def test_a_block_that_ran_out_of_memory_counts_on_no_buffers(monkeypatch, nth):
    block = _block()
    with monkeypatch.context() as m:
        _out_of_memory_at(m, nth)
        with pytest.raises(torch.OutOfMemoryError):
            block._reserve(9)
    assert block._tokens == 0
    block._reserve(2)
    assert block._tokens == 2 and all(getattr(block, n).shape[0] == 2 for n in ("topk_weights", "topk_indices", "gammas", "partial"))


@pytest.mark.parametrize("nth", range(1, 4))
def test_experts_that_ran_out_of_memory_count_on_no_buffers(monkeypatch, nth):
    import inkling_b200 as ib

    experts = ib.ResidentExperts.__new__(ib.ResidentExperts)
    nn.Module.__init__(experts)
    experts.local, experts.device, experts.dtype, experts.hidden_dim, experts.intermediate_dim, experts.capacity = 3, "cpu", torch.bfloat16, D, F, 0
    experts.rows = experts.activated = experts.down = None
    experts._reserve(4)
    with monkeypatch.context() as m:
        _out_of_memory_at(m, nth)
        with pytest.raises(torch.OutOfMemoryError):
            experts._reserve(9)
    assert experts.capacity == 0
    experts._reserve(2)
    assert experts.capacity == 2 and experts.rows.shape == (3, 2) and experts.activated.shape == (2, F) and experts.down.shape == (2, D)


@pytest.mark.parametrize("error,change", [
    (AssertionError, dict(query=lambda t: t.float())), (AssertionError, dict(k_cache=lambda t: t.transpose(2, 3))),
    (AssertionError, dict(position=lambda t: 3)), (AssertionError, dict(position=lambda t: t.int())), (AssertionError, dict(proj=lambda t: t.t())),
    (AssertionError, dict(pad_counts=lambda t: t.int())), (AssertionError, dict(pad_counts=lambda t: t[:1])), (AssertionError, dict(v_cache=lambda t: t[:, :, :-1])),
    (AssertionError, dict(relative_states=lambda t: t[..., :-1].contiguous())), (RuntimeError, dict(query=lambda t: torch.cat([t, t], 2))), (RuntimeError, {}),
    (TypeError, dict(k_cache=lambda t: None)),
], ids=lambda v: v.__name__ if isinstance(v, type) else "-".join(v) or "on the host")
def test_what_attention_refuses_and_with_which_error(error, change):
    """Arguments of the wrong form are assertions, whichever device they are on; then come the tensors that are not on a GPU."""
    import inkling_b200 as ib

    zeros = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)  # noqa: E731
    args = dict(query=zeros(2, 4, 1, 64), relative_states=zeros(2, 1, 4, 16), proj=zeros(16, 8), k_cache=zeros(2, 2, 20, 64), v_cache=zeros(2, 2, 20, 64),
                position=torch.tensor(3), pad_counts=torch.zeros(2, dtype=torch.int64))
    args.update({n: f(args[n]) for n, f in change.items()})
    with pytest.raises(error) as caught:
        ib.kernels.decode_attention(**args)
    assert caught.type is error


@pytest.mark.parametrize("tokens,pieces", [(1, [1]), (8, [8]), (20, [8, 8, 4])])
def test_a_decode_call_of_the_experts_makes_no_views(monkeypatch, tokens, pieces):
    """Banks that are not evenly spaced, recorded launches: a call that fits one launch hands its own tensors over (each view
    is a microsecond of a host-bound call), a larger one pieces of eight tokens in order."""
    import inkling_b200 as ib

    layer = __import__("sys").modules[ib.ResidentExperts.__module__]
    experts = ib.ResidentExperts.__new__(ib.ResidentExperts)
    nn.Module.__init__(experts)
    experts.local, experts.device, experts.dtype, experts.hidden_dim, experts.intermediate_dim, experts.capacity = 3, "cpu", torch.bfloat16, 32, 32, 0
    experts.rows = experts.activated = experts.down = experts.bank_maps = experts.device_mesh = None
    experts.quantized, experts.pointers, experts.max_expert, experts.status = True, None, 2, None
    planned, launched = [], []
    monkeypatch.setattr(ib.ResidentExperts, "_plan", lambda self, indices: planned.append(indices))
    monkeypatch.setattr(layer, "routed_decode", lambda x, i, w, p, a, out, *_, **__: (launched.append((x, i, w)), out.copy_(x.float() + 1)))
    x, indices, weights = torch.randn(tokens, 32).to(torch.bfloat16), torch.zeros(tokens, 2, dtype=torch.int64), torch.ones(tokens, 2, dtype=torch.bfloat16)
    got = experts(x, indices, weights)
    assert torch.equal(got, (x.float() + 1).to(torch.bfloat16)) and planned[0] is indices and len(planned) == 1
    assert [len(t[0]) for t in launched] == pieces
    if len(pieces) == 1:
        assert launched[0][0] is x and launched[0][1] is indices and launched[0][2] is weights
