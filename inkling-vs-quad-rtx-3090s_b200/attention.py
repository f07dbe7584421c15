"""The decode step of the reference's attention module on this library's kernels.

`MyInklingAttention.forward` with a decoding cache (my_inkling/model.py:504-622) is: the fused QKVR projection,
RMS norm of the query heads, short convolution + RMS norm of the key, short convolution of the value, `update_kv`,
relative-position bias + mask + `scaled_dot_product_attention`, the output projection (and its all-reduce under
tensor parallelism). Here that is `ink_linear` (up to eight sequences; library GEMMs above), `ink_attention_heads`,
`ink_decode_attention` (which also stores the token in the caches) and `ink_linear` again. The cache object is the reference's `MyInklingCache` (or anything with the same fields:
`layers[i].k_cache / v_cache / conv_caches[0 | 1].cache`, `position`, `pad_counts`).
"""
from __future__ import annotations

import torch
import torch.nn as nn
import torch.nn.functional as F

from .kernels import attention_heads, decode_attention, gated, linear, rmsnorm, short_conv, short_conv_norm
from .kernels.paired_all_reduce import all_reduce


def _norm_rows(rows: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """RMS norm over the last dimension of BF16 [n, c], of any strides, with the reference's rounding (kernels/decode.py:36-43)."""
    rows = rows.contiguous()
    return rmsnorm(rows if rows.data_ptr() % 16 == 0 else rows.clone(), weight, eps)


def _aligned(*tensors: torch.Tensor) -> bool:
    return all(t.data_ptr() % 16 == 0 for t in tensors)


def _runs_alone(module, kind) -> bool:
    """A call of `module` launches `kind`'s kernels and nothing before them: no hook, no other forward."""
    return (type(module) is kind and "forward" not in vars(module) and not module._forward_pre_hooks
            and not nn.modules.module._global_forward_pre_hooks)


class _Projections(nn.Module):
    """Modules whose projections report a bounded wait that gave up in one status word."""

    def _make_status(self, weight: torch.Tensor) -> None:
        self.register_buffer("status", torch.zeros(1, dtype=torch.int32, device=weight.device), persistent=False)

    def check_status(self) -> None:
        """Host read (synchronises): raises if a wait inside a projection of this module, or of those it holds, gave up
        since the last check; the outputs of that call are invalid. Call outside graph capture."""
        words = [m.status for m in self.modules() if isinstance(m, _Projections)]
        flags = [int(w.item()) for w in words]
        for w in words:
            w.zero_()
        if any(flags):
            raise RuntimeError(f"{type(self).__name__}: a bounded wait inside a projection timed out; the output of that call is invalid")


class DecodeAttention(_Projections):
    def __init__(self, qkvr_weight, o_weight, q_norm_weight, k_norm_weight, k_taps, v_taps, rel_proj, *, layer_idx: int,
                 heads: int, kv_heads: int, head_dim: int, d_rel: int, window: int = 0, log_scaling_n_floor=None,
                 log_scaling_alpha: float = 0.1, eps: float = 1e-6, group=None):
        """Weights as the reference module holds them after `fuse_projections`: qkvr_weight BF16
        [(h + 2 hk) c + h d_rel, d], o_weight BF16 [d, h c], norm weights BF16 [c], taps FP32 [hk c, 1, K],
        rel_proj BF16 [d_rel, rel_extent]. `window` > 0 for a sliding layer. `group`: the tensor-parallel process
        group whose ranks hold slices of the heads (the output projection's partial sums are all-reduced)."""
        super().__init__()
        self.layer_idx, self.heads, self.kv_heads, self.head_dim, self.d_rel = layer_idx, heads, kv_heads, head_dim, d_rel
        self.window, self.n_floor, self.alpha, self.eps, self.group = window, log_scaling_n_floor, log_scaling_alpha, eps, group
        self.sizes = [heads * head_dim, kv_heads * head_dim, kv_heads * head_dim, heads * d_rel]
        assert qkvr_weight.shape[0] == sum(self.sizes)
        for name, t in (("qkvr_weight", qkvr_weight), ("o_weight", o_weight), ("q_norm_weight", q_norm_weight),
                        ("k_norm_weight", k_norm_weight), ("k_taps", k_taps), ("v_taps", v_taps), ("rel_proj", rel_proj)):
            self.register_buffer(name, t.contiguous())
        self._make_status(self.qkvr_weight)

    @classmethod
    def from_reference(cls, attention, group=None) -> "DecodeAttention":
        """From a `MyInklingAttention` whose projections are fused (`fuse_projections`), on its device."""
        return cls(attention.qkvr_proj.weight.detach(), attention.o_proj.weight.detach(), attention.q_norm.weight.detach(),
                   attention.k_norm.weight.detach(), attention.k_sconv.conv1d.weight.detach(),
                   attention.v_sconv.conv1d.weight.detach(), attention.rel_logits_proj.proj.detach(),
                   layer_idx=attention.layer_idx, heads=attention.num_heads, kv_heads=attention.num_key_value_heads,
                   head_dim=attention.head_dim, d_rel=attention.rel_logits_proj.d_rel, window=attention.sliding_window or 0,
                   log_scaling_n_floor=attention.log_scaling_n_floor, log_scaling_alpha=attention.log_scaling_alpha,
                   eps=attention.q_norm.variance_epsilon, group=group)

    def _norm(self, rows: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
        return _norm_rows(rows, weight, self.eps)

    def forward(self, hidden_states: torch.Tensor, cache, *, settled: bool = False) -> torch.Tensor:
        """hidden_states BF16 [bs, 1, d], cache in decode mode -> BF16 [bs, 1, d]; the caches and the convolution
        histories of this layer are updated in place, `cache.position` is left to the caller (`cache.advance`).
        `settled`: the launch in front is a kernel that does not write this module's weights (see `linear`)."""
        bs, s, _ = hidden_states.shape
        assert s == 1, "one token per sequence"
        layer = cache.layers[self.layer_idx]
        h, hk, c = self.heads, self.kv_heads, self.head_dim
        qkvr = linear(hidden_states, self.qkvr_weight, settled=settled, status=self.status)
        k_history, v_history = layer.conv_caches[0].cache, layer.conv_caches[1].cache
        if c % 8 == 0 and c <= 256 and (h * self.d_rel) % 8 == 0 and self.k_taps.shape == self.v_taps.shape and _aligned(qkvr, self.q_norm_weight, self.k_norm_weight, self.k_taps, self.v_taps, k_history, v_history):
            q, k, v, r = attention_heads(qkvr.view(bs, -1), self.q_norm_weight, self.k_norm_weight, self.k_taps, self.v_taps, k_history, v_history, self.eps,
                                         h, hk, c, self.d_rel)
        else:   # heads of other widths, convolutions of two lengths, histories that start anywhere
            q, k, v, r = qkvr.split(self.sizes, dim=-1)
            q = self._norm(q.reshape(bs * h, c).contiguous(), self.q_norm_weight)
            k = short_conv(k.contiguous(), self.k_taps, k_history, None)
            k = self._norm(k.reshape(bs * hk, c), self.k_norm_weight)
            v = short_conv(v.contiguous(), self.v_taps, v_history, None)
        out = decode_attention(q.view(bs, h, c), r.reshape(bs, h, self.d_rel), self.rel_proj, layer.k_cache, layer.v_cache,
                               cache.position, cache.pad_counts, window=self.window, log_scaling_n_floor=self.n_floor,
                               log_scaling_alpha=self.alpha, scale=1.0 / c, new_key=k.view(bs, hk, 1, c),
                               new_value=v.reshape(bs, hk, 1, c))
        y = linear(out.reshape(bs, 1, h * c), self.o_weight, settled=True, status=self.status)   # (the attention is in front)
        if self.group is not None:
            y = all_reduce(y, self.group)   # (nothing to do with one rank)
        return y


class DecodeLayer(nn.Module):
    """One sparse decoder layer at decode, `MyInklingDecoderLayer.forward` (my_inkling/model.py:661-675):
    h' = attn_sconv(attention(input_norm(h)), residual=h);  out = mlp_sconv(moe(post_norm(h')), residual=h').
    `attention` is a DecodeAttention, `moe` a FusedMoE (a sparse layer) or a DenseMLP (a dense one); the two short
    convolutions use the layer's convolution caches 2 and 3 of the reference's cache object."""

    def __init__(self, attention: DecodeAttention, moe, input_norm_weight, post_norm_weight, attn_taps, mlp_taps, eps: float = 1e-6):
        super().__init__()
        self.attention, self.moe, self.eps = attention, moe, eps
        for name, t in (("input_norm_weight", input_norm_weight), ("post_norm_weight", post_norm_weight),
                        ("attn_taps", attn_taps), ("mlp_taps", mlp_taps)):
            self.register_buffer(name, t.contiguous())

    def _norm(self, x: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
        return _norm_rows(x.reshape(-1, x.shape[-1]), weight, self.eps).view(x.shape)

    def forward(self, hidden_states: torch.Tensor, cache) -> torch.Tensor:
        """hidden_states BF16 [bs, 1, d] -> BF16 [bs, 1, d]; the layer's caches are updated in place."""
        bs, _, d = hidden_states.shape
        layer = cache.layers[self.attention.layer_idx]
        normed = self._norm(hidden_states, self.input_norm_weight)
        attended = self.attention(normed, cache, settled=True) if _runs_alone(self.attention, DecodeAttention) else self.attention(normed, cache)
        attended, history, residual = attended.contiguous(), layer.conv_caches[2].cache, hidden_states.contiguous()
        if d % 8 == 0 and attended.dtype == torch.bfloat16 and _aligned(self.attn_taps, history):
            h, normed = short_conv_norm(attended, self.attn_taps, history, residual, self.post_norm_weight, self.eps)
        else:
            h = short_conv(attended, self.attn_taps, history, residual)
            normed = self._norm(h, self.post_norm_weight).view(bs, d)
        if _runs_alone(self.moe, DenseMLP):
            block = self.moe(normed, settled=True)
        else:
            block = self.moe.forward_partial(normed) if hasattr(self.moe, "forward_partial") else self.moe(normed)   # [bs, d], all-reduced
        return short_conv(block.view(bs, 1, d).contiguous(), self.mlp_taps, layer.conv_caches[3].cache, h)


class DenseMLP(_Projections):
    """`MyInklingMLP` (my_inkling/model.py:153-171), the block of a dense layer: two launches of `ink_linear`,
    down(silu(gate(x)) * up(x)) * global_scale, BF16 like the reference's; all-reduced over `group` when the rows of
    gate/up and the columns of down are sliced."""

    def __init__(self, gate_weight, up_weight, down_weight, global_scale, group=None):
        super().__init__()
        for name, t in (("gate_weight", gate_weight), ("up_weight", up_weight), ("down_weight", down_weight), ("global_scale", global_scale)):
            self.register_buffer(name, t.contiguous())
        self._make_status(self.gate_weight)
        self.group = group

    def forward(self, x: torch.Tensor, *, settled: bool = False) -> torch.Tensor:
        """`settled`: as of DecodeAttention."""
        y = linear(gated(x, self.gate_weight, self.up_weight, settled=settled, status=self.status), self.down_weight, self.global_scale, settled=True,
                   status=self.status)
        return y if self.group is None else all_reduce(y, self.group)


class DecodeModel(_Projections):
    """One decode step of the reference's model, `MyInkling.forward` with a decoding cache (my_inkling/model.py:679-800):
    normed embedding, the decoder layers, the final norm, the logits (hidden / mup multiplier through the LM head), and
    the cache's position counter moved on by one token."""

    def __init__(self, embedding, embed_norm_weight, layers, final_norm_weight, lm_head_weight, mup_multiplier: float,
                 eps: float = 1e-6, unpadded_vocab_size=None):
        super().__init__()
        for name, t in (("embedding", embedding), ("embed_norm_weight", embed_norm_weight), ("final_norm_weight", final_norm_weight),
                        ("lm_head_weight", lm_head_weight)):
            self.register_buffer(name, t.contiguous())
        self._make_status(self.lm_head_weight)
        self.layers = nn.ModuleList(layers)
        self.mup, self.eps, self.unpadded = float(mup_multiplier), eps, unpadded_vocab_size

    def forward(self, input_ids: torch.Tensor, cache) -> torch.Tensor:
        """input_ids int64 [bs, 1] -> logits BF16 [bs, 1, vocab]."""
        norm = self.layers[0]._norm
        hidden = norm(F.embedding(input_ids, self.embedding), self.embed_norm_weight)
        for layer in self.layers:
            hidden = layer(hidden, cache)
        hidden = norm(hidden, self.final_norm_weight) / self.mup
        logits = linear(hidden, self.lm_head_weight, settled=True, status=self.status)   # (the division is in front)
        cache.position.add_(1)
        return logits if self.unpadded is None else logits[..., : self.unpadded]
