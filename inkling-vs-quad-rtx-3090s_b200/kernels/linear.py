"""Dense BF16 projections of a decode step (ink_linear)."""
from __future__ import annotations

from functools import partial

import torch
import torch.nn.functional as F

from . import _abi

MOST_TOKENS, MOST_COLUMNS = 8, 8192


def _plain(*tensors) -> bool:
    """Nothing but the values is asked for: no gradient, no transform, mode or subclass that has to see the operation."""
    if torch.compiler.is_compiling() or torch.jit.is_tracing() or torch.is_autocast_enabled("cuda") or torch._C._len_torch_dispatch_stack() or torch._C._len_torch_function_stack():
        return False
    if torch._C._functorch.peek_interpreter_stack() is not None or torch.autograd.forward_ad._current_level >= 0:
        return False
    grad = torch.is_grad_enabled()
    return all(type(t) in (torch.Tensor, torch.nn.Parameter) and not (grad and t.requires_grad) for t in tensors)


def _fits(x, *weights) -> bool:
    """What the kernel takes: up to eight tokens, BF16 rows on one GPU, on 16-byte boundaries."""
    k = x.shape[-1]
    return (x.dtype == torch.bfloat16 and x.is_cuda and x.is_contiguous() and 0 < k <= MOST_COLUMNS and k % 32 == 0 and 0 < x.numel() <= MOST_TOKENS * k
            and x.data_ptr() % 16 == 0
            and all(w.dtype == torch.bfloat16 and w.dim() == 2 and w.shape[1] == k and 0 < w.shape[0] <= 1 << 24 and w.device == x.device
                    and w.is_contiguous() and w.data_ptr() % 16 == 0 for w in weights))


def _launch(x, weight, up, scale, settled=False, status=None):
    n, k = weight.shape
    y = x.new_empty(*x.shape[:-1], n)
    with torch.cuda.device(x.device):
        _abi.check(_abi.lib().ink_linear_settled(x.data_ptr(), weight.data_ptr(), _abi.ptr(up), _abi.ptr(scale), y.data_ptr(), x.numel() // k, n, k, int(settled),
                                                 _abi.ptr(status), _abi.stream()))
    return y


def _launcher(settled, status):
    return partial(_launch, settled=settled, status=status) if settled or status is not None else _launch


def linear(x, weight, scale=None, *, settled: bool = False, status=None):
    """x . weight^T, times `scale` (one BF16 value) if there is one: F.linear and a multiplication, as one kernel where it takes
    the operands and as these operations where it does not. `settled`: the caller vouches that the launch in front on this
    stream does not write the weights, which may then be read before it has ended. `status` (optional int32[1]) gets bit 1 set if
    a bounded wait inside the kernel gave up (the result is NaN then)."""
    if _plain(x, weight, *(() if scale is None else (scale,))) and _fits(x, weight):
        if scale is None or (scale.dtype == torch.bfloat16 and scale.shape == (1,) and scale.device == x.device):
            return _launcher(settled, status)(x, weight, None, scale)
    y = F.linear(x, weight)
    return y if scale is None else y * scale


def gated(x, gate, up, *, settled: bool = False, status=None):
    """silu(x . gate^T) * (x . up^T); `settled` and `status` as above."""
    if _plain(x, gate, up) and _fits(x, gate, up) and gate.shape == up.shape:
        return _launcher(settled, status)(x, gate, up, None)
    return F.silu(F.linear(x, gate)) * F.linear(x, up)
