"""Drop-in counterpart of the reference's `kernels` package for the NVFP4
routed-expert path: same names, same call signatures, sm_100a library underneath."""
from .expert_planner import expert_copy, expert_plan
from .grouped_experts import (block_scaled_supported, encode_bank_maps, encode_bf16_bank_maps, encode_shared_maps,
                              expert_bank_names, expert_gemm, expert_reduce, moe_grouped)
from .attention import decode_attention, update_kv
from .linear import gated, linear
from .routed_decode import add_rmsnorm, attention_heads, moe_decode, rmsnorm, routed_decode, short_conv, short_conv_norm
from .stack import StackDescriptor, set_wait_limit, stack_supported
from .router import router_forward, router_forward_static, router_plan_forward, router_workspace

__all__ = [
    "add_rmsnorm",
    "attention_heads",
    "block_scaled_supported",
    "encode_bank_maps",
    "encode_bf16_bank_maps",
    "encode_shared_maps",
    "expert_bank_names",
    "expert_copy",
    "expert_gemm",
    "expert_reduce",
    "expert_plan",
    "moe_decode",
    "moe_grouped",
    "routed_decode",
    "StackDescriptor",
    "set_wait_limit",
    "short_conv",
    "short_conv_norm",
    "rmsnorm",
    "linear",
    "gated",
    "decode_attention",
    "update_kv",
    "stack_supported",
    "router_forward",
    "router_forward_static",
    "router_plan_forward",
    "router_workspace",
]
