"""Host side of the path: the modules that stand where the reference's expert runtime
stands.

* `ResidentExperts`  -- same constructor shape, tables and `forward(hidden, top_k_index,
  top_k_weights)` as the reference's OffloadedExperts (my_inkling/offloaded_experts.py:
  25-314), with every expert resident in HBM: no cache slots, no LRU, no copy kernel.
* `FusedMoE`         -- the whole of MyInklingMoE.forward (my_inkling/model.py:361-374): one token in
  one launch, several in the router, the plan and five launches around the grouped kernel (or, with banks
  that are not evenly spaced, router+plan, gate/up, down+combine), plus one all-reduce.
* `apply_resident_plan` / `apply_fused_moe_plan` install them into a model the way
  apply_offload_plan does (my_inkling/offloaded_experts.py:317-340).

Everything here is capture-safe: a module's buffers are made on first use for a given
token count and kept, a call's scratch comes from the caching allocator (under capture,
from the graph's pool), and a forward issues a fixed sequence of launches. One token and
several run different arithmetic (FP16 products on the CUDA cores; E2M1 digits on the
tensor cores), so a token's result may differ in its last bits with its company; its
routing does not.
"""
from __future__ import annotations

import struct

import torch
from torch import nn

from .kernels import (StackDescriptor, encode_bank_maps, encode_bf16_bank_maps, encode_shared_maps, expert_bank_names, expert_copy,
                      expert_gemm, expert_plan, expert_reduce, moe_decode, moe_grouped, routed_decode,
                      router_plan_forward, router_workspace, stack_supported)
from .kernels._abi import require_cuda
from .kernels._host import host
from .kernels.paired_all_reduce import all_reduce

# Up to this many tokens each route runs its own matrix-vector product
# (my_inkling/offloaded_experts.py:22).
MATVEC_TOKENS = 8
# Up to this many tokens are planned and projected together (the native calls' kMostTokens, see there).
GROUPED_TOKENS = 32768


def _group_of(device_mesh):
    if device_mesh is None:
        return None
    return device_mesh.get_group() if hasattr(device_mesh, "get_group") else device_mesh


def triton_cdiv(a: int, b: int) -> int:
    return (a + b - 1) // b


def _next_pow2(n: int) -> int:
    return 1 << (max(n, 1) - 1).bit_length()


class KeepsForGraphs:
    """A captured graph holds the addresses of a module's buffers and nothing that keeps them alive: buffers that a captured
    call has used are not given back when larger ones take their place, they stay as long as the module does."""

    _captured = False   # the present buffers are in a captured graph
    _kept = ()

    def __getstate__(self):   # (no graph has the addresses of a copy's buffers)
        return {k: v for k, v in self.__dict__.items() if k not in ("_captured", "_kept")}

    def _note_capture(self) -> None:
        if torch.cuda.is_current_stream_capturing():
            self.__dict__["_captured"] = True

    def _keep(self, *old) -> None:
        self.__dict__["_kept"] = (*self._kept, *(o for o in old if o is not None))

    def _replace(self, *old) -> None:
        """`old`, all that captured calls may have used, are about to be replaced."""
        if self._captured:
            self._keep(*old)
        self.__dict__["_captured"] = False


class ResidentExperts(KeepsForGraphs, nn.Module):
    """Drop-in for the routed-experts module with every expert's banks resident.

    `weights` is keyed by global expert id, each value the bank dictionary
    {gate_up_proj, gate_up_proj_scale, gate_up_proj_scale2, down_proj, down_proj_scale,
    down_proj_scale2} of CUDA tensors already sliced for this rank (slices of every
    expert on the FFN width), inputs replicated across ranks. With `quantized=False` the
    banks are the unquantised layer's {gate_up_proj BF16 [2f, d] (rows interleave gate and
    up), down_proj BF16 [d, f]} and the pointer table has stride 2
    (kernels/grouped_experts.py:9-22); that layer runs one matrix-vector product per route
    for one token, and at every token count where the banks are not evenly spaced in memory.
    """

    def __init__(self, hidden_dim: int, intermediate_dim: int, device_mesh, weights: dict, quantized: bool = True,
                 dtype=torch.bfloat16):
        super().__init__()
        self.device_mesh = device_mesh
        self.weights = weights  # keeps the allocations alive
        self.hidden_dim, self.intermediate_dim, self.dtype = hidden_dim, intermediate_dim, dtype
        self.quantized = bool(quantized)
        names = expert_bank_names(self.quantized)
        self.stride = len(names)
        ids = sorted(weights)
        self.start, self.local, self.max_expert = ids[0], len(ids), ids[-1]
        assert ids == list(range(self.start, self.start + self.local))
        first = weights[ids[0]]
        self.device = first[names[0]].device
        assert all(w.is_contiguous() and w.is_cuda for e in weights.values() for w in e.values())
        packed = 2 if self.quantized else 1
        assert first["gate_up_proj"].shape == (2 * intermediate_dim, hidden_dim // packed)
        assert first["down_proj"].shape == (hidden_dim, intermediate_dim // packed)
        assert first["gate_up_proj"].dtype == (torch.uint8 if self.quantized else torch.bfloat16)
        self.num_slots = 0
        i32 = dict(dtype=torch.int32, device=self.device)
        self.sources = torch.tensor([[weights[e][n].data_ptr() for n in names] for e in ids],
                                    dtype=torch.int64, device=self.device)
        # banks of one kind evenly spaced in memory (one allocation per kind, say): (address of the first,
        # byte distance) per kind, for the TMA descriptors of the one-launch kernel; otherwise None
        kinds = ("gate_up_proj", "gate_up_proj_scale", "down_proj", "down_proj_scale") if self.quantized else ("gate_up_proj", "down_proj")
        self.bank_layout = self._even_spacing([[weights[e][n].data_ptr() for e in ids] for n in kinds],
                                              [first[n].numel() * first[n].element_size() for n in kinds])
        # TMA descriptors of the banks for the grouped tensor-core kernel, where they are evenly spaced
        self.bank_maps = None
        step, widest = (256 if self.quantized else 128), max(hidden_dim, intermediate_dim)
        if self.bank_layout is not None and hidden_dim % step == 0 and intermediate_dim % step == 0 and widest <= 4096 and self.local <= 1024:
            encode = encode_bank_maps if self.quantized else encode_bf16_bank_maps
            self.bank_maps = encode(self.bank_layout, self.local, hidden_dim, intermediate_dim, self.device)
        self.resident = torch.ones(self.local, **i32)
        self.destinations = torch.zeros((0, self.stride), dtype=torch.int64, device=self.device)
        self.slot_experts = torch.full((0,), -1, **i32)
        self.ages = torch.zeros(0, **i32)
        self.clock = torch.zeros((), **i32)
        self.copy_experts = torch.empty(0, **i32)
        self.pointers = torch.zeros((self.max_expert + 1) * self.stride, dtype=torch.int64, device=self.device)
        # decode reads the table without a plan when the caller skips it: start fully active
        self.pointers.view(-1, self.stride)[self.start:self.start + self.local] = self.sources
        self.experts = torch.empty(self.local, **i32)
        self.counts = torch.empty(self.local, **i32)
        self.status = torch.zeros(1, **i32)
        self.capacity = 0
        self.rows = self.activated = self.down = None

    # What the native calls need of this module is taken down once (`record_fields`); replacing a tensor, or growing the
    # buffers, makes a new one, and so does a call that finds a tensor's storage exchanged.
    _native = None
    generation = 0

    def __setattr__(self, name, value):
        if isinstance(value, torch.Tensor) or name in ("weights", "capacity"):
            self.__dict__["_native"] = None
            self.__dict__["generation"] = self.generation + 1
        super().__setattr__(name, value)

    def __getstate__(self):   # copies and pickles make their own record
        return {k: v for k, v in super().__getstate__().items() if k != "_native"}

    def record_fields(self) -> dict:
        return dict(hidden=self.hidden_dim, width=self.intermediate_dim, start=self.start, local=self.local, stride=self.stride,
                    capacity=self.capacity, max_expert=self.max_expert, quantized=int(self.quantized), sources=self.sources,
                    pointers=self.pointers, experts=self.experts, counts=self.counts, rows=self.rows,
                    activated=self.activated, down=self.down, status=self.status, bank_maps=self.bank_maps)

    @staticmethod
    def _even_spacing(addresses: list[list[int]], sizes: list[int]):
        layout = []
        for per_expert, size in zip(addresses, sizes):
            stride = per_expert[1] - per_expert[0] if len(per_expert) > 1 else size
            if stride < size or stride % 16 or per_expert[0] % 16:
                return None
            if any(b - a != stride for a, b in zip(per_expert, per_expert[1:])):
                return None
            layout.append((per_expert[0], stride))
        return layout

    def _reserve(self, routes: int) -> None:
        if routes > self.capacity:
            capacity, options = _next_pow2(routes), dict(dtype=self.dtype, device=self.device)
            self._replace(self.rows, self.activated, self.down)
            self.capacity, self.rows, self.activated, self.down = 0, None, None, None   # (so it stays if memory runs out here)
            self.rows = torch.empty((self.local, capacity), dtype=torch.int32, device=self.device)
            self.activated = torch.empty((capacity, self.intermediate_dim), **options)
            self.down = torch.empty((capacity, self.hidden_dim), **options)
            self.capacity = capacity
        self._note_capture()

    def _plan(self, indices) -> None:
        routes = indices.numel()
        expert_plan[(1,)](indices, self.sources, self.resident, self.destinations, self.slot_experts, self.ages,
                          self.clock, self.copy_experts, self.pointers, self.experts, self.counts, self.rows,
                          self.start, self.local, self.num_slots, self.stride, routes, self.capacity,
                          _next_pow2(self.local), 1, _next_pow2(routes), num_warps=4)
        expert_copy[(128, 0)](self.sources, self.destinations, self.copy_experts, (), self.stride, 1024, 128)

    def grouped_supported(self) -> bool:
        """Banks the grouped tensor-core path takes: evenly spaced in memory, or NVFP4 banks anywhere whose contraction
        widths are multiples of 128."""
        return self.bank_maps is not None or (self.quantized and self.hidden_dim % 128 == 0 and self.intermediate_dim % 128 == 0)

    def _project(self, x, indices, weights, output) -> None:
        """GEMV per route for one token (up to MATVEC_TOKENS where the banks are not evenly spaced), grouped tensor-core
        GEMMs above (my_inkling/offloaded_experts.py:224-296). `output` must be zero on entry."""
        tokens = x.shape[0]
        if tokens > (1 if self.bank_maps is not None else MATVEC_TOKENS) and self.grouped_supported():
            self._project_grouped(x, indices, weights, output)
            return
        if tokens <= MATVEC_TOKENS:
            routed_decode(x, indices, weights, self.pointers, self.activated, output, self.max_expert, self.quantized, status=self.status)
            return
        for t0 in range(0, tokens, MATVEC_TOKENS):
            t1 = min(tokens, t0 + MATVEC_TOKENS)
            routed_decode(x[t0:t1], indices[t0:t1], weights[t0:t1], self.pointers,
                          self.activated[t0 * indices.shape[1]:], output[t0:t1], self.max_expert, self.quantized,
                          status=self.status)

    def grouped(self, x, indices, weights, output=None, output_bf16=None, shared_maps=None, gammas=None, n_shared: int = 0) -> None:
        """Both projections and the weighted sum over the plan's groups in one call (banks with `bank_maps`); with
        `shared_maps` the block's shared experts too. The outputs are overwritten."""
        moe_grouped(x, indices, weights, self.pointers, self.experts, self.rows, self.counts, self.bank_maps, self.activated,
                    self.down, output=output, output_bf16=output_bf16, groups=min(indices.numel(), self.local), start=self.start,
                    local=self.local, capacity=self.capacity, max_expert=self.max_expert, quantized=self.quantized,
                    shared_maps=shared_maps, gammas=gammas, n_shared=n_shared, status=self.status)

    def _project_grouped(self, x, indices, weights, output) -> None:
        """Both projections as grouped tensor-core GEMMs over the plan's groups, then the weighted
        sum per token (my_inkling/offloaded_experts.py:249-296). `output` must be zero on entry."""
        if self.bank_maps is not None:
            self.grouped(x, indices, weights, output)
            return
        tokens, routes, top_k = x.shape[0], indices.numel(), indices.shape[1]
        groups = min(routes, self.local)
        for projection, inputs, target, n, k in (
                (0, x, self.activated, 2 * self.intermediate_dim, self.hidden_dim),
                (1, self.activated, self.down, self.hidden_dim, self.intermediate_dim)):
            grid = (triton_cdiv(routes, 16), triton_cdiv(n, 64), groups)
            expert_gemm[grid](inputs, self.pointers, self.experts, self.rows, self.counts, target, self.capacity,
                              n, k, top_k, projection, True, self.stride, 16, 64, 64, status=self.status)
        expert_reduce[(tokens, triton_cdiv(self.hidden_dim, 256))](
            self.down, indices, weights, self.pointers, output, self.hidden_dim, top_k, self.stride,
            self.max_expert, 256)

    def forward(self, hidden_states, top_k_index, top_k_weights):
        if self.device_mesh is None and self.bank_maps is not None and hidden_states.shape[0] > 1 and hidden_states.dim() == 2:
            self._reserve(top_k_index.numel())
            top_k = top_k_index.shape[1]
            out = NotImplemented
            while out is NotImplemented:
                if self._native is None or self._native[0] != top_k:
                    self.__dict__["_native"] = (top_k, host().make_block(dict(self.record_fields(), top_k=top_k)))
                out = host().run_experts(self._native[1], hidden_states, top_k_index, top_k_weights)
                if out is NotImplemented:
                    self.__dict__["_native"] = None
            return out
        final = torch.zeros_like(hidden_states, dtype=torch.float32)
        self._reserve(top_k_index.numel())
        x, index, weights = hidden_states.contiguous(), top_k_index.contiguous(), top_k_weights.contiguous()
        if x.shape[0] <= GROUPED_TOKENS:   # (a decode call is bound by the host: views of all of it would cost a fifth)
            self._plan(index)
            self._project(x, index, weights, final)
        else:
            for t0 in range(0, x.shape[0], GROUPED_TOKENS):
                part = slice(t0, t0 + GROUPED_TOKENS)
                self._plan(index[part])
                self._project(x[part], index[part], weights[part], final[part])
        final = all_reduce(final, _group_of(self.device_mesh))
        return final.to(hidden_states.dtype)

    def check_status(self) -> None:
        """Host read (synchronises): raises if any call since the last check routed to an
        expert id outside [0, max_expert] (bit 0 of the status word), or if a bounded wait
        inside a streaming or grouped kernel gave up (bit 1: that call's output is partial).
        Call outside graph capture."""
        flags = int(self.status.item())
        self.status.zero_()
        if flags & 2:
            raise RuntimeError("ResidentExperts: a bounded wait inside a kernel timed out; the output of that call is invalid")
        if flags & 1:
            raise RuntimeError("ResidentExperts: a route named an expert id outside the pointer table")


class FusedMoE(KeepsForGraphs, nn.Module):
    """Router + routed NVFP4 experts + shared BF16 experts + one all-reduce.

    Parameters are this rank's: router replicated, shared experts and routed experts
    sliced on the FFN width. forward(hidden [bs, s, d]) -> [bs, s, d] in the input dtype.
    """

    # True: one token also takes the separate launches (router + plan, gate/up, down) and the NCCL all-reduce,
    # the shape of the reference's block (my_inkling/offloaded_experts.py:298-314); used as the baseline of A/B runs
    separate_launches = False

    def __init__(self, router_weight, router_bias, global_scale, route_scale: float, top_k: int,
                 shared_gate, shared_up, shared_down, experts: ResidentExperts, device_mesh=None):
        super().__init__()
        self.router_weight, self.router_bias, self.global_scale = router_weight, router_bias.float(), global_scale
        self.route_scale, self.top_k = float(route_scale), top_k
        self.shared_gate, self.shared_up, self.shared_down = shared_gate, shared_up, shared_down
        self.n_shared = shared_gate.shape[0]
        assert experts.quantized, "FusedMoE takes NVFP4 experts; an unquantised layer keeps its own block around ResidentExperts"
        self.experts = experts
        self.device_mesh = device_mesh
        self._tokens = 0
        self._of_capture = False   # the buffers were made under capture: their zeros are filled in by that graph alone
        self._fused = None   # one-launch descriptor for a single token, built on first use
        self._maps = self._maps_of = None
        if experts.bank_maps is not None and self.n_shared and self._shared_as_expected() and all(
                w.is_cuda for w in (shared_gate, shared_up, shared_down)):
            self._shared_maps()   # here, so that a first call may be one under graph capture

    _native = None   # what the native calls know of this block, and the experts' generation it was taken down at

    def __setattr__(self, name, value):
        if isinstance(value, (torch.Tensor, StackDescriptor)) or name in ("experts", "top_k", "n_shared", "route_scale", "_fused"):
            self.__dict__["_native"] = None
        super().__setattr__(name, value)

    def __getstate__(self):   # copies and pickles make their own record and table
        return dict({k: v for k, v in super().__getstate__().items() if k != "_native"}, _fused=None)

    def _shared_as_expected(self) -> bool:
        d, f, n = self.experts.hidden_dim, self.experts.intermediate_dim, self.n_shared
        gate, up, down = self.shared_gate, self.shared_up, self.shared_down
        return (gate.shape == up.shape == (n, f, d) and down.shape == (n, d, f)
                and all(t.dtype == torch.bfloat16 and t.is_contiguous() for t in (gate, up, down)))

    def _check(self) -> None:
        """The block's tensors as the kernels read them, by address alone: made sure of whenever addresses are taken down."""
        weight, bias, scale = self.router_weight, self.router_bias, self.global_scale
        assert weight.dtype == scale.dtype == torch.bfloat16 and bias.dtype == torch.float32
        assert weight.dim() == 2 and weight.shape[1] == self.experts.hidden_dim and bias.shape == (weight.shape[0] - self.n_shared,)
        assert scale.numel() >= 1 and all(t.is_contiguous() for t in (weight, bias, scale))
        assert self._shared_as_expected()
        require_cuda(weight, bias, scale, self.shared_gate, self.shared_up, self.shared_down)

    def _record(self, one_token: bool):
        """The record for several tokens, with `one_token` also the one-launch kernel's table (made on the first such call only)."""
        self._check()
        ex = self.experts
        ex._reserve(self._tokens * self.top_k)   # (experts that were put in the place of others may have less room)
        fields = dict(ex.record_fields() if ex.bank_maps is not None else dict(hidden=ex.hidden_dim, width=ex.intermediate_dim),
                      tokens=self._tokens if ex.bank_maps is not None else 1, routed=self.router_weight.shape[0] - self.n_shared,
                      shared=self.n_shared, top_k=self.top_k, router_weight=self.router_weight, router_bias=self.router_bias,
                      global_scale=self.global_scale, topk_weights=self.topk_weights, topk_indices=self.topk_indices,
                      gammas=self.gammas, workspace=self.workspace, workspace_bytes=self.workspace.numel(), partial=self.partial,
                      shared_gate=self.shared_gate, shared_up=self.shared_up, shared_down=self.shared_down,
                      route_scale_bits=struct.unpack("<I", struct.pack("<f", self.route_scale))[0])
        if ex.bank_maps is not None and self.n_shared:
            fields["shared_maps"] = self._shared_maps()
        if one_token:
            if self._fused is None:
                self._fused = self._one_launch()
            f = self._fused
            fields.update(table=f.table, scratch=f.scratch, scratch_bytes=f.scratch.numel(), stack_status=f.status,
                          stack_flags=2 if f.bank_maps is not None else 0)
        return host().make_block(fields)

    def _one_launch(self) -> StackDescriptor:
        # across ranks the kernel delivers and sums the partials itself: no separate collective
        ex = self.experts
        return StackDescriptor([self.block_descriptor()], ex.hidden_dim, ex.intermediate_dim, ex.local, self.n_shared, self.top_k,
                               self.router_weight.device, group=_group_of(self.device_mesh))

    def _call_native(self, tokens: int, x, want_partial: bool):
        """The block in one native call, or NotImplemented where the launches are put together here: several ranks, banks that
        are not evenly spaced, one token without the one-launch kernel."""
        if self.device_mesh is not None or (tokens == 1 and self.separate_launches):
            return NotImplemented
        ex = self.experts
        one = tokens == 1
        for _ in range(2):   # (again where the record turns out to be of storage that has been exchanged)
            native = self._native
            if native is None or native[0] != ex.generation or not native[2 if one else 3]:
                if not (self.one_launch_supported() if one else ex.bank_maps is not None):
                    return NotImplemented
                record = self._record(one)
                native = self.__dict__["_native"] = (ex.generation, record, one, ex.bank_maps is not None)
            out = host().run_block(native[1], x, want_partial)
            if out is not NotImplemented:
                return out
            if self._captured:
                self._keep(self._fused)
            self._fused = None   # (drops the record too)
        raise RuntimeError("FusedMoE: a tensor's storage was exchanged during the call")

    def block_descriptor(self, norm_weight=None) -> dict:
        """This block as the one-launch kernel takes it (addresses of the module's tensors)."""
        self._check()
        if not self._tokens:
            self._reserve(1)
        ex = self.experts
        return dict(router_weight=self.router_weight, router_bias=self.router_bias, global_scale=self.global_scale,
                    sources=ex.sources, shared_gate=self.shared_gate, shared_up=self.shared_up,
                    shared_down=self.shared_down, norm_weight=norm_weight, topk_indices=self.topk_indices,
                    topk_weights=self.topk_weights, gammas=self.gammas, route_scale=self.route_scale,
                    bank_layout=ex.bank_layout if ex.start == 0 else None)

    def world_size(self) -> int:
        group = _group_of(self.device_mesh)
        if group is not None and torch.distributed.is_available() and torch.distributed.is_initialized():
            return torch.distributed.get_world_size(group)
        return 1

    def one_launch_supported(self) -> bool:
        """One token through this block in one persistent launch (the all-reduce, if any,
        follows as its own collective)."""
        ex = self.experts
        return ex.start == 0 and stack_supported(ex.hidden_dim, ex.intermediate_dim, ex.local, self.n_shared,
                                                 self.top_k)

    def _reserve(self, tokens: int) -> None:
        """Buffers for `tokens` tokens. Those of a first call under capture serve that call alone: the router's counters in them
        are cleared by that graph, when it is replayed, so the next call, eager or of another graph, has its own."""
        capturing = torch.cuda.is_current_stream_capturing()
        if tokens <= self._tokens and not self._of_capture and not capturing:
            return
        if tokens > self._tokens or self._of_capture:
            if self._tokens:
                self._replace(self.topk_weights, self.topk_indices, self.gammas, self.shared_activated, self.workspace, self.partial, self._fused)
            self._tokens = 0            # (so it stays if memory runs out here)
            self._fused = None          # descriptors hold addresses of the buffers replaced here
            self.topk_weights = self.topk_indices = self.gammas = self.shared_activated = self.workspace = self.partial = None
            self.experts._reserve(tokens * self.top_k)
            dev, bf = self.router_weight.device, torch.bfloat16
            self.generation = getattr(self, "generation", 0) + 1
            self.topk_weights = torch.empty(tokens, self.top_k, dtype=bf, device=dev)
            self.topk_indices = torch.empty(tokens, self.top_k, dtype=torch.int64, device=dev)
            self.gammas = torch.empty(tokens, self.n_shared, dtype=bf, device=dev)
            self.shared_activated = torch.empty(tokens * self.n_shared, self.experts.intermediate_dim, dtype=bf, device=dev)
            self.workspace = router_workspace(tokens, self.router_weight.shape[0], dev)
            self.partial = torch.empty(tokens, self.experts.hidden_dim, dtype=torch.float32, device=dev)
            self._of_capture = capturing
            self._tokens = tokens
        self.experts._note_capture()
        self._note_capture()

    def _shared_maps(self):
        """TMA descriptors of the shared experts, made when they are first needed (and again if the tensors are replaced)."""
        at = (self.shared_gate.data_ptr(), self.shared_up.data_ptr(), self.shared_down.data_ptr())
        if self._maps_of != at:
            assert self._shared_as_expected()
            self._keep(self._maps)   # (a graph, or another stream, may still read them: 384 bytes)
            self._maps, self._maps_of = encode_shared_maps(self.shared_gate, self.shared_up, self.shared_down), at
        return self._maps

    def route(self, flat, t0: int = 0):
        """Router and plan for `flat` [t, d]; fills the module's routing buffers from token t0 on."""
        t1 = t0 + flat.shape[0]
        ex = self.experts
        args = (flat, self.router_weight, self.router_bias, self.global_scale, self.route_scale, self.top_k,
                self.n_shared, self.topk_weights[t0:t1], self.topk_indices[t0:t1], self.gammas[t0:t1], self.workspace)
        router_plan_forward(*args, ex.sources, ex.pointers, ex.experts, ex.counts, ex.rows, ex.start,
                            ex.local, ex.stride, ex.capacity)

    def forward(self, hidden_states):
        shape = hidden_states.shape
        tokens = hidden_states.numel() // shape[-1]
        self._reserve(tokens)
        out = self._call_native(tokens, hidden_states, False)
        if out is not NotImplemented:
            return out
        flat = hidden_states.reshape(-1, shape[-1]).contiguous()
        return self._partial(flat).to(hidden_states.dtype).view(shape)

    def forward_partial(self, flat):
        """flat BF16 [t, d] -> the all-reduced FP32 layer output [t, d] (a view of the
        module's own buffer, overwritten by the next call)."""
        t = flat.shape[0]
        self._reserve(t)
        if self._call_native(t, flat, True) is not NotImplemented:
            return self.partial[:t]
        return self._partial(flat)

    def _partial(self, flat):
        t, ex = flat.shape[0], self.experts
        if t == 1 and self.one_launch_supported() and not self.separate_launches:
            if self._fused is None:
                self._fused = self._one_launch()
            self._fused.decode(flat, self.partial[:1])
            return self.partial[:1]
        if t > 1 and ex.bank_maps is not None:
            for t0 in range(0, t, GROUPED_TOKENS):
                t1 = min(t, t0 + GROUPED_TOKENS)
                self.route(flat[t0:t1], t0)
                ex.grouped(flat[t0:t1], self.topk_indices[t0:t1], self.topk_weights[t0:t1], self.partial[t0:t1],
                           shared_maps=self._shared_maps() if self.n_shared else None, gammas=self.gammas[t0:t1], n_shared=self.n_shared)
            return all_reduce(self.partial[:t], _group_of(self.device_mesh))
        self.route(flat)
        for t0 in range(0, t, MATVEC_TOKENS):
            t1 = min(t, t0 + MATVEC_TOKENS)
            moe_decode(flat[t0:t1], self.topk_indices[t0:t1], self.topk_weights[t0:t1], ex.pointers,
                       ex.activated[t0 * self.top_k:], self.shared_gate, self.shared_up, self.shared_down,
                       self.gammas[t0:t1], self.shared_activated[t0 * self.n_shared:], self.partial[t0:t1],
                       ex.max_expert, status=ex.status)
        return all_reduce(self.partial[:t], _group_of(self.device_mesh))


def apply_resident_plan(model: nn.Module, device_mesh, expert_state_dict: dict) -> nn.Module:
    """Replace every routed-experts module (a module with `gate_up_proj`, `down_proj`,
    `hidden_dim` and `intermediate_dim`, i.e. the reference's MyInklingExperts) named in
    `expert_state_dict` by ResidentExperts over this rank's banks."""
    for name, module in list(model.named_modules()):
        if name in expert_state_dict and hasattr(module, "intermediate_dim") and hasattr(module, "hidden_dim"):
            banks = expert_state_dict[name]
            quantized = "gate_up_proj_scale" in next(iter(banks.values()))   # offloaded_experts.py:333
            model.set_submodule(name, ResidentExperts(module.hidden_dim, module.intermediate_dim, device_mesh,
                                                      banks, quantized))
    return model


def apply_fused_moe_plan(model: nn.Module, device_mesh, expert_state_dict: dict) -> nn.Module:
    """Replace every MoE block (a module with `gate`, `experts` and `shared_experts`
    children, i.e. the reference's MyInklingMoE) whose experts are named in
    `expert_state_dict` by FusedMoE. The block's own router and (already sharded)
    shared-expert parameters are reused."""
    for name, module in list(model.named_modules()):
        key = name + ".experts"
        if key in expert_state_dict and all(hasattr(module, a) for a in ("gate", "experts", "shared_experts")):
            gate, shared, old = module.gate, module.shared_experts, module.experts
            experts = ResidentExperts(old.hidden_dim, old.intermediate_dim, device_mesh, expert_state_dict[key])
            fused = FusedMoE(gate.weight.data, gate.e_score_correction_bias.data, gate.global_scale.data,
                             gate.route_scale, gate.top_k, shared.gate_proj.data, shared.up_proj.data,
                             shared.down_proj.data, experts, device_mesh)
            model.set_submodule(name, fused)
    return model
