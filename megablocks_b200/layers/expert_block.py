"""The routed expert computation of one device as one native call, or two where it is differentiated.

Plan, permutation, expert GEMMs and weighted un-permutation are the kernels that the ops of
``megablocks_b200.ops`` launch one by one; ``csrc/expert_block.cpp`` launches them back to back, and two
autograd nodes (the experts, the un-permutation) stand for what are otherwise three.  That takes the
Python between the launches out, which is what small calls are made of: a decode step (8 tokens, 64
experts) has 60 us of kernels in 205 us, a 256-token training pass 110 in 730.

:func:`route` says whether a layer's call may take this path: stock steps and expert modules without
hooks, 16-bit CUDA tensors that the kernels take, an activation they know, none of the modes that give an
autograd node a meaning of its own (autocast, tracing, functorch, forward-mode).  Everything else runs
op by op as before.
"""

from typing import Any

import torch
from torch.autograd import forward_ad

from megablocks_b200._ext import ext
from megablocks_b200.layers.fused_mlp import capacity_act
from megablocks_b200.ops import gg as G
from megablocks_b200.utils import debug


class _Experts(torch.autograd.Function):
    """Plan, permutation and expert GEMMs: the copies' results in expert order.  ``plan`` is a list that
    receives ``(tokens_per_expert, indices, inverse, bins)``; as outputs of the node they would each cost the
    host a wrapper."""

    @staticmethod
    def forward(ctx: Any, x, top_experts, w1, w2, v1, gemm_bins, plan, num_experts, top_k, act, capacity,
                memory_optimized, wgrad_scale):
        need = ctx.needs_input_grad
        keep = need[0] or need[2] or need[3] or need[4]
        y, counts, indices, inverse, bins, *kept = ext().expert_rows_forward(
            x, top_experts, w1, w2, v1, gemm_bins, num_experts, top_k, act, capacity, keep, G._PAIR_MODE)
        if keep:
            rows, z1, z2, h = kept
            ctx.save_for_backward(w1, w2, v1, gemm_bins, inverse, bins, rows, z1, z2 if v1 is not None else None,
                                  None if memory_optimized else h)
        ctx.top_k, ctx.act, ctx.capacity, ctx.wgrad_scale = top_k, act, capacity, wgrad_scale
        ctx.set_materialize_grads(False)
        plan += (counts, indices, inverse, bins)
        return y

    @staticmethod
    def backward(ctx: Any, dy):
        if dy is None:
            return (None,) * 13
        w1, w2, v1, gemm_bins, inverse, bins, rows, z1, z2, h = ctx.saved_tensors
        need = ctx.needs_input_grad
        needs = [need[0], need[2], need[3], need[4]]
        sink = G._GRAD_NORM_SINK
        views, slots = [None, None, None], [None, None, None]
        if sink is not None:
            wanted = [k for k in (1, 0, 2) if needs[1 + k] and (k < 2 or v1 is not None)]     # launch order
            for k, (slot, view) in zip(wanted, sink.reserve(len(wanted))):
                slots[k], views[k] = slot, view
        dx, *dw = ext().expert_rows_backward(dy.contiguous(), inverse, bins, gemm_bins, rows, z1, z2, h, w1, w2, v1,
                                             needs, views, ctx.top_k, ctx.act, ctx.wgrad_scale, ctx.capacity,
                                             G._PAIR_MODE)
        for k in (1, 0, 2):
            if slots[k] is not None:
                sink._record(dw[k], slots[k])
        return (dx, None, *dw) + (None,) * 8


def _hooked(module: torch.nn.Module) -> bool:
    return bool(module._forward_hooks or module._forward_pre_hooks or module._backward_hooks
                or module._backward_pre_hooks or 'forward' in module.__dict__)


def special_mode() -> bool:
    """A mode in which calling the kernels without (or with another) autograd node would change a result."""
    return (torch.is_autocast_enabled('cuda') or torch.jit.is_tracing() or forward_ad._current_level >= 0
            or torch._C._functorch.peek_interpreter_stack() is not None or debug.enabled()
            or torch.nn.modules.module._has_any_global_hook())


def route(x, expert_weights, top_experts, mlp, w1, w2, v1, bias, activation_fn) -> bool:
    """Whether :func:`expert_block` takes this call.  ``w1`` and ``w2`` are 3-D; ``bias`` may be ``None``."""
    dtype = x.dtype
    if not (x.is_cuda and dtype in (torch.bfloat16, torch.float16) and x.numel() > 0):
        return False
    experts, hidden = w2.shape[0], w2.shape[2]
    ffn = w2.shape[1]
    for t in (w1, w2, v1, expert_weights, bias):
        if t is not None and not (t.dtype == dtype and t.device == x.device and t.is_contiguous()
                                  and not hasattr(t, 'to_local')):
            return False
    if (hidden % 8 or ffn % 8 or hidden < 64 or ffn < 64 or experts > 1024 or (v1 is not None and ffn < 128)
            or hidden != x.shape[-1] or top_experts.numel() != expert_weights.numel()
            or (bias is not None and (bias.data_ptr() % 16 or bias.shape != (hidden,)))):
        return False
    return G.activation_id(activation_fn) is not None and not _hooked(mlp) and not special_mode()


def expert_block(x, expert_weights, top_experts, w1, w2, v1, bias, gemm_bins, num_experts, top_k, activation_fn,
                 capacity, memory_optimized, wgrad_scale):
    """``(out[tokens, hidden], tokens_per_expert)`` for calls that :func:`route` accepts."""
    x, top_experts = x.reshape(-1, x.shape[-1]).contiguous(), top_experts.contiguous()
    act = capacity_act(activation_fn) if capacity > 0 else G.activation_id(activation_fn)
    tensors = (x, expert_weights, w1, w2, v1, bias)
    if not (torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)):
        out, counts = ext().expert_block_forward(x, top_experts, expert_weights, w1, w2, v1, bias, gemm_bins, num_experts,
                                                 top_k, act, capacity, G._PAIR_MODE)
        return out, counts
    plan = []
    y = _Experts.apply(x, top_experts, w1, w2, v1, gemm_bins, plan, num_experts, top_k, act, capacity,
                       memory_optimized, wgrad_scale)
    counts, indices, inverse, bins = plan
    return ext().expert_combine(y, expert_weights, bias, indices, inverse, bins, top_k, capacity), counts
