"""The routed expert computation of one device as a single native call.

Plan, permutation, expert GEMMs and weighted un-permutation are the kernels that the ops of
``megablocks_b200.ops`` launch one by one; ``csrc/expert_block.cpp`` launches them back to back, and one
autograd node stands for what are otherwise three.  That takes the Python between the launches out,
which is what small calls are made of: a decode step (8 tokens, 64 experts) has 60 us of kernels in 205
us, a 256-token training pass 110 in 730.

:func:`route` says whether a layer's call may take this path: stock steps and expert modules without
hooks, 16-bit CUDA tensors that the kernels take, an activation they know, none of the modes that give an
autograd node a meaning of its own (autocast, tracing, functorch, forward-mode).  Everything else runs
op by op as before.
"""

from typing import Any

import torch
from torch.autograd import forward_ad

from megablocks_b200._ext import ext
from megablocks_b200.ops import gg as G
from megablocks_b200.utils import debug


class _ExpertBlock(torch.autograd.Function):

    @staticmethod
    def forward(ctx: Any, x, weights, top_experts, w1, w2, v1, bias, gemm_bins, num_experts, top_k, act, capacity,
                memory_optimized, wgrad_scale):
        out, counts, indices, inverse, bins, rows, y, z1, z2, h = ext().expert_block_forward(
            x, top_experts, weights, w1, w2, v1, bias, gemm_bins, num_experts, top_k, act, capacity, True, G._PAIR_MODE)
        ctx.save_for_backward(weights, w1, w2, v1, gemm_bins, indices, inverse, bins, rows, y, z1,
                              z2 if v1 is not None else None, None if memory_optimized else h)
        ctx.top_k, ctx.act, ctx.capacity, ctx.wgrad_scale = top_k, act, capacity, wgrad_scale
        ctx.mark_non_differentiable(counts)
        ctx.set_materialize_grads(False)        # no zero tensor for the counts
        return out, counts

    @staticmethod
    def backward(ctx: Any, dout, _dcounts):
        weights, w1, w2, v1, gemm_bins, indices, inverse, bins, rows, y, z1, z2, h = ctx.saved_tensors
        if dout is None:
            return (None,) * 14
        need = ctx.needs_input_grad
        needs = [need[0], need[1], need[3], need[4], need[5], need[6]]
        sink = G._GRAD_NORM_SINK
        views, slots = [None, None, None], [None, None, None]
        if sink is not None:
            wanted = [k for k in (1, 0, 2) if needs[2 + k] and (k < 2 or v1 is not None)]     # launch order
            for k, (slot, view) in zip(wanted, sink.reserve(len(wanted))):
                slots[k], views[k] = slot, view
        dx, dweights, *dw, dbias = ext().expert_block_backward(
            dout.contiguous(), indices, inverse, bins, gemm_bins, rows, y, z1, z2, h, weights, w1, w2, v1, needs, views,
            ctx.top_k, ctx.act, ctx.wgrad_scale, ctx.capacity, G._PAIR_MODE)
        for k in (1, 0, 2):
            if slots[k] is not None:
                sink._record(dw[k], slots[k])
        return (dx, dweights, None, *dw, dbias, None, None, None, None, None, None, None)


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
            or (bias is not None and bias.data_ptr() % 16)):
        return False
    return G.activation_id(activation_fn) is not None and not _hooked(mlp) and not special_mode()


def expert_block(x, expert_weights, top_experts, w1, w2, v1, bias, gemm_bins, num_experts, top_k, activation_fn,
                 capacity, memory_optimized, wgrad_scale):
    """``(out[tokens, hidden], tokens_per_expert)`` for calls that :func:`route` accepts."""
    x = x.reshape(-1, x.shape[-1]).contiguous()
    act = G.activation_id(activation_fn)
    tensors = (x, expert_weights, w1, w2, v1, bias)
    if not (torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)):
        out, counts = ext().expert_block_forward(x, top_experts, expert_weights, w1, w2, v1, bias, gemm_bins, num_experts,
                                                 top_k, act, capacity, False, G._PAIR_MODE)
        return out, counts
    return _ExpertBlock.apply(x, expert_weights, top_experts, w1, w2, v1, bias, gemm_bins, num_experts, top_k, act,
                              capacity, memory_optimized, wgrad_scale)
