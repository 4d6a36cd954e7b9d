"""Layer-level checks: shapes, numerics against dense per-expert loops, losses, state dicts.

Mirrors the reference layer tests (tests/layers/dmoe_test.py:17-241, moe_test.py:155-199,
glu_test.py:64-123) and adds backward numerics, which the reference only smoke-tests.
"""

import gc
import math
from functools import partial

import pytest
import torch
import torch.nn.functional as F
from conftest import DEVICES

import megablocks_b200 as mb
from megablocks_b200 import ops
from megablocks_b200.layers import mlp as mlp_mod
from megablocks_b200.layers import moe as moe_mod
from megablocks_b200.layers import router as router_mod
from megablocks_b200.layers.arguments import from_megatron
from megablocks_b200.ops import gg as ops_gg

CONFIGS = [(8, 16, 128, 1, 1), (8, 16, 128, 2, 1), (8, 16, 128, 4, 1), (8, 16, 128, 4, 2), (8, 16, 256, 8, 4),
           (2, 64, 128, 8, 2), (1, 33, 128, 5, 3)]


def _args(device, hs=128, ffn=None, ne=8, top_k=2, **kw):
    half = device == 'cuda'
    base = dict(hidden_size=hs, ffn_hidden_size=ffn or 2 * hs, moe_num_experts=ne, moe_top_k=top_k, fp16=False,
                bf16=half, device=torch.device(device), moe_capacity_factor=1, memory_optimized_mlp=False,
                init_method=partial(torch.nn.init.normal_, mean=0.0, std=0.1))
    base.update(kw)
    return mb.Arguments(**base)


def _tol(device):
    return dict(rtol=3e-2, atol=3e-2) if device == 'cuda' else dict(rtol=1e-5, atol=1e-5)


def dense_oracle(layer, x, mlp_type='mlp'):
    """Per-expert dense loop in fp32: the definition of the dropless layer."""
    args = layer.experts.args
    E, k, h = args.moe_num_experts, args.moe_top_k, args.hidden_size
    xf = x.reshape(-1, h).float()
    wr = layer.router.layer.weight.float()
    scores = (xf @ wr.t()).softmax(-1)
    if x.is_cuda:
        # 16-bit scores can order a near-tie differently from fp32; take the layer's own
        # choice of experts and check everything else (weights, experts, gradients) in fp32.
        with torch.no_grad():
            e = layer.router(x)[2]
        w = scores.gather(1, e)
    else:
        w, e = torch.topk(scores, k, dim=-1)
    if args.moe_normalize_expert_weights:
        w = w / torch.norm(w, p=args.moe_normalize_expert_weights, dim=-1, keepdim=True)
    w1 = layer.experts.mlp.w1.float().view(E, -1, h)
    w2 = layer.experts.mlp.w2.float().view(E, -1, h)
    v1 = layer.experts.mlp.v1.float().view(E, -1, h) if mlp_type == 'glu' else None
    out = torch.zeros_like(xf)
    for ex in range(E):
        for s in range(k):
            sel = e[:, s] == ex
            if not sel.any():
                continue
            hid = args.activation_fn(xf[sel] @ w1[ex].t())
            if v1 is not None:
                hid = hid * (xf[sel] @ v1[ex].t())
            out[sel] += w[sel, s:s + 1] * (hid @ w2[ex])
    return out.view(x.shape), scores, e


@pytest.mark.parametrize('device', DEVICES)
@pytest.mark.parametrize('bs,sl,hs,ne,top_k', CONFIGS)
@pytest.mark.parametrize('mlp_impl', ['grouped', 'sparse'])
@pytest.mark.parametrize('mlp_type', ['mlp', 'glu'])
@pytest.mark.parametrize('mem_opt', [False, True])
def test_dmoe_matches_dense_loop(device, bs, sl, hs, ne, top_k, mlp_impl, mlp_type, mem_opt):
    args = _args(device, hs=hs, ne=ne, top_k=top_k, mlp_impl=mlp_impl, mlp_type=mlp_type,
                 memory_optimized_mlp=mem_opt)
    layer = mb.dMoE(args)
    x = torch.randn(sl, bs, hs, device=device).to(layer.router.layer.weight.dtype).requires_grad_(True)
    out, bias = layer(x)
    assert out.shape == x.shape and bias.shape == (hs,)
    ref, _, _ = dense_oracle(layer, x, mlp_type)
    torch.testing.assert_close(out.float(), ref, **_tol(device))

    params = [layer.experts.mlp.w1, layer.experts.mlp.w2, layer.router.layer.weight, x]
    if mlp_type == 'glu':
        params.append(layer.experts.mlp.v1)
    probe = torch.randn_like(ref)
    got = torch.autograd.grad((out.float() * probe).sum(), params)
    want = torch.autograd.grad((ref * probe).sum(), params)
    for g, w_ in zip(got, want):
        tol = _tol(device)
        if device == 'cuda':   # 16-bit gradients carry rounding proportional to their magnitude
            tol = dict(rtol=5e-2, atol=3e-2 * float(w_.abs().max()) + 1e-3)
        torch.testing.assert_close(g.float(), w_.float(), **tol)


def test_config1_cpu_plumbing():
    """One dMoE layer, hidden 128, ffn 512, 8 experts, top-2, GELU, x[32,2,128] from seed 0: 1e-5."""
    torch.manual_seed(0)
    args = mb.Arguments(hidden_size=128, ffn_hidden_size=512, moe_num_experts=8, moe_top_k=2, fp16=False,
                        device=torch.device('cpu'))
    layer = mb.dMoE(args)
    x = torch.randn(32, 2, 128, requires_grad=True)
    out, _ = layer(x)
    ref, _, _ = dense_oracle(layer, x)
    torch.testing.assert_close(out, ref, rtol=1e-5, atol=1e-5)
    g = torch.autograd.grad(out.square().sum(), [x, layer.experts.mlp.w1, layer.experts.mlp.w2])
    r = torch.autograd.grad(ref.square().sum(), [x, layer.experts.mlp.w1, layer.experts.mlp.w2])
    for a, b in zip(g, r):
        torch.testing.assert_close(a, b, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize('device', DEVICES)
@pytest.mark.parametrize('bs,sl,hs,ne,top_k', CONFIGS[:5])
def test_moe_capacity0_equals_dmoe(device, bs, sl, hs, ne, top_k):
    args = _args(device, hs=hs, ne=ne, top_k=top_k, moe_capacity_factor=0)
    moe = mb.MoE(args)
    dmoe = mb.dMoE(_args(device, hs=hs, ne=ne, top_k=top_k, mlp_impl='grouped'))
    with torch.no_grad():
        dmoe.router.layer.weight.copy_(moe.router.layer.weight)
        E = ne
        dmoe.experts.mlp.w1.copy_(moe.experts.mlp.w1.transpose(1, 2).reshape(-1, hs))
        dmoe.experts.mlp.w2.copy_(moe.experts.mlp.w2.reshape(-1, hs))
    x = torch.randn(sl, bs, hs, device=device).to(moe.router.layer.weight.dtype)
    a, _ = moe(x)
    b, _ = dmoe(x)
    torch.testing.assert_close(a.float(), b.float(), **_tol(device))


@pytest.mark.parametrize('device', DEVICES)
def test_moe_drops_tokens_beyond_capacity(device):
    args = _args(device, hs=128, ne=4, top_k=1, moe_capacity_factor=1, bias=False)
    layer = mb.MoE(args)
    with torch.no_grad():  # route everything to expert 0
        layer.router.layer.weight.zero_()
        layer.router.layer.weight[0].fill_(1.0)
    x = torch.rand(64, 1, 128, device=device).to(layer.router.layer.weight.dtype) + 0.5
    out = layer(x)
    kept = (out.float().abs().sum(-1) > 0).sum().item()
    assert kept == 16  # capacity = 1 * 64 / 4


@pytest.mark.parametrize('device', DEVICES)
def test_forward_return_modes_and_shared_expert(device):
    x = torch.randn(16, 2, 128, device=device)
    for bias, return_bias in [(True, True), (True, False), (False, True)]:
        layer = mb.dMoE(_args(device, bias=bias, return_bias=return_bias))
        out = layer(x.to(layer.router.layer.weight.dtype))
        if bias and return_bias:
            assert isinstance(out, tuple) and out[1] is layer.experts.bias
        else:
            assert out.shape == x.shape
    for typ in ('mlp', 'glu'):
        for weighted in (False, True):
            layer = mb.dMoE(_args(device, bias=False, shared_expert=True, mlp_type=typ,
                                  shared_expert_weighted_sum=weighted, shared_expert_hidden_size=64))
            layer.shared_expert.to(layer.router.layer.weight.dtype)
            xx = x.to(layer.router.layer.weight.dtype)
            out = layer(xx)
            experts_only = layer.experts(xx, *layer.router(xx))
            sh = layer.shared_expert(xx)
            k = layer.experts.args.moe_top_k
            ref = sh / (k + 1) + experts_only * (k / (k + 1)) if weighted else sh + experts_only
            torch.testing.assert_close(out.float(), ref.float(), **_tol(device))
            keys = set(layer.state_dict())
            assert {'shared_expert.up_proj.weight', 'shared_expert.down_proj.weight'} <= keys
            assert ('shared_expert.gate_proj.weight' in keys) == (typ == 'glu')


def test_state_dict_keys_and_shapes():
    E, h, f = 4, 128, 256
    for impl in ('sparse', 'grouped'):
        sd = mb.dMoE(_args('cpu', hs=h, ffn=f, ne=E, mlp_impl=impl, mlp_type='glu')).state_dict()
        assert {k: tuple(v.shape) for k, v in sd.items()} == {
            'router.layer.weight': (E, h), 'experts.bias': (h,), 'experts.mlp.w1': (E * f, h),
            'experts.mlp.w2': (E * f, h), 'experts.mlp.v1': (E * f, h)}
    sd = mb.MoE(_args('cpu', hs=h, ffn=f, ne=E)).state_dict()
    assert {k: tuple(v.shape) for k, v in sd.items()} == {
        'router.layer.weight': (E, h), 'experts.bias': (h,), 'experts.mlp.w1': (E, h, f),
        'experts.mlp.w2': (E, f, h)}
    # Round trip through load_state_dict with reference-shaped tensors.
    src = mb.dMoE(_args('cpu', hs=h, ffn=f, ne=E))
    dst = mb.dMoE(_args('cpu', hs=h, ffn=f, ne=E))
    dst.load_state_dict({k: v.clone() for k, v in src.state_dict().items()})
    x = torch.randn(8, 1, h)
    torch.testing.assert_close(src(x)[0], dst(x)[0])


def test_same_seed_same_weights_any_impl():
    torch.manual_seed(7)
    a = mb.dMoE(_args('cpu', mlp_impl='sparse'))
    torch.manual_seed(7)
    b = mb.dMoE(_args('cpu', mlp_impl='grouped'))
    for (ka, va), (kb, vb) in zip(a.state_dict().items(), b.state_dict().items()):
        assert ka == kb and torch.equal(va, vb)


@pytest.mark.parametrize('device', DEVICES)
def test_losses(device):
    L = 3
    args = _args(device, ne=8, top_k=2, num_layers=L, moe_loss_weight=0.1, moe_zloss_weight=1e-3,
                 moe_lbl_in_fp32=True, moe_zloss_in_fp32=True)
    layers = [mb.dMoE(args) for _ in range(L)]
    x = torch.randn(16, 2, 128, device=device).to(layers[0].router.layer.weight.dtype)
    for layer in layers:
        layer.train()
        layer(x)
    lbl = moe_mod.batched_load_balancing_loss(args)
    zl = router_mod.batched_router_zloss(args)
    assert zl.shape == (L,)
    expected = 0.0
    for layer in layers:
        _, scores, e = dense_oracle(layer, x)
        tpe = torch.bincount(e.flatten(), minlength=8).float()
        expected = expected + (tpe * scores.mean(0)).sum()
    expected = expected * 8 * 0.1 / (L * 32 * 2)
    torch.testing.assert_close(lbl.float().cpu(), expected.cpu(), rtol=2e-2, atol=1e-3)
    logits = x.view(-1, 128).float() @ layers[0].router.layer.weight.float().t()
    torch.testing.assert_close(zl[0].float(), 1e-3 * torch.logsumexp(logits, 1).square().mean(), rtol=2e-2,
                               atol=1e-4)
    (lbl + zl.sum()).backward()
    assert layers[0].router.layer.weight.grad is not None
    with pytest.raises(ValueError):
        moe_mod.save_load_balancing_loss(moe_mod.get_load_balancing_loss()[0])
        moe_mod.batched_load_balancing_loss(args)
    moe_mod.clear_load_balancing_loss()
    router_mod.clear_router_zloss()
    assert moe_mod.get_load_balancing_loss() == []
    layers[0].eval()
    layers[0](x)
    assert moe_mod.get_load_balancing_loss() == []


@pytest.mark.parametrize('device', DEVICES)
def test_router_options(device):
    args = _args(device, ne=8, top_k=2, moe_normalize_expert_weights=1, moe_jitter_eps=0.1)
    layer = mb.dMoE(args)
    x = torch.randn(16, 2, 128, device=device).to(layer.router.layer.weight.dtype)
    layer.eval()
    scores, w, e = layer.router(x)
    torch.testing.assert_close(w.float().sum(-1), torch.ones(32, device=device), rtol=1e-2, atol=1e-2)
    assert scores.shape == (32, 8) and e.shape == (32, 2)
    layer.train()
    layer.router(x)  # jitter path
    uni = mb.dMoE(_args(device, ne=8, top_k=1, uniform_expert_assignment=True))
    _, _, e = uni.router(x.to(uni.router.layer.weight.dtype))
    assert torch.equal(e.flatten().cpu(), torch.arange(32) % 8)
    # top-1 ties resolve to the lowest expert id
    tie = mb.dMoE(_args(device, ne=4, top_k=1))
    with torch.no_grad():
        tie.router.layer.weight.zero_()
    _, _, e = tie.router(x.to(tie.router.layer.weight.dtype))
    assert int(e.max()) == 0


def test_arguments_defaults_and_from_megatron():
    a = mb.Arguments()
    assert (a.hidden_size, a.ffn_hidden_size, a.mlp_impl, a.mlp_type, a.fp16, a.bf16) == (1024, 4096, 'grouped',
                                                                                         'mlp', True, False)
    assert a.shared_expert_hidden_size == 4096 and a.moe_loss_weight == 0.1 and a.return_bias
    with pytest.raises(ValueError):
        mb.Arguments(mlp_impl='dense')

    class NS:
        hidden_size = 64
        moe_num_experts = 4
        unrelated = 1

    b = from_megatron(NS())
    assert b.hidden_size == 64 and b.moe_num_experts == 4


@pytest.mark.parametrize('device', DEVICES)
@pytest.mark.parametrize('on_instance', [True, False])
def test_replaced_scaling_of_the_token_dropping_weights_is_used(device, on_instance):
    layer = mb.MoE(_args(device, activation_fn=F.silu, bias=False, return_bias=False))
    x = torch.randn(64, 1, 128).to(device, next(layer.parameters()).dtype)
    with torch.no_grad():
        for w in layer.experts.mlp.parameters():
            w.mul_(2)
        want = layer(x)
        for w in layer.experts.mlp.parameters():
            w.mul_(0.5)
        if on_instance:
            layer.experts.mlp.scale_grad = lambda w: w * 2
        else:
            layer.experts.mlp.__class__ = type('Scaled', (mlp_mod.MLP,), {'scale_grad': lambda self, w: w * 2})
        torch.testing.assert_close(layer(x), want, **_tol(device))


@pytest.mark.parametrize('device', DEVICES)
@pytest.mark.parametrize('dropless', [True, False])
def test_activation_modules_with_a_forward_or_hooks_of_their_own(device, dropless):
    """A subclass of a known activation module computes what it says, and hooks on one are called."""

    class Twice(torch.nn.GELU):

        def forward(self, z):
            return 2 * super().forward(z)

    def run(act):
        torch.manual_seed(0)
        layer = (mb.dMoE if dropless else mb.MoE)(_args(device, activation_fn=act, mlp_impl='grouped', bias=False,
                                                        return_bias=False))
        return layer(torch.randn(8, 2, 128).to(device, next(layer.parameters()).dtype)).float()

    torch.testing.assert_close(run(Twice()), run(lambda z: 2 * F.gelu(z)), **_tol(device))
    act, calls = torch.nn.SiLU(), []
    act.register_forward_hook(lambda *a: calls.append(1))
    run(act)
    assert calls
    assert [ops_gg.activation_id(m) for m in (torch.nn.GELU(), torch.nn.GELU('tanh'), torch.nn.SiLU(), torch.nn.ReLU())] == [
        ops_gg.ACT_GELU_ERF, ops_gg.ACT_GELU_TANH, ops_gg.ACT_SILU, ops_gg.ACT_RELU]


@pytest.mark.parametrize('device', DEVICES)
def test_custom_activation_callable(device):
    act = lambda t: F.relu(t) ** 2  # noqa: E731 - not known to the kernel: unfused route
    layer = mb.dMoE(_args(device, activation_fn=act, ne=4, top_k=2))
    x = torch.randn(8, 2, 128, device=device).to(layer.router.layer.weight.dtype).requires_grad_(True)
    out, _ = layer(x)
    ref, _, _ = dense_oracle(layer, x)
    torch.testing.assert_close(out.float(), ref, **_tol(device))
    out.float().sum().backward()
    assert layer.experts.mlp.w1.grad is not None


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize('top_k,hidden,dropped', [(1, 136, False), (3, 136, True), (1, 100, True), (2, 100, False)])
def test_scatter_adds_the_output_bias(dtype, top_k, hidden, dropped):
    """The bias of the un-permutation, its gradient and copies without a row, against the sum in fp32."""
    torch.manual_seed(0)
    tokens, experts = 77, 5
    top = torch.randint(0, experts, (tokens * top_k,), device='cuda')
    indices, bin_ids, bins, _, _ = ops.route_plan(top, experts)
    bias = torch.randn(hidden, device='cuda').to(dtype).requires_grad_(True)
    weights = torch.rand(tokens * top_k, device='cuda').to(dtype)
    if dropped:
        x = torch.randn(experts, 9, hidden, device='cuda').to(dtype)
        call = lambda b: ops.binned_scatter(x, indices, weights, bins, top_k, b)
    else:
        x = torch.randn(tokens * top_k, hidden, device='cuda').to(dtype)
        call = lambda b: ops.scatter(x, indices, bin_ids, weights, bins, top_k, b)
    out = call(bias)
    want = call(None).float() + bias.detach().float()
    # One rounding instead of two: at most one unit of the type's last place of either term.
    eps = torch.finfo(dtype).eps
    assert torch.all((out.float() - want).abs() <= eps * (want.abs() + call(None).float().abs()) + 1e-6)
    dy = torch.randn_like(out)
    db, = torch.autograd.grad(out, bias, dy)
    exact = dy.double().sum(0)
    assert torch.all((db.double() - exact).abs() <= eps * exact.abs() + 1e-5 * dy.double().abs().sum(0))


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
@pytest.mark.parametrize('layout', ['ragged', 'padded', 'capacity'])
@pytest.mark.parametrize('top_k,hidden', [(1, 136), (2, 1032), (3, 100)])
def test_unpermutation_backward_in_one_pass(dtype, layout, top_k, hidden):
    """Both gradients of the weighted un-permutation against the CPU statements, with pad rows, dropped
    copies, an empty expert and row lengths around the vector width."""
    torch.manual_seed(1)
    tokens, experts, capacity = 61, 6, 12
    top = torch.randint(0, experts - 1, (tokens * top_k,))
    indices, bin_ids, bins, padded, _ = ops.route_plan(top, experts)
    rows = {'ragged': tokens * top_k, 'padded': int(padded[-1]) + 7, 'capacity': experts * capacity}[layout]
    x = torch.randn(rows, hidden).to(dtype)
    weights = torch.rand(tokens * top_k).to(dtype)
    dy = torch.randn(tokens, hidden).to(dtype)

    def grads(dev):
        args = [t.to(dev) for t in (indices, bin_ids, bins, padded)]
        xx, ww = x.to(dev).requires_grad_(True), weights.to(dev).requires_grad_(True)
        if layout == 'capacity':
            y = ops.binned_scatter(xx.view(experts, capacity, hidden), args[0], ww, args[2], top_k)
        elif layout == 'padded':
            y = ops.padded_scatter(xx, args[0], args[1], ww, args[2], args[3], top_k)
        else:
            y = ops.scatter(xx, args[0], args[1], ww, args[2], top_k)
        return torch.autograd.grad(y, [xx, ww], dy.to(dev))

    eps = torch.finfo(dtype).eps
    for got, want in zip(grads('cuda'), grads('cpu')):
        # Sums of `hidden` fp32 products in another order, then one rounding.
        torch.testing.assert_close(got.cpu().float(), want.float(), rtol=2 * eps, atol=1e-5 * hidden ** 0.5 + eps)


@pytest.mark.gpu
@pytest.mark.parametrize('act', [partial(F.gelu, approximate='tanh'), F.silu, F.gelu])
@pytest.mark.parametrize('tokens,hidden,ffn', [(40, 64, 72), (333, 136, 256)])
def test_token_dropping_experts_in_gemm_epilogues(act, tokens, hidden, ffn):
    """Experts of the token-dropping layer with the activation in the GEMM epilogues, against the same
    layer with a callable the kernel does not know (elementwise passes)."""
    torch.manual_seed(0)
    grads = []
    for fn in (act, lambda z: act(z)):
        torch.manual_seed(0)
        layer = mb.MoE(mb.Arguments(hidden_size=hidden, ffn_hidden_size=ffn, moe_num_experts=4, moe_top_k=2,
                                    moe_capacity_factor=1, activation_fn=fn, bias=False, return_bias=False, fp16=False,
                                    bf16=True, device=torch.device('cuda')))
        x = torch.randn(tokens, 1, hidden, device='cuda').bfloat16().requires_grad_(True)
        y = layer(x)
        moe_mod.clear_load_balancing_loss()
        grads.append([y] + list(torch.autograd.grad(y, [x] + list(layer.parameters()), torch.ones_like(y))))
    for got, want in zip(*grads):
        # bf16 intermediates are rounded alike on both sides; sums differ in order and in the last place.
        torch.testing.assert_close(got, want, rtol=3e-2, atol=2e-2 * float(want.detach().float().abs().max()) + 1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
@pytest.mark.parametrize('act,exact', [
    # In 64 bits, and in the forms that do not cancel where the function is close to zero.
    (partial(F.gelu, approximate='tanh'), lambda z: z * torch.sigmoid(2 * (2 / math.pi) ** 0.5 * (z + 0.044715 * z ** 3))),
    (F.silu, F.silu), (F.gelu, lambda z: 0.5 * z * torch.erfc(-z / 2 ** 0.5))], ids=['gelu_tanh', 'silu', 'gelu'])
def test_token_dropping_activation_is_as_exact_as_the_library(dtype, act, exact):
    """Activation and derivative at every 16-bit value up to 1e4, through experts whose weights are the
    identity, in units of the last place from the 64-bit function: the largest and the mean square error are
    at most the library's fp32 function's, or what one rounding leaves (a half)."""
    args = mb.Arguments(hidden_size=64, ffn_hidden_size=64, moe_num_experts=1, activation_fn=act, bias=False,
                        fp16=dtype == torch.float16, bf16=dtype == torch.bfloat16, device=torch.device('cuda'))
    experts = mlp_mod.MLP(args)
    with torch.no_grad():
        experts.w1.copy_(torch.eye(64))
        experts.w2.copy_(torch.eye(64))
    z = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(dtype)
    z = torch.where(z.abs() <= 1e4, z, torch.zeros_like(z)).cuda()

    def both(fn, t):
        t = t.clone().requires_grad_(True)
        y = fn(t)
        return [y.detach().double().view(-1), torch.autograd.grad(y, t, torch.ones_like(y))[0].double().view(-1)]

    exact = both(exact, z.double())
    floor = max(torch.finfo(dtype).smallest_normal, 1e-30)
    for got, lib, want in zip(both(experts, z.view(1, 1024, 64)), both(act, z), exact):
        unit = torch.finfo(dtype).eps * torch.exp2(torch.floor(torch.log2(want.abs().clamp_min(floor))))
        e, ref = (got - want).abs() / unit, (lib - want).abs() / unit
        # fp32's last place is 2^-13 of fp16's: eight of them may tip a rounding that the library does not.
        assert float(e.max()) <= max(float(ref.max()), 0.5) + 8 * 2 ** -13
        assert float(e.square().mean()) <= 1.0001 * float(ref.square().mean())


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
def test_token_dropping_relu_shows_nan_and_closes_like_the_library(dtype):
    """ReLU in the epilogues against the library's: NaN stays NaN, closed units pass no gradient (an infinite
    one included), and every other 16-bit value goes through."""
    args = mb.Arguments(hidden_size=64, ffn_hidden_size=64, moe_num_experts=2, activation_fn=F.relu, bias=False,
                        fp16=dtype == torch.float16, bf16=dtype == torch.bfloat16, device=torch.device('cuda'))
    experts = mlp_mod.MLP(args)
    with torch.no_grad():
        for w in experts.parameters():
            w.copy_(torch.eye(64))
    z = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(dtype).cuda()
    z = torch.where(z.abs() < float('inf'), z, torch.zeros_like(z)).view(2, 512, 64).requires_grad_(True)
    y = experts(z)
    dz, = torch.autograd.grad(y, z, torch.ones_like(y))
    lib = F.relu(z.detach())
    # The multiplication by one flushes fp32 subnormals (bf16's own) to zero.
    normal = (lib >= 2.0 ** -120) | (lib == 0)
    assert torch.equal(y[normal], lib[normal]) and float(y.detach()[~normal].abs().max() if (~normal).any() else 0) < 2.0 ** -119
    assert torch.equal(dz[normal], (z > 0).to(dtype)[normal])
    x = torch.randn(2, 8, 64, device='cuda').to(dtype)
    x[1, 3, 5] = float('nan')
    out = experts(x)
    assert out[1, 3].isnan().all() and int(out.isnan().sum()) == 64


@pytest.mark.gpu
@pytest.mark.parametrize('kind', ['mlp', 'glu', 'dropping'])
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16])
@pytest.mark.parametrize('tokens,top_k,bias,memory_optimized', [(1, 1, True, False), (37, 2, False, True), (300, 1, True, True)])
def test_native_expert_block_equals_the_separate_ops(kind, dtype, tokens, top_k, bias, memory_optimized):
    """One native call against the same kernels launched op by op (a hook on the expert module sends the
    layer there): outputs and every gradient are equal, with and without autograd."""
    torch.manual_seed(0)
    args = mb.Arguments(hidden_size=72, ffn_hidden_size=264, moe_num_experts=5, moe_top_k=top_k, moe_capacity_factor=1,
                        mlp_type='glu' if kind == 'glu' else 'mlp', mlp_impl='grouped', activation_fn=F.silu, bias=bias,
                        return_bias=False, memory_optimized_mlp=memory_optimized, fp16=dtype == torch.float16,
                        bf16=dtype == torch.bfloat16, device=torch.device('cuda'))
    layer = (mb.MoE if kind == 'dropping' else mb.dMoE)(args)
    if bias:
        torch.nn.init.normal_(layer.experts.bias)
    x = torch.randn(tokens, 1, 72, device='cuda').to(dtype).requires_grad_(True)
    dy = torch.randn_like(x)

    def run():
        y = layer(x)
        moe_mod.clear_load_balancing_loss()
        with torch.no_grad():
            plain = layer(x)
        moe_mod.clear_load_balancing_loss()
        return [y, plain] + list(torch.autograd.grad(y, [x] + list(layer.parameters()), dy))

    assert layer.experts._block_call(x, *layer.router(x)[1:]) is not None or (
        kind == 'dropping' and layer.experts.expert_capacity(tokens) == 0)
    moe_mod.clear_load_balancing_loss()
    fast = run()
    hook = layer.experts.mlp.register_forward_hook(lambda *a: None)
    assert layer.experts._block_call(x, *layer.router(x)[1:]) is None
    slow = run()
    hook.remove()
    for got, want in zip(fast, slow):
        assert torch.equal(got, want)


def _stock_layer(kind, dtype=torch.bfloat16, hidden=72, ffn=264, experts=5, top_k=2, **kw):
    """A layer whose calls take the native expert block (kind 'sparse': only its output-bias rule)."""
    args = dict(hidden_size=hidden, ffn_hidden_size=ffn, moe_num_experts=experts, moe_top_k=top_k, moe_capacity_factor=1,
                mlp_type='glu' if kind == 'glu' else 'mlp', mlp_impl='sparse' if kind == 'sparse' else 'grouped',
                activation_fn=F.silu, bias=True, return_bias=False, fp16=dtype == torch.float16,
                bf16=dtype == torch.bfloat16, device=torch.device('cuda'))
    args.update(kw)
    layer = (mb.MoE if kind == 'dropping' else mb.dMoE)(mb.Arguments(**args))
    if layer.experts.bias is not None:
        torch.nn.init.normal_(layer.experts.bias)
    return layer


@pytest.mark.gpu
@pytest.mark.parametrize('kind', ['mlp', 'glu', 'dropping'])
@pytest.mark.parametrize('offset', [0, 1, 3])
def test_output_gradient_at_any_address(kind, offset):
    """A contiguous output gradient may start at any element of a flat buffer; the kernels that read 16 bytes
    at a time must not be handed one that does not start on 16 bytes."""
    layer = _stock_layer(kind)
    x = torch.randn(37, 1, 72, device='cuda').bfloat16().requires_grad_(True)
    flat = torch.randn(37 * 72 + 8, device='cuda').bfloat16()
    dy = flat[offset:offset + 37 * 72].view(37, 1, 72)
    assert dy.is_contiguous() and (dy.data_ptr() % 16 == 0) == (offset == 0)
    y = layer(x)
    moe_mod.clear_load_balancing_loss()
    leaves = [x] + list(layer.parameters())
    got = torch.autograd.grad(y, leaves, dy, retain_graph=True)
    want = torch.autograd.grad(y, leaves, dy.clone())
    for leaf, g, w in zip(leaves, got, want):
        if leaf is layer.experts.bias:      # fp32 sums in another order, rounded once
            torch.testing.assert_close(g, w, rtol=2 ** -7, atol=1e-5 * 37)
        else:
            torch.testing.assert_close(g, w, rtol=2 ** -7, atol=2 ** -8 * float(w.float().abs().max()))


@pytest.mark.gpu
@pytest.mark.parametrize('kind', ['mlp', 'glu', 'dropping'])
@pytest.mark.parametrize('top_k,memory_optimized,ffn', [(1, True, 512), (2, True, 256), (2, False, 1024), (1, True, 128)])
def test_native_block_holds_no_more_memory_than_the_separate_ops(kind, top_k, memory_optimized, ffn):
    """Peak of a training pass: the rows before the un-permutation are free before the experts' backward."""
    layer = _stock_layer(kind, hidden=512, ffn=ffn, experts=4, top_k=top_k, memory_optimized_mlp=memory_optimized)
    x = torch.randn(4096, 1, 512, device='cuda').bfloat16().requires_grad_(True)
    dy = torch.randn_like(x)

    def peak():
        for _ in range(2):          # the second pass finds what the first one laid out
            gc.collect()            # nothing of an earlier test is freed in between
            torch.cuda.reset_peak_memory_stats()
            base = torch.cuda.memory_stats()['requested_bytes.all.current']
            y = layer(x)
            moe_mod.clear_load_balancing_loss()
            grads = torch.autograd.grad(y, [x] + list(layer.parameters()), dy)
            top = torch.cuda.memory_stats()['requested_bytes.all.peak'] - base
            del y, grads
        return top

    fast = peak()
    layer.experts.mlp.register_forward_hook(lambda *a: None)
    slow = peak()
    assert fast <= slow + 8 * 4 * 4096 * top_k      # index arrays, of 4 bytes a copy


@pytest.mark.gpu
@pytest.mark.parametrize('kind', ['mlp', 'glu', 'dropping'])
@pytest.mark.parametrize('trained', ['experts.bias', 'router', 'w1', 'w2', 'x', 'all'])
def test_native_block_keeps_no_more_for_backward_than_the_separate_ops(kind, trained):
    """Bytes saved by a forward pass when only some of the layer is trained."""
    layer = _stock_layer(kind)
    for name, p in layer.named_parameters():
        p.requires_grad_(trained == 'all' or trained in name)
    x = torch.randn(300, 1, 72, device='cuda').bfloat16().requires_grad_(trained in ('x', 'all'))
    own = {t.untyped_storage().data_ptr() for t in [x, *layer.parameters()]}

    def kept():
        held = {}

        def pack(t):
            held.setdefault(t.untyped_storage().data_ptr(), t)
            return t

        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
            layer(x)
        moe_mod.clear_load_balancing_loss()
        return sum(t.untyped_storage().nbytes() for ptr, t in held.items() if ptr not in own)

    fast = kept()
    layer.experts.mlp.register_forward_hook(lambda *a: None)
    assert fast <= kept() + 600 * 4         # one index of 4 bytes a copy


@pytest.mark.gpu
@pytest.mark.parametrize('kind,step', [('mlp', 'indices_and_bins'), ('mlp', 'grouped_permute_and_compute'),
                                       ('mlp', 'grouped_forward_once'), ('glu', 'grouped_permute_and_compute'),
                                       ('dropping', 'permute_and_compute'), ('dropping', 'expert_capacity'),
                                       ('dropping', 'indices_and_bins'), ('sparse', 'sparse_forward_once'),
                                       ('sparse', 'topology')])
def test_step_replaced_on_the_instance_is_called(kind, step):
    """A step of the layer patched on one object is honoured, with the arguments the step always had."""
    layer = _stock_layer(kind, hidden=128, ffn=256)
    x = torch.randn(37, 1, 128, device='cuda').bfloat16()
    want = layer(x)
    plain, calls = getattr(layer.experts, step), []

    def replaced(*args):
        calls.append(step)
        return plain(*args)

    setattr(layer.experts, step, replaced)
    got = layer(x)
    assert calls
    # The bias is added by the kernel or afterwards: one rounding of the sum apart.
    torch.testing.assert_close(got, want, rtol=2 ** -7, atol=2 ** -7 * float(layer.experts.bias.detach().abs().max()))


@pytest.mark.gpu
@pytest.mark.parametrize('kind', ['mlp', 'sparse', 'dropping'])
def test_tangent_of_the_output_bias(kind):
    """Forward-mode differentiation with respect to the output bias: its tangent on every row."""
    from torch.autograd import forward_ad
    experts = _stock_layer(kind, hidden=128, ffn=256).experts.requires_grad_(False)
    x, scores, weights = (torch.rand(37, n, device='cuda').bfloat16() for n in (128, 5, 2))
    ids = torch.randint(0, 5, (37, 2), device='cuda')
    tangent = torch.randn(128, device='cuda').bfloat16()
    with forward_ad.dual_level():
        bias = forward_ad.make_dual(experts.bias.detach(), tangent)
        out = torch.func.functional_call(experts, {'bias': bias}, (x, scores, weights, ids))
        assert torch.equal(forward_ad.unpack_dual(out).tangent, tangent.expand(37, 128))


@pytest.mark.gpu
@pytest.mark.parametrize('kind', ['mlp', 'dropping'])
def test_expert_ids_of_any_stride(kind):
    experts = _stock_layer(kind, top_k=1).experts
    x, scores, weights = (torch.rand(37, n, device='cuda').bfloat16() for n in (72, 5, 1))
    ids = torch.randint(0, 5, (37, 2), device='cuda')[:, 0]
    assert not ids.is_contiguous()
    with torch.no_grad():
        assert torch.equal(experts(x, scores, weights, ids), experts(x, scores, weights, ids.contiguous()))


@pytest.mark.gpu
@pytest.mark.parametrize('kind', ['mlp', 'sparse', 'dropping'])
@pytest.mark.parametrize('shape', [(1,), (37, 128), ()])
def test_output_bias_of_another_shape_is_broadcast(kind, shape):
    """A bias that is not one value per column never reaches the kernels, which read one per column."""
    layer = _stock_layer(kind, hidden=128, ffn=256)
    x = torch.randn(37, 128, device='cuda').bfloat16()
    with torch.no_grad():
        layer.experts.bias.zero_()
        plain = layer(x)
        layer.experts.bias = torch.nn.Parameter(torch.randn(shape, device='cuda').bfloat16())
        assert torch.equal(layer(x), plain + layer.experts.bias)
    from megablocks_b200._ext import ext
    rows = torch.arange(37, dtype=torch.int32, device='cuda')
    with pytest.raises(RuntimeError, match='bias'):
        ext().combine_rows(x, rows, None, 1, 37, x.new_zeros(64))


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
def test_column_sum_of_rows_at_any_address(dtype):
    from megablocks_b200._ext import ext
    flat = torch.randn(100 * 72 + 8, device='cuda').to(dtype)
    for offset in (0, 1, 2, 7):
        x = flat[offset:offset + 100 * 72].view(100, 72)
        want = x.double().sum(0)
        assert torch.all((ext().column_sum(x).double() - want).abs() <= torch.finfo(dtype).eps * want.abs() + 1e-5 * x.double().abs().sum(0))


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize('experts', [4, 8, 24, 32, 64, 128, 256, 320])
@pytest.mark.parametrize('top_k,norm_p', [(1, 0), (2, 1), (4, 2), (8, 0)])
def test_router_selection_over_expert_counts(dtype, experts, top_k, norm_p):
    """Vector and warp-per-token router kernels, forward and backward, around their size limits, with equal
    logits (ties go to the lowest id) and an infinite one."""
    if top_k > experts:
        return
    torch.manual_seed(experts)
    logits = torch.randn(37, experts).to(dtype)
    logits[3] = 0.5
    logits[5, 1] = -float('inf')
    got = router_mod._FusedTopK.apply(logits.cuda().requires_grad_(True), top_k, float(norm_p))
    scores = logits.float().softmax(-1).to(dtype)
    # An fp32 exponential and sum: within one unit of the last place after rounding.
    torch.testing.assert_close(got[0].detach().cpu().float(), scores.float(), rtol=2 * torch.finfo(dtype).eps + 1e-5, atol=1e-7)
    own = got[0].detach().cpu()
    order = torch.sort(own.float(), dim=-1, descending=True, stable=True)[1][:, :top_k]
    assert torch.equal(got[2].cpu(), order)
    x = own.double().requires_grad_(True)       # d logits = s (g - <g, s>) for the scores that were selected from
    w = x.gather(1, order)
    if norm_p:
        w = w / w.norm(p=norm_p, dim=-1, keepdim=True)
    torch.testing.assert_close(got[1].detach().cpu().double(), w.detach(), rtol=3 * torch.finfo(dtype).eps, atol=1e-7)
    ds, dw = torch.randn_like(own), torch.randn(37, top_k).to(dtype)
    g, = torch.autograd.grad([x, w], x, [ds.double(), dw.double()])
    want = own.double() * (g - (g * own.double()).sum(-1, keepdim=True))
    leaf = logits.cuda().requires_grad_(True)
    out = router_mod._FusedTopK.apply(leaf, top_k, float(norm_p))
    dl, = torch.autograd.grad([out[0], out[1]], leaf, [ds.cuda(), dw.cuda()])
    torch.testing.assert_close(dl.cpu().double(), want, rtol=4 * torch.finfo(dtype).eps + 1e-5,
                               atol=1e-5 + torch.finfo(dtype).eps * float(want.abs().max()))


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize('experts', [4, 24, 64, 256, 320])
@pytest.mark.parametrize('top_k,norm_p', [(1, 0), (2, 1), (4, 2)])
def test_router_selection_of_non_finite_logits(dtype, experts, top_k, norm_p):
    """Tokens with NaN or infinite logits (an fp16 overflow) get distinct ids of real experts and NaN scores,
    weights and gradients, like the library's softmax and top-k; their neighbours are untouched."""
    torch.manual_seed(experts)
    clean = torch.randn(37, experts).to(dtype)
    logits, bad = clean.clone(), [3, 4, 9, 20, 36]
    logits[3, 1] = float('nan')
    logits[4, 2] = float('inf')
    logits[9] = float('nan')
    logits[20] = float('inf')
    logits[36] = -float('inf')
    run = lambda t: router_mod._FusedTopK.apply(t, top_k, float(norm_p))
    leaf = logits.cuda().requires_grad_(True)
    scores, weights, ids = run(leaf)
    with torch.no_grad():
        plain = router_mod._fused_top_k(leaf, top_k, float(norm_p))
    assert torch.equal(plain[2], ids)
    assert int(ids.min()) >= 0 and int(ids.max()) < experts
    assert all(len(set(row)) == top_k for row in ids.tolist())
    assert scores[bad].isnan().all() and weights[bad].isnan().all()
    assert torch.equal(logits.float().softmax(-1).isnan(), scores.detach().cpu().isnan())
    own = clean.cuda().requires_grad_(True)
    want = run(own)
    rest = [t for t in range(37) if t not in bad]
    for got, ref in zip((scores, weights, ids), want):
        assert torch.equal(got[rest], ref[rest])
    ds, dw = torch.randn(37, experts, device='cuda').to(dtype), torch.randn(37, top_k, device='cuda').to(dtype)
    got, = torch.autograd.grad([scores, weights], leaf, [ds, dw])
    ref, = torch.autograd.grad(want[:2], own, [ds, dw])
    assert got[bad].isnan().all() and torch.equal(got[rest], ref[rest])


@pytest.mark.gpu
@pytest.mark.parametrize('experts,copies', [(5, 1), (64, 4096), (64, 5000), (1000, 300), (1200, 50)])
@pytest.mark.parametrize('capacity', [0, 3])
def test_plan_gives_the_rows_of_the_copies(experts, copies, capacity):
    """Rows of the copies from the plan (both its paths, and the search that serves the rest) against the
    sorted order; dropped copies are -1."""
    from megablocks_b200._ext import ext
    torch.manual_seed(copies)
    top = torch.randint(0, experts, (copies,), device='cuda')
    indices, bin_ids, bins, _, _, rows = ext().route_plan_rows(top, experts, 128, capacity)
    want = torch.empty_like(indices)
    place = torch.arange(copies, device='cuda', dtype=torch.int32)
    if capacity:
        first = torch.cat([bins.new_zeros(1), bins[:-1]])[bin_ids.long()]
        place = torch.where(place - first < capacity, bin_ids * capacity + place - first, -1)
    want[indices.long()] = place.to(torch.int32)
    assert torch.equal(rows, want)


@pytest.mark.gpu
@pytest.mark.parametrize('copies', [100, 5000])
@pytest.mark.parametrize('capacity', [0, 4])
def test_plan_drops_copies_of_no_expert(copies, capacity):
    """An id past the last expert (but inside the sort's key bits) has no row on either path."""
    from megablocks_b200._ext import ext
    top = torch.arange(copies, device='cuda') % 8
    rows = ext().route_plan_rows(top, 5, 128, capacity)[5]
    assert torch.all((rows == -1) | (top < 5))
    assert int(rows.max()) < (5 * capacity if capacity else copies)
    if not capacity:
        assert torch.equal(rows == -1, top >= 5)


@pytest.mark.gpu
@pytest.mark.parametrize('dtype', [torch.bfloat16, torch.float32])
@pytest.mark.parametrize('top_k', [1, 2, 3, 5])
@pytest.mark.parametrize('tokens,hidden', [(19, 8), (19, 100), (19, 512), (19, 520), (19, 1032), (5000, 8), (9600, 264),
                                           (9600, 8)])
def test_combine_slices_and_copy_pairs(dtype, top_k, tokens, hidden):
    """Un-permutation over row lengths around a warp's slice, odd numbers of copies, some dropped, and token
    counts on both sides of those that fill the SMs."""
    torch.manual_seed(hidden)
    experts, capacity = 4, tokens // 2
    top = torch.randint(0, experts, (tokens * top_k,))
    indices, _, bins, _, _ = ops.route_plan(top, experts)
    x = torch.randn(experts, capacity, hidden).to(dtype)
    w = torch.rand(tokens * top_k).to(dtype)
    got = ops.binned_scatter(x.cuda(), indices.cuda(), w.cuda(), bins.cuda(), top_k)
    want = ops.binned_scatter(x, indices, w, bins, top_k)
    # The same products, then one rounding; fp32 sums of top_k terms below 6 in any order.
    torch.testing.assert_close(got.cpu().float(), want.float(), rtol=torch.finfo(dtype).eps,
                               atol=1e-6 + 6 * top_k ** 2 * 2 ** -24)
