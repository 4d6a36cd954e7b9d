"""The work this library does for its users, as measurable cases.

A case is a dict of plain values.  ``listed()`` names the twelve that stand for the library's main
paths; ``draw(rng)`` makes further ones over the same ranges.  Four kinds:

* ``layer``  one dMoE (dropless) or MoE (token-dropping) layer: inference, or a training pass that
  returns the output, the load-balancing loss and every gradient;
* ``gmm``    the grouped GEMM behind ``grouped_gemm.ops.gmm``, forward and backward;
* ``sparse`` a two-layer block-sparse network ``dsd(gelu(sdd(x, w1^T)), w2)``, forward and backward;
* ``step``   one optimizer step of a dMoE language model through ``Trainer.step``.

Sizes are those of the presets (``models/transformer.py``), the experiment scripts (``exp/``) and
the benchmarks (``benchmarks/``): hidden 512 / 768 / 1024 with ffn = 4 x hidden and 64 experts, and
the Mixtral-8x7B shape (4096 / 14336, 8 experts, top-2, GLU).
"""

import math

import torch
import torch.nn.functional as F

from megablocks_b200 import Arguments, MoE, dMoE, ops
from megablocks_b200.layers.moe import batched_load_balancing_loss, clear_load_balancing_loss
from megablocks_b200.models.transformer import MoETransformer, preset
from megablocks_b200.ops import sparse
from megablocks_b200.train import Trainer, TrainerConfig

_DTYPES = {'bf16': torch.bfloat16, 'fp16': torch.float16}
_BLOCK = 128


def _layer(name, tokens, hidden, ffn, experts, top_k, *, train, mlp='mlp', impl='grouped', dtype='bf16',
           memory_optimized=False, dropless=True):
    return dict(name=name, kind='layer', tokens=tokens, hidden=hidden, ffn=ffn, experts=experts, top_k=top_k,
                train=train, mlp=mlp, impl=impl, dtype=dtype, memory_optimized=memory_optimized, dropless=dropless)


def listed():
    return [
        # A decode step of the 125M dMoE with a batch of eight sequences: the smallest call, all latency.
        _layer('decode_125m', 8, 768, 3072, 64, 1, train=False),
        # A decode step of a Mixtral-8x7B layer, sixteen sequences: every expert's weights are read once.
        _layer('decode_mixtral', 16, 4096, 14336, 8, 2, train=False, mlp='glu'),
        # Prefill of a prompt of odd length through the same layer.
        _layer('prefill_mixtral', 2047, 4096, 14336, 8, 2, train=False, mlp='glu'),
        # Training pass of a layer of the `tiny` preset (batch 4 x 64): debugging and unit-test sizes.
        _layer('train_tiny', 256, 128, 256, 8, 2, train=True),
        # Training pass of the 46M dMoE's layer at its script's micro-batch (64 x 1024): fp16,
        # block-sparse formulation, activation recompute.
        _layer('train_46m_sparse_fp16', 65536, 512, 2048, 64, 1, train=True, impl='sparse', dtype='fp16',
               memory_optimized=True),
        # The headline layer: 125M dMoE, micro-batch 32 x 1024.
        _layer('train_125m', 32768, 768, 3072, 64, 1, train=True),
        # A ragged batch of a GLU layer, top-2, odd token count (packed sequences, last batch).
        _layer('train_glu_ragged', 5003, 1024, 4096, 32, 2, train=True, mlp='glu', memory_optimized=True),
        # One sequence of 4096 tokens through a Mixtral-8x7B layer, forward and backward: the largest.
        _layer('train_mixtral', 4096, 4096, 14336, 8, 2, train=True, mlp='glu', memory_optimized=True),
        # Token-dropping MoE of the 46M model (capacity factor 1), the `exp/moe` scripts' layer.
        _layer('train_dropping', 16384, 512, 2048, 64, 1, train=True, dropless=False),
        # The grouped GEMM alone, as users of the grouped_gemm package call it.
        dict(name='gmm_ragged', kind='gmm', rows=8191, k=1024, n=4096, groups=64, trans_b=True, dtype='bf16'),
        # A block-sparse network over a random topology, a quarter of the 128 x 128 blocks present.
        dict(name='block_sparse', kind='sparse', rows=4096, k=1024, cols=8192, density=0.25, dtype='bf16'),
        # A whole training step of the 46M dMoE (4 of its 6 layers, micro-batch 8 x 1024), replayed from
        # the recorded step as the benchmark and the training scripts run it.
        dict(name='step_46m', kind='step', model='dmoe-46m', layers=4, batch=8, seq=1024, graph=True),
    ]


# ----------------------------------------------------------------------------
# Drawing
# ----------------------------------------------------------------------------
_MAX_WEIGHT_BYTES = 2 * 3 * 8 * 4096 * 14336       # the Mixtral layer's
_MAX_FLOPS = 18 * 2 * 4096 * 4096 * 14336          # the largest listed case's


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_layer(rng):
    train = rng.random() < 0.65
    dropless = not train or rng.random() < 0.8
    if rng.random() < 0.25:
        hidden, ffn, experts, top_k, mlp = 4096, 14336, 8, 2, 'glu'
    else:
        hidden = rng.choice((128, 256, 512, 768, 1024, 1536))
        ffn = hidden * rng.choice((2, 4))
        experts = rng.choice((8, 16, 32, 64))
        top_k = rng.choice((1, 1, 2, 4))
        mlp = rng.choice(('mlp', 'glu'))
    if not dropless:
        hidden, ffn, mlp = min(hidden, 1536), min(ffn, 6144), 'mlp'
    tokens = _log(rng, 1, 64) if not train and rng.random() < 0.5 else _log(rng, 200, 65536)
    case = dict(kind='layer', tokens=tokens, hidden=hidden, ffn=ffn, experts=experts, top_k=top_k, train=train,
                mlp=mlp, impl=rng.choice(('grouped', 'grouped', 'sparse')) if dropless else 'grouped',
                dtype=rng.choice(('bf16', 'bf16', 'fp16')), memory_optimized=dropless and rng.random() < 0.5,
                dropless=dropless)
    while 2 * experts * hidden * ffn * (3 if mlp == 'glu' else 2) > _MAX_WEIGHT_BYTES:
        case['experts'] = experts = experts // 2
    flops = work(case)['flops']
    if flops > _MAX_FLOPS:
        case['tokens'] = max(1, int(tokens * _MAX_FLOPS / flops))
    # Rows are kept few enough that three states with their gradients fit beside each other.
    case['tokens'] = max(1, min(case['tokens'], 200_000_000 // (top_k * max(hidden, ffn // 2))))
    return case


def draw(rng):
    kind = rng.choice(('layer', 'layer', 'layer', 'layer', 'layer', 'gmm', 'sparse', 'step'))
    if kind == 'layer':
        return _draw_layer(rng)
    if kind == 'gmm':
        k, n = rng.choice((512, 768, 1024, 2048)), rng.choice((1024, 2048, 3072, 4096))
        return dict(kind='gmm', rows=_log(rng, 64, 65536), k=k, n=n, groups=rng.choice((4, 8, 16, 64)),
                    trans_b=rng.random() < 0.5, dtype=rng.choice(('bf16', 'bf16', 'fp16')))
    if kind == 'sparse':
        return dict(kind='sparse', rows=_BLOCK * _log(rng, 4, 64), k=_BLOCK * rng.randint(2, 12),
                    cols=_BLOCK * _log(rng, 8, 64), density=rng.choice((0.1, 0.25, 0.5)),
                    dtype=rng.choice(('bf16', 'bf16', 'fp16')))
    model = rng.choice(('tiny', 'tiny-mixtral', 'dmoe-46m'))
    if model == 'dmoe-46m':
        return dict(kind='step', model=model, layers=rng.randint(1, 4), batch=rng.randint(1, 8),
                    seq=rng.choice((256, 512, 1000, 1024)), graph=True)
    return dict(kind='step', model=model, layers=2, batch=rng.randint(1, 64), seq=rng.randint(32, 64), graph=False)


# ----------------------------------------------------------------------------
# What a program has in hand before the call
# ----------------------------------------------------------------------------
def _randn(gen, *shape, dtype, scale=1.0):
    return (torch.randn(*shape, generator=gen, device='cuda', dtype=torch.float32) * scale).to(dtype)


def _prepare_layer(case, gen):
    dtype = _DTYPES[case['dtype']]
    glu = case['mlp'] == 'glu'
    args = Arguments(
        hidden_size=case['hidden'], ffn_hidden_size=case['ffn'], moe_num_experts=case['experts'],
        moe_top_k=case['top_k'], moe_capacity_factor=1, mlp_type=case['mlp'], mlp_impl=case['impl'],
        activation_fn=F.silu if glu else Arguments.activation_fn, bias=not glu, return_bias=False,
        moe_normalize_expert_weights=1 if glu else None, memory_optimized_mlp=case['memory_optimized'],
        moe_loss_weight=0.1, moe_lbl_in_fp32=True, fp16=dtype == torch.float16, bf16=dtype == torch.bfloat16,
        device=torch.device('cuda', torch.cuda.current_device()))
    layer = (dMoE if case['dropless'] else MoE)(args).train(case['train'])
    params = list(layer.parameters())
    if not glu:     # a layer in use has a bias
        with torch.no_grad():
            layer.experts.bias.copy_(_randn(gen, case['hidden'], dtype=dtype, scale=0.02))
    # Hidden states as a norm layer leaves them: unit variance around a direction that the tokens
    # share, which skews the expert loads as in trained models.
    shared = _randn(gen, 1, 1, case['hidden'], dtype=torch.float32, scale=0.5)
    x = (torch.randn(case['tokens'], 1, case['hidden'], generator=gen, device='cuda') + shared).to(dtype)
    state = dict(kind='layer', args=args, layer=layer, params=params, x=x, train=case['train'])
    if case['train']:
        x.requires_grad_(True)
        state['dy'] = _randn(gen, *x.shape, dtype=dtype)
        state['one'] = torch.ones((), device='cuda')
    return state


def _prepare_gmm(case, gen):
    dtype = _DTYPES[case['dtype']]
    rows, k, n, groups = case['rows'], case['k'], case['n'], case['groups']
    # Uneven groups: expert popularity falls off as 1 / sqrt(rank).
    p = 1.0 / torch.arange(1, groups + 1, device='cuda', dtype=torch.float32).sqrt()
    choice = torch.multinomial(p / p.sum(), rows, replacement=True, generator=gen)
    sizes = torch.bincount(choice, minlength=groups)
    a = _randn(gen, rows, k, dtype=dtype).requires_grad_(True)
    shape = (groups, n, k) if case['trans_b'] else (groups, k, n)
    b = _randn(gen, *shape, dtype=dtype, scale=0.02).requires_grad_(True)
    return dict(kind='gmm', a=a, b=b, sizes=sizes, trans_b=case['trans_b'], dy=_randn(gen, rows, n, dtype=dtype))


def _prepare_sparse(case, gen):
    dtype = _DTYPES[case['dtype']]
    rows, k, cols = case['rows'], case['k'], case['cols']
    topo = sparse.random_mask(rows, cols, 1.0 - case['density'], _BLOCK, device='cuda', dtype=dtype)
    x = _randn(gen, rows, k, dtype=dtype).requires_grad_(True)
    w1 = _randn(gen, cols, k, dtype=dtype, scale=0.02).requires_grad_(True)
    w2 = _randn(gen, cols, k, dtype=dtype, scale=0.02).requires_grad_(True)
    return dict(kind='sparse', topo=topo, x=x, w1=w1, w2=w2, dy=_randn(gen, rows, k, dtype=dtype))


def _prepare_step(case, gen):
    cfg = preset(case['model'], num_layers=case['layers'], device=torch.device('cuda', torch.cuda.current_device()))
    model = MoETransformer(cfg)
    with torch.no_grad():       # a model under way: its biases are no longer zero
        for name, p in model.named_parameters():
            if name.endswith('bias'):
                p.copy_(_randn(gen, *p.shape, dtype=p.dtype, scale=0.02))
    trainer = Trainer(model, TrainerConfig(lr=6e-4, total_steps=20000, cuda_graph=case['graph'],
                                           graph_warmup_steps=1))
    batch = torch.randint(0, cfg.vocab_size, (case['batch'], case['seq'] + 1), generator=gen, device='cuda')
    state = dict(kind='step', trainer=trainer, params=list(model.parameters()),
                 tokens=batch[:, :-1].contiguous(), targets=batch[:, 1:].contiguous())
    if case['graph']:           # the step is recorded once, at the start of training
        for _ in range(2):
            trainer.step(state['tokens'], state['targets'])
    return state


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device='cuda').manual_seed(seed + 1)
    return {'layer': _prepare_layer, 'gmm': _prepare_gmm, 'sparse': _prepare_sparse,
            'step': _prepare_step}[case['kind']](case, gen)


# ----------------------------------------------------------------------------
# One pass
# ----------------------------------------------------------------------------
def run(state):
    kind = state['kind']
    if kind == 'layer':
        if not state['train']:
            with torch.no_grad():
                return state['layer'](state['x'])
        out = state['layer'](state['x'])
        aux = batched_load_balancing_loss(state['args'])
        clear_load_balancing_loss()
        grads = torch.autograd.grad([out, aux], [state['x']] + state['params'], [state['dy'], state['one']])
        return [out.detach(), aux.detach(), *grads]
    if kind == 'gmm':
        out = ops.gmm(state['a'], state['b'], state['sizes'], trans_b=state['trans_b'])
        return [out.detach(), *torch.autograd.grad(out, [state['a'], state['b']], state['dy'])]
    if kind == 'sparse':
        hidden = sparse.sdd(state['x'], state['w1'].t(), state['topo'])
        hidden = sparse.with_data(hidden, F.gelu(hidden.data, approximate='tanh'))
        out = sparse.dsd(hidden, state['w2'])
        return [out.detach(), *torch.autograd.grad(out, [state['x'], state['w1'], state['w2']], state['dy'])]
    loss = state['trainer'].step(state['tokens'], state['targets'])
    return [loss, *state['params']]


# ----------------------------------------------------------------------------
# What a pass cannot do without
# ----------------------------------------------------------------------------
def _work_layer(case):
    t, h, f, e, k = case['tokens'], case['hidden'], case['ffn'], case['experts'], case['top_k']
    mats = 3 if case['mlp'] == 'glu' else 2
    passes = 3 if case['train'] else 1
    flops = passes * 2.0 * t * h * (k * f * mats + e)
    touched = min(e, t * k) if not case['train'] else e
    weights = 2.0 * touched * h * f * mats * (2 if case['train'] else 1)     # read; gradients written
    rows = 2.0 * t * h * (4 if case['train'] else 2)                          # x, out (, dout, dx)
    return dict(bytes=weights + rows, flops=flops)


def _work_step(case):
    cfg = preset(case['model'], num_layers=case['layers'])
    h, f, e, v, n_layers = cfg.hidden_size, cfg.ffn_hidden_size, cfg.moe_num_experts, cfg.vocab_size, cfg.num_layers
    glu = cfg.flavour == 'mixtral'
    head = h // cfg.num_heads
    attn = h * (cfg.num_heads + 2 * cfg.kv_heads) * head + h * h
    expert = h * f * (3 if glu else 2)
    params = n_layers * (attn + e * expert + e * h) + v * h * (2 if glu else 1)
    tokens = case['batch'] * case['seq']
    active = n_layers * (attn + cfg.moe_top_k * expert + e * h) + v * h
    flops = 6.0 * tokens * active + n_layers * 3 * 2.0 * tokens * case['seq'] * h
    # Per parameter: fp32 master and both moments read and written, the 16-bit weight read and written.
    return dict(bytes=28.0 * params, flops=flops)


def work(case):
    if case['kind'] == 'layer':
        return _work_layer(case)
    if case['kind'] == 'gmm':
        m, k, n, g = case['rows'], case['k'], case['n'], case['groups']
        return dict(bytes=2.0 * (2 * m * k + 2 * m * n + 2 * g * k * n), flops=6.0 * m * k * n)
    if case['kind'] == 'sparse':
        m, k, n = case['rows'], case['k'], case['cols']
        return dict(bytes=2.0 * (4 * m * k + 4 * n * k), flops=12.0 * m * k * n * case['density'])
    return _work_step(case)


def tolerance(case):
    # About four times the distance of a layer's outputs and gradients from the same layer in 64 bits
    # with the same expert choice (2048 x 512 x 2048, 16 experts, MLP / GLU / token-dropping, top-1 / 2 / 4):
    # bf16 up to 5.5e-3 in norm and 0.09 in the worst element, fp16 up to 6.4e-4 and 0.01.
    if case['kind'] == 'step':
        # Weights after one step: the clip coefficient's sum has no fixed order, so the same step
        # taken twice differs by 2e-4 in norm (most of it in the loss) and 4e-3 in the worst element.
        return {'rel': 1e-3, 'max': 0.02}
    return {'rel': 2.5e-3, 'max': 0.06} if case['dtype'] == 'fp16' else {'rel': 2e-2, 'max': 0.5}


# ----------------------------------------------------------------------------
# The same pass in 64 bits, in plain torch
# ----------------------------------------------------------------------------
def _exact_layer(case, state):
    train, top_k, experts = case['train'], case['top_k'], case['experts']
    dtype, glu = _DTYPES[case['dtype']], case['mlp'] == 'glu'
    names = [name for name, _ in state['layer'].named_parameters()]
    params = [p.detach().double().requires_grad_(train) for p in state['params']]
    by_name = {name.rsplit('.', 1)[-1]: p for name, p in zip(names, params)}
    x = state['x'].detach().double().requires_grad_(train)
    rows = x.reshape(-1, case['hidden'])
    logits = rows @ by_name['weight'].t()
    with torch.no_grad():       # the choice is made on scores rounded to the layer's type, ties to the lowest id
        rounded = logits.to(dtype).double().softmax(-1).to(dtype)
        choice = torch.sort(rounded.float(), dim=-1, descending=True, stable=True)[1][:, :top_k]
    scores = logits.softmax(-1)
    weights = scores.gather(1, choice)
    if glu:
        weights = weights / weights.abs().sum(-1, keepdim=True)
    counts = torch.bincount(choice.flatten(), minlength=experts)
    capacity = int(top_k * case['tokens'] / experts) or int(counts.max())
    out = 0
    for e in range(experts):
        token, slot = (choice == e).nonzero(as_tuple=True)      # in token order
        if not case['dropless']:
            token, slot = token[:capacity], slot[:capacity]
        w1, w2 = by_name['w1'].view(experts, -1, by_name['w1'].shape[-1])[e], by_name['w2'].view(
            experts, -1, case['hidden'])[e]
        z = rows[token] @ (w1.t() if case['dropless'] else w1)
        if glu:
            h = F.silu(z) * (rows[token] @ by_name['v1'].view(experts, -1, case['hidden'])[e].t())
        else:
            h = F.gelu(z, approximate='tanh')
        y = (h @ w2) * weights[token, slot].unsqueeze(1)
        out = out + torch.zeros_like(rows).index_add(0, token, y)
    if 'bias' in by_name:
        out = out + by_name['bias']
    out = out.view(x.shape)
    if not train:
        return out
    aux = experts * 0.1 / (case['tokens'] * top_k) * torch.dot(counts.double(), scores.mean(0))
    grads = torch.autograd.grad([out, aux], [x] + params, [state['dy'].double(), state['one'].double()])
    return [out.detach(), aux.detach(), *grads]


def _exact_gmm(case, state):
    a, b = (state[n].detach().double().requires_grad_(True) for n in ('a', 'b'))
    sizes = state['sizes'].tolist()
    out = torch.cat([part @ (b[g].t() if case['trans_b'] else b[g]) for g, part in enumerate(a.split(sizes))])
    return [out.detach(), *torch.autograd.grad(out, [a, b], state['dy'].double())]


def _exact_sparse(case, state):
    x, w1, w2 = (state[n].detach().double().requires_grad_(True) for n in ('x', 'w1', 'w2'))
    topo = state['topo']
    present = torch.zeros(case['rows'] // _BLOCK, case['cols'] // _BLOCK, device='cuda', dtype=torch.float64)
    present[topo.row_indices.long(), topo.column_indices.long()] = 1
    mask = present.repeat_interleave(_BLOCK, 0).repeat_interleave(_BLOCK, 1)
    out = (F.gelu(x @ w1.t(), approximate='tanh') * mask) @ w2
    return [out.detach(), *torch.autograd.grad(out, [x, w1, w2], state['dy'].double())]


def exact(case, seed):
    if case['kind'] == 'step':
        return None
    # The expert loop keeps one [tokens, hidden] array per expert for its backward pass.
    if case['kind'] == 'layer' and 8 * case['tokens'] * case['hidden'] * case['experts'] > 40e9:
        return None
    return {'layer': _exact_layer, 'gmm': _exact_gmm, 'sparse': _exact_sparse}[case['kind']](case, prepare(case, seed))
