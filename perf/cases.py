"""Workloads of this library on one GPU, from a single decode token to a full training step, for timing and for comparing outputs.

Every case runs through the public entry points (``ElasticBuffer``, ``FusedMoE``, ``ops.gemm``) with the settings a user's
program has.  Sizes are those of the repository's own benchmarks and tests: 4096 / 8192 tokens per rank, hidden 7168 (4096 for
the Zipf workload), top-8 of 256 / top-6 of 64 experts, intermediate 2048 with the 32 experts that one rank of eight holds.
Data is synthetic: N(0, 1) tokens, softmax routing weights, N(0, 0.02) layer weights.

    listed()        the cases
    draw(rng)       one more case of the same ranges
    prepare / run   inputs and kept state of a case / one pass
    work            bytes and operations that one pass cannot do without
    tolerance       how far the outputs of another correct implementation may be off
    exact           the computed outputs in 64 bits, without this library's code
"""
import math

import torch

from deepep_ascend_b200 import ElasticBuffer
from deepep_ascend_b200.models.moe import FusedMoE
from deepep_ascend_b200.ops import gemm as G


def listed():
    return [
        # The smallest exchange: a few dozen tokens of a nearly idle server, rows cast to e4m3 on the way; launch and host time.
        dict(name='ep_forward_61', kind='ep', tokens=61, hidden=7168, topk=8, experts=256, fp8=True, expand=False, backward=False,
             prequantized=False, plain=False, sms=0, masked=0.0, zipf=0.0),
        # The headline exchange of the benchmark: prefill / training forward of 8192 tokens, experts write the combine region.
        dict(name='ep_forward_8192', kind='ep', tokens=8192, hidden=7168, topk=8, experts=256, fp8=True, expand=False, backward=False,
             prequantized=False, plain=False, sms=0, masked=0.0, zipf=0.0),
        # The same exchange beside compute kernels: 24 SMs, tokens quantised by the layer before, an odd token count, expert
        # outputs in an ordinary tensor.
        dict(name='ep_forward_24sms', kind='ep', tokens=5003, hidden=7168, topk=8, experts=256, fp8=True, expand=False, backward=False,
             prequantized=True, plain=True, sms=24, masked=0.0, zipf=0.0),
        # A training step's four exchanges in bf16 (4096 tokens, top-6): dispatch, combine, and their backward passes (a dispatch
        # with the cached layout, a combine that carries the routing-weight gradients home).
        dict(name='ep_train_4096', kind='ep', tokens=4096, hidden=7168, topk=6, experts=256, fp8=False, expand=False, backward=True,
             prequantized=False, plain=True, sms=0, masked=0.0, zipf=0.0),
        # One row per (token, expert) for a caller with its own grouped GEMM: skewed routing, dropped selections, zeroed
        # alignment rows, routing weights applied in the combine.
        dict(name='ep_expand_3001', kind='ep', tokens=3001, hidden=4096, topk=6, experts=64, fp8=False, expand=True, backward=False,
             prequantized=False, plain=False, sms=0, masked=0.1, zipf=1.2),
        # Decode exchange without a CUDA graph, bf16 rows, a ragged batch.
        dict(name='ll_decode_40', kind='ll', tokens=40, hidden=7168, topk=8, experts=256),
        # A decode MoE layer as a server replays it: low-latency dispatch (e4m3), two grouped GEMMs, low-latency combine, all
        # in one CUDA graph; 32 experts per rank.
        dict(name='ll_moe_graph_128', kind='ll_moe', tokens=128, hidden=7168, topk=8, experts=32, inter=2048),
        # The fused layer at inference: a short prompt (bound by the experts' weights) ...
        dict(name='moe_forward_64', kind='moe', tokens=64, hidden=7168, topk=8, experts=32, inter=2048, mode='infer'),
        # ... and a long one.
        dict(name='moe_forward_4096', kind='moe', tokens=4096, hidden=7168, topk=8, experts=32, inter=2048, mode='infer'),
        # One optimizer step of the layer: new bf16 weights arrive from the optimizer, forward, backward in bf16.
        dict(name='moe_step_4096', kind='moe', tokens=4096, hidden=7168, topk=8, experts=32, inter=2048, mode='step'),
        # One micro-batch of gradient accumulation (the weights stay) of a smaller layer, data gradients in e4m3, ragged batch.
        dict(name='moe_fp8_grad_1999', kind='moe', tokens=1999, hidden=2048, topk=6, experts=32, inter=1024, mode='fp8_grad'),
        # A plain linear layer on the tensor cores.
        dict(name='gemm_8192', kind='gemm', m=8192, n=7168, k=7168),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['ep', 'ep', 'ep', 'll', 'll_moe', 'moe', 'moe', 'moe', 'gemm'])
    if kind == 'gemm':
        return dict(kind='gemm', m=_log_int(rng, 64, 8192), n=8 * _log_int(rng, 16, 896), k=8 * _log_int(rng, 16, 896))
    hidden = 128 * _log_int(rng, 4, 56)
    if kind == 'll':
        return dict(kind='ll', tokens=_log_int(rng, 1, 128), hidden=hidden, topk=rng.randint(1, 8), experts=rng.choice([16, 64, 160, 256]))
    if kind == 'll_moe':
        return dict(kind='ll_moe', tokens=_log_int(rng, 1, 128), hidden=hidden, topk=rng.randint(2, 8), experts=rng.choice([8, 16, 24, 32]),
                    inter=128 * rng.randint(2, 16))
    if kind == 'moe':
        return dict(kind='moe', tokens=_log_int(rng, 16, 4096), hidden=hidden, topk=rng.randint(2, 8), experts=rng.choice([8, 16, 24, 32]),
                    inter=128 * rng.randint(2, 16), mode=rng.choice(['infer', 'step', 'fp8_grad']))
    fp8, expand = rng.random() < 0.5, rng.random() < 0.3
    return dict(kind='ep', tokens=_log_int(rng, 8, 8192), hidden=hidden, topk=rng.randint(1, 8), experts=rng.choice([16, 64, 160, 256]),
                fp8=fp8, expand=expand, backward=not expand and rng.random() < 0.4, prequantized=fp8 and rng.random() < 0.3,
                plain=rng.random() < 0.5, sms=rng.choice([0, 0, 24]), masked=rng.choice([0.0, 0.1]), zipf=rng.choice([0.0, 1.2]))


# ---------------------------------------------------------------------------------------------------------------- inputs
def _routing(gen, tokens, experts, topk, masked=0.0, zipf=0.0):
    """Top-k of random gate logits with softmax weights; ``zipf``: expert popularity falls as rank^-zipf; ``masked``: share of
    selections that were dropped (-1).  Every seed has the same tokens' choices in another order, so that the number of rows
    that arrive (and with it the shape of the outputs) belongs to the case."""
    order = torch.randperm(tokens, generator=gen, device='cuda')
    gen = torch.Generator(device='cuda').manual_seed(tokens + experts)
    logits = torch.randn(tokens, experts, generator=gen, device='cuda')
    if zipf:
        logits -= zipf * torch.log(torch.arange(1, experts + 1, device='cuda', dtype=torch.float32))
    weights, idx = torch.softmax(logits, dim=-1).topk(topk, dim=-1)
    if masked:
        idx = torch.where(torch.rand(tokens, topk, generator=gen, device='cuda') < masked, -1, idx)
    return idx[order].contiguous(), weights[order].contiguous()


def _bf16(gen, *shape, std=1.0):
    return torch.empty(shape, dtype=torch.bfloat16, device='cuda').normal_(0.0, std, generator=gen)


def _prepare_ep(c, gen):
    T, H, K, E = c['tokens'], c['hidden'], c['topk'], c['experts']
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K, use_fp8_dispatch=c['fp8'] and not c['backward'],
                        enable_expand=c['expand'], num_experts=E, expert_alignment=128 if c['expand'] else 1)
    idx, w = _routing(gen, T, E, K, c['masked'], c['zipf'])
    x = _bf16(gen, T, H)
    s = dict(buf=buf, x=G.per_token_cast_to_fp8(x) if c['prequantized'] else x, idx=idx, w=w)
    rows = T * K + E * 127 if c['expand'] else T
    y = _bf16(gen, rows, H)
    if c['plain']:
        s['y'] = y
    else:
        # the experts' last GEMM writes into the two combine regions in turn
        for _ in range(2):
            _, _, _, h, _ = buf.dispatch(s['x'], idx, w, num_experts=E, do_expand=c['expand'], expert_alignment=128 if c['expand'] else 1)
            region = buf.get_combine_buffer(h)
            region.copy_(y[:region.shape[0]])
            buf.combine(region, h)
    if c['backward']:
        s['grad'], s['grad_rows'] = _bf16(gen, T, H), _bf16(gen, rows, H)
        s['grad_w'] = torch.randn(rows, K, generator=gen, device='cuda')
    return s


def _run_ep(c, s):
    buf, sms = s['buf'], c['sms']
    recv, recv_idx, recv_w, handle, _ = buf.dispatch(s['x'], s['idx'], s['w'], num_experts=c['experts'], num_sms=sms, do_expand=c['expand'],
                                                     expert_alignment=128 if c['expand'] else 1, do_zero_padding=c['expand'],
                                                     fused_fp8_cast=c['fp8'])
    y = s['y'] if c['plain'] else buf.get_combine_buffer(handle)
    out, _, _ = buf.combine(y, handle, weighted=c['expand'], num_sms=sms)
    res = dict(recv=recv, counts=handle.num_unaligned_recv_tokens_per_expert, out=out)
    if not c['expand']:
        res.update(recv_idx=recv_idx, recv_w=recv_w)
    if c['backward']:
        rows, _, _, _, _ = buf.dispatch(s['grad'], handle=handle, num_sms=sms, fused_fp8_cast=False)
        dx, dw, _ = buf.combine(s['grad_rows'], handle, topk_weights=s['grad_w'], num_sms=sms)
        res.update(grad_rows=rows, dx=dx, dw=dw)
    for v in res.values():           # received rows are views of the buffer: it lives as long as they do
        for t in v if isinstance(v, tuple) else (v,):
            t.owner = buf
    return res


LL_MAX_TOKENS = 128


def _ll_buffer(c):
    extra = ElasticBuffer.get_low_latency_size_hint(LL_MAX_TOKENS, c['hidden'], 1, c['experts'], c['topk'])
    return ElasticBuffer(None, num_max_tokens_per_rank=LL_MAX_TOKENS, hidden=c['hidden'], num_topk=c['topk'], extra_bytes=extra + (1 << 20))


def _prepare_ll(c, gen):
    idx, w = _routing(gen, c['tokens'], c['experts'], c['topk'])
    s = dict(buf=_ll_buffer(c), idx=idx, w=w, x=_bf16(gen, c['tokens'], c['hidden']))
    _run_ll(c, s)
    return s


def _run_ll(c, s):
    recv, count, handle, _, _ = s['buf'].low_latency_dispatch(s['x'], s['idx'], LL_MAX_TOKENS, c['experts'], use_fp8=False)
    out, _, _ = s['buf'].low_latency_combine(recv, s['idx'], s['w'], handle)      # experts that return their input
    return dict(count=count, out=out)


def _prepare_ll_moe(c, gen):
    T, H, I, E = c['tokens'], c['hidden'], c['inter'], c['experts']
    idx, w = _routing(gen, T, E, c['topk'])
    q13, s13 = G.quantize_weight_blocks(_bf16(gen, E, 2 * I, H, std=0.02))
    q2, s2 = G.quantize_weight_blocks(_bf16(gen, E, H, I, std=0.02))
    s = dict(buf=_ll_buffer(c), idx=idx, w=w, x=_bf16(gen, T, H), weights=(q13, s13, q2, s2))
    tiles = torch.arange(E, dtype=torch.int32, device='cuda')       # 128 slots per expert: one tile each

    def layer():
        buf = s['buf']
        (rx, rsf), count, handle, _, _ = buf.low_latency_dispatch(s['x'], idx, LL_MAX_TOKENS, E, use_fp8=True)
        group = torch.where(count > 0, tiles, -1)
        rx, rsf = rx.view(E * LL_MAX_TOKENS, H), rsf.reshape(E * LL_MAX_TOKENS, -1)
        h = G.grouped_gemm_nt(rx, q13, group, sfa=rsf, sfb=s13, buffer=buf)
        a, sfa = G.swiglu_quant(h)
        y = G.grouped_gemm_nt(a, q2, group, sfa=sfa, sfb=s2, buffer=buf)
        out, _, _ = buf.low_latency_combine(y.view(E, LL_MAX_TOKENS, H), idx, w, handle)
        return dict(count=count, out=out)
    for _ in range(2):
        layer()
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        s['out'] = layer()
    s['graph'] = graph
    return s


def _run_ll_moe(c, s):
    s['graph'].replay()
    return s['out']


def _prepare_moe(c, gen):
    T, H, I, E, K = c['tokens'], c['hidden'], c['inter'], c['experts'], c['topk']
    buf = ElasticBuffer(None, num_max_tokens_per_rank=T, hidden=H, num_topk=K)
    layer = FusedMoE(buf, E, H, I, fp8_backward=c['mode'] == 'fp8_grad')
    w13, w2 = _bf16(gen, E, 2 * I, H, std=0.02), _bf16(gen, E, H, I, std=0.02)
    with torch.no_grad():
        layer.w13.copy_(w13)
        layer.w2.copy_(w2)
    idx, w = _routing(gen, T, E, K)
    s = dict(layer=layer, x=_bf16(gen, T, H), idx=idx, w=w)
    if c['mode'] == 'step':
        s['new_w13'], s['new_w2'] = w13, w2
    else:
        layer.fp8_weights()
    if c['mode'] == 'fp8_grad':
        layer.fp8_transposed_weights()
    if c['mode'] != 'infer':
        s['x'].requires_grad_(True)
        s['w'].requires_grad_(True)
        s['grad'] = _bf16(gen, T, H)
    return s


def _run_moe(c, s):
    layer = s['layer']
    if c['mode'] == 'infer':
        with torch.no_grad():
            return layer(s['x'], s['idx'], s['w'])
    if c['mode'] == 'step':
        with torch.no_grad():            # the (sharded) optimizer hands over the bf16 weights of this step
            layer.w13.copy_(s['new_w13'])
            layer.w2.copy_(s['new_w2'])
    out = layer(s['x'], s['idx'], s['w'])
    dx, dw, dw13, dw2 = torch.autograd.grad(out, [s['x'], s['w'], layer.w13, layer.w2], s['grad'])
    return dict(out=out, dx=dx, dw=dw, dw13=dw13, dw2=dw2)


def _prepare_gemm(c, gen):
    return dict(a=_bf16(gen, c['m'], c['k']), b=_bf16(gen, c['n'], c['k'], std=0.02))


def _run_gemm(c, s):
    return G.gemm_nt(s['a'], s['b'])


_KINDS = {'ep': (_prepare_ep, _run_ep), 'll': (_prepare_ll, _run_ll), 'll_moe': (_prepare_ll_moe, _run_ll_moe),
          'moe': (_prepare_moe, _run_moe), 'gemm': (_prepare_gemm, _run_gemm)}


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device='cuda').manual_seed(seed)
    return case, _KINDS[case['kind']][0](case, gen)


def run(state):
    case, s = state
    return _KINDS[case['kind']][1](case, s)


# ------------------------------------------------------------------------------------------------------------------ work
def work(case):
    c = case
    if c['kind'] == 'gemm':
        m, n, k = c['m'], c['n'], c['k']
        return dict(bytes=2 * (m * k + n * k + m * n), flops=2 * m * n * k)
    T, H, K = c['tokens'], c['hidden'], c['topk']
    routing = T * K * 12                                     # int64 ids and fp32 weights
    if c['kind'] == 'ep':
        cast = H + 4 * (H // 128)
        sent = T * (1 - c['masked']) * K if c['expand'] else T
        row = cast if c['fp8'] else 2 * H
        b = T * (cast if c['prequantized'] else 2 * H) + sent * row + routing * (1 if c['expand'] else 2)     # dispatch
        b += sent * 2 * H + T * 2 * H                                                                       # combine
        if c['backward']:
            b += 4 * T * 2 * H + 2 * T * K * 4
        return dict(bytes=b, flops=0)
    if c['kind'] == 'll':
        # every selection's row is delivered, read back and reduced
        return dict(bytes=T * 2 * H + T * K * 2 * H + T * K * 2 * H + T * 2 * H + 2 * routing, flops=2 * T * K * H)
    I, E = c['inter'], c['experts']
    weights = E * 3 * I * H                                  # elements
    touched = weights * (1 - (1 - K / E) ** T)               # of the experts that get a token
    flops = 6 * T * K * H * I
    b = touched + T * 2 * H * 2 + routing                    # e4m3 weights, tokens in and out
    if c['kind'] == 'moe' and c['mode'] != 'infer':
        flops *= 3
        # weights once more for the data gradients, both weight gradients out, output gradient in, token gradient out
        b += touched * (1 if c['mode'] == 'fp8_grad' else 2) + 2 * weights + 2 * T * 2 * H + T * K * 4
        if c['mode'] == 'step':
            b += 2 * weights + 2 * weights + weights         # new bf16 weights read and stored, e4m3 copies written
    return dict(bytes=b, flops=flops)


def tolerance(case):
    c = case
    if c['kind'] == 'ep':
        # copies, casts and sums of one row are the same bits everywhere; K weighted rows may be added in another order
        return {'rel': 1e-3, 'max': 0.03} if c['expand'] else 'exact'
    if c['kind'] in ('ll', 'gemm'):
        # fp32 sums in another order, rounded to bf16: measured 1.4e-4 / 7.8e-3 (one rounding step) with k permuted
        return {'rel': 1e-3, 'max': 0.03}
    # Permuting the reduction dimensions gives up to 9.7e-4 / 2.3e-2 (token gradient, weight gradient of the bf16 backward pass)
    return {'rel': 4e-3, 'max': 0.1}


# ----------------------------------------------------------------------------------------------------------------- exact
def _exact_moe(x, idx, w, w13, w2, grad=None):
    """The SwiGLU expert layer and its gradients in 64 bits, one expert at a time."""
    I = w2.shape[2]
    out, dx, dw = (torch.zeros(t.shape, dtype=torch.float64, device='cuda') for t in (x, x, w))
    dw13, dw2 = [], []
    for e in range(w2.shape[0]):
        t, k = (idx == e).nonzero(as_tuple=True)
        a13, a2, xe, we = w13[e].double(), w2[e].double(), x[t].double(), w[t, k].double().unsqueeze(1)
        h = xe @ a13.t()
        gate, up = h[:, :I], h[:, I:]
        sig = torch.sigmoid(gate)
        act = gate * sig * up
        y = act @ a2.t()
        out.index_add_(0, t, we * y)
        if grad is None:
            continue
        g = grad[t].double()
        dw[t, k] = (g * y).sum(1)
        d_act = (we * g) @ a2
        dh = torch.cat([d_act * up * sig * (1 + gate * (1 - sig)), d_act * gate * sig], dim=1)
        dx.index_add_(0, t, dh @ a13)
        dw2.append((we * g).t() @ act)
        dw13.append(dh.t() @ xe)
    return out if grad is None else dict(out=out, dx=dx, dw=dw, dw13=torch.stack(dw13), dw2=torch.stack(dw2))


def exact(case, seed):
    """The computed outputs of ``run`` from the same inputs in 64 bits; ``None`` where an output is a copy or a cast."""
    c = case
    torch.manual_seed(seed)
    gen = torch.Generator(device='cuda').manual_seed(seed)
    if c['kind'] == 'gemm':
        s = _prepare_gemm(c, gen)
        return s['a'].double() @ s['b'].double().t()
    T, H, K, E = c['tokens'], c['hidden'], c['topk'], c['experts']
    if c['kind'] == 'ep':
        if not c['expand']:
            return None
        idx, w = _routing(gen, T, E, K, c['masked'], c['zipf'])
        _bf16(gen, T, H)
        y = _bf16(gen, T * K + E * 127, H)
        out, row0 = torch.zeros(T, H, dtype=torch.float64, device='cuda'), 0
        for e in range(E):
            t, k = (idx == e).nonzero(as_tuple=True)            # rows of an expert: in token order, segments 128-aligned
            out.index_add_(0, t, w[t, k].double().unsqueeze(1) * y[row0:row0 + t.numel()].double())
            row0 += (t.numel() + 127) // 128 * 128
        return dict(recv=None, counts=None, out=out)
    if c['kind'] == 'll':
        idx, w = _routing(gen, T, E, K)
        return dict(count=None, out=_bf16(gen, T, H).double() * w.double().sum(1, keepdim=True))
    I = c['inter']
    if c['kind'] == 'll_moe':
        idx, w = _routing(gen, T, E, K)
        w13, w2 = _bf16(gen, E, 2 * I, H, std=0.02), _bf16(gen, E, H, I, std=0.02)
        return dict(count=None, out=_exact_moe(_bf16(gen, T, H), idx, w, w13, w2))
    w13, w2 = _bf16(gen, E, 2 * I, H, std=0.02), _bf16(gen, E, H, I, std=0.02)
    idx, w = _routing(gen, T, E, K)
    x = _bf16(gen, T, H)
    return _exact_moe(x, idx, w, w13, w2, None if c['mode'] == 'infer' else _bf16(gen, T, H))
