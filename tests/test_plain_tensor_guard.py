"""Where a kernel stands in for a PyTorch statement, tracers, transforms and dispatch modes must still see the statement."""
import pytest
import torch

from deepep_ascend_b200.ops import gemm as ops


def _watchers():
    """name -> call(f, x): runs f(x) with something that records, transforms or intercepts operations."""
    from torch._subclasses import FakeTensorMode
    from torch.fx.experimental.proxy_tensor import make_fx
    from torch.utils.flop_counter import FlopCounterMode

    def under(mode):
        def call(f, x):
            with mode:
                return f(x)
        return call

    def dual(f, x):
        with torch.autograd.forward_ad.dual_level():
            return f(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)))
    return {
        'jit.trace': lambda f, x: torch.jit.trace(f, x, check_trace=False),
        'make_fx': lambda f, x: make_fx(f)(x),
        'make_fx symbolic': lambda f, x: make_fx(f, tracing_mode='symbolic')(x),
        'dispatch mode': under(FlopCounterMode(display=False)),
        'fake tensors': under(FakeTensorMode(allow_non_fake_inputs=True)),
        'functionalize': lambda f, x: torch.func.functionalize(f)(x),
        'vmap': lambda f, x: torch.vmap(f)(x.unsqueeze(0)),
        'forward mode': dual,
        'gradient': lambda f, x: f(x.clone().requires_grad_(True)),
    }


@pytest.mark.parametrize('name', sorted(_watchers()))
def test_watched_tensors_are_not_plain(name):
    seen = []

    def f(x):
        seen.append(ops._plain(x))
        return x * 2
    x = torch.randn(2, 4)
    assert ops._plain(x) and ops._plain(torch.nn.Parameter(x, requires_grad=False))
    with torch.no_grad():
        assert ops._plain(torch.nn.Parameter(x))
    _watchers()[name](f, x)
    assert seen and not any(seen)
    assert ops._plain(x)


@pytest.mark.gpu
@pytest.mark.parametrize('tracer', ['jit.trace', 'make_fx'])
def test_traced_weight_cast_replays_on_new_weights(tracer):
    """A recorded cast gives the bits of the PyTorch statement for weights that it has not seen (TorchScript's own fuser, which does
    not know e4m3, stays out)."""
    w = torch.randn(2, 136, 264, device='cuda').bfloat16()
    traced = _watchers()[tracer](ops.quantize_weight_blocks, w)
    for v in (w, torch.randn_like(w) * 3):
        with torch.jit.optimized_execution(False):
            q, sf = traced(v)
        q_ref, sf_ref = ops.quantize_weight_blocks_ref(v)
        assert torch.equal(q.view(torch.uint8), q_ref.view(torch.uint8)) and torch.equal(sf, sf_ref)
