"""What decides whether the fused paths of decoding and training may stand in for the individual operations."""
import pytest
import torch
import torch.nn as nn
from torch.utils.flop_counter import FlopCounterMode

from flash_pop_b200 import _lib, layer_ops, token_stack


def test_nothing_is_watching():
    assert not layer_ops.observed()


def test_both_paths_ask_the_same_questions():
    assert token_stack.observed is layer_ops.observed and token_stack.plain_linear is layer_ops.plain_linear


def test_every_observer_is_seen():
    seen = []

    def ask(t):
        seen.append(layer_ops.observed())
        return t

    x = torch.ones(2)
    torch.vmap(ask)(x)
    torch.func.grad(lambda t: ask(t).sum())(x)
    torch.func.jvp(ask, (x,), (x,))
    with torch.autograd.forward_ad.dual_level():
        ask(x)
    with FlopCounterMode(display=False):
        ask(x)
    with torch.overrides.TorchFunctionMode():
        ask(x)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        watching = torch.is_autocast_enabled("cuda")           # (off where there is no CUDA device)
        assert layer_ops.observed() == watching
    handle = nn.modules.module.register_module_forward_hook(lambda *a: None)
    ask(x)
    handle.remove()
    torch.jit.trace(ask, x, check_trace=False)
    assert len(seen) == 8 and all(seen)


@pytest.mark.parametrize("owner,name", [(torch._C, "_len_torch_dispatch_stack"), (torch._C, "_len_torch_function_stack"),
                                        (torch._C._functorch, "maybe_current_level"), (torch.autograd.forward_ad, "_current_level")])
def test_a_name_that_torch_no_longer_has_leaves_the_individual_operations(monkeypatch, owner, name):
    monkeypatch.delattr(owner, name)
    assert layer_ops.observed()


def test_plain_linear():
    assert layer_ops.plain_linear(nn.Linear(2, 2))

    class Sub(nn.Linear):
        pass

    hooked = [nn.Linear(2, 2) for _ in range(5)]
    hooked[0].register_forward_hook(lambda *a: None)
    hooked[1].register_forward_pre_hook(lambda *a: None)
    hooked[2].register_full_backward_hook(lambda *a: None)
    hooked[3].register_full_backward_pre_hook(lambda *a: None)
    hooked[4].forward = lambda t: t
    assert not any(layer_ops.plain_linear(m) for m in (Sub(2, 2), nn.Identity(), None, *hooked))


def _grouped():
    """The Functions of the training path and the modules they stand in for, on the CPU (fp32): (function, plain, leaves)."""
    torch.manual_seed(0)
    p = lambda *s: nn.Parameter(torch.randn(*s) * 0.1)
    x, ws, bs = torch.randn(2, 9, 64, requires_grad=True), [p(64, 64) for _ in range(3)], [p(64) for _ in range(3)]
    F = torch.nn.functional
    yield (lambda h: sum(o.square().sum() for o in layer_ops.SharedInputLinears.apply(h, *(t for pair in zip(ws, bs) for t in pair))),
           lambda h: sum(F.linear(h, w, b).square().sum() for w, b in zip(ws, bs)), x, [*ws, *bs])
    w1, b1, w2, b2 = p(128, 64), p(128), p(64, 128), p(64)
    yield (lambda h: layer_ops.SwishFeedForward.apply(h, w1, b1, w2, b2).square().sum(),
           lambda h: F.linear(F.silu(F.linear(h, w1, b1)), w2, b2).square().sum(), x, [w1, b1, w2, b2])


def _close(a, b):
    # the same products added up in another order: a random walk over some 10^3 roundings of 2^-24, 2e-6 of the tensor's norm
    assert float((a - b).norm()) <= 1e-5 * float(b.norm())


@pytest.mark.parametrize("which", [0, 1])
def test_only_the_gradients_asked_for_are_made(which):
    """autograd.grad(y, x) and backward(inputs=...) cost no more products than through the modules, and every subset of
    the gradients is right."""
    _lib.build()
    function, plain, x, params = list(_grouped())[which]

    def grads(f, wanted):
        h = x * 1
        y = f(h)
        with FlopCounterMode(display=False) as count:
            got = torch.autograd.grad(y, [h if t is x else t for t in wanted])
        return got, count.get_total_flops()

    for wanted in ([x], [params[0]], params[-1:], params, [x, params[1]], [x, *params]):
        got, flops = grads(function, wanted)
        want, most = grads(plain, wanted)
        assert flops <= most, (flops, most)
        for a, b in zip(got, want):
            _close(a, b)
    for p in params:
        p.grad = None
    function(x).backward(inputs=[params[0]])
    assert params[0].grad is not None and x.grad is None and all(p.grad is None for p in params[1:])
    frozen = [p.requires_grad_(False) for p in params[:1]]
    got, _ = grads(function, [x])
    for a, b in zip(got, grads(plain, [x])[0]):
        _close(a, b)
    assert not any(p.requires_grad for p in frozen)
    params[0].requires_grad_(True)
    h = x * 1                                          # a graph of the backward: second derivatives, of a subset too
    (g,) = torch.autograd.grad(function(h), [h], create_graph=True)
    (g0,) = torch.autograd.grad(plain(h), [h], create_graph=True)
    second = lambda t: torch.autograd.grad(t.square().sum(), [x, params[0]], retain_graph=True)
    for a, b in zip(second(g), second(g0)):
        _close(a, b)
