"""What decides whether the fused paths of decoding and training may stand in for the individual operations."""
import pytest
import torch
import torch.nn as nn
from torch.utils.flop_counter import FlopCounterMode

from flash_pop_b200 import layer_ops, token_stack


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
