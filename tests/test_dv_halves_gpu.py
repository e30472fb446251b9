"""dv = 256 gradient walks: the two halves of dv as launches of their own (the second adds to what the first stored) give bit
for bit what one launch of both over a zeroed output gives, at the numbers of heads where the choice changes."""
import pytest
import torch

from oracle import retention_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T,state", [(2, 37, 130, torch.bfloat16), (5, 15, 130, torch.bfloat16), (5, 15, 64, torch.float32), (4, 37, 71, None),
                                         (1, 149, 65, torch.bfloat16)])
def test_halves_apart_equal_halves_together(B, H, T, state):
    import flash_pop_b200 as fp
    from flash_pop_b200 import _lib
    dk, dv = 128, 256
    decays = tuple(orc.head_decays(H, (5, 12)))
    g = torch.Generator(device="cuda").manual_seed(H)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda") * 0.1
    q, k, v, dO = (r(B, T, H, d).bfloat16() for d in (dk, dk, dv, dv))
    s = None if state is None else r(B, H, dk, dv).to(state)

    def grads(rows, heads):
        x = [t[rows][:, :, heads].contiguous().requires_grad_(True) for t in (q, k, v)]
        s0 = None if s is None else s[rows][:, heads].contiguous().requires_grad_(True)
        o, _ = fp.fused_chunk_retention(*x, s0, decays[heads])
        n0 = _lib.launch_count()
        out = torch.autograd.grad(o, x + ([] if s0 is None else [s0]), dO[rows][:, :, heads].contiguous())
        assert _lib.launch_count() - n0 == 4           # two halves each way, or a zero fill and a launch each way
        return out

    whole = grads(slice(0, B), slice(0, H))
    _lib.device_status()
    for lo in range(0, H, 37):                         # few heads at a time: always together
        heads = slice(lo, min(lo + 37, H))
        for b in range(B):
            for i, (a, c) in enumerate(zip(whole, grads(slice(b, b + 1), heads))):
                want = a[b:b + 1][:, :, heads] if i < 3 else a[b:b + 1][:, heads]
                assert torch.equal(want, c)
