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


@pytest.mark.parametrize("B,H,apart", [(1, 74, False), (1, 75, True), (4, 37, True), (1, 149, False), (1, 222, False), (1, 223, True)])
def test_which_calls_keep_the_halves_apart(B, H, apart):
    """Apart where two launches of one half take no more waves than one of both: four launches of walks in the backward, the
    last of which the diagnostics build can refuse; together there are two, over outputs zeroed first."""
    import flash_pop_b200 as fp
    from flash_pop_b200 import _lib
    assert torch.cuda.get_device_properties(0).multi_processor_count == 148
    decays = tuple(orc.head_decays(H, (5, 12)))
    r = lambda d: (torch.randn(B, 70, H, d, device="cuda") * 0.1).bfloat16()
    q, k, v, dO = r(128).requires_grad_(True), r(128).requires_grad_(True), r(256).requires_grad_(True), r(256)
    with _lib.diagnostics_build() as diag:
        try:
            o, _ = fp.fused_chunk_retention(q, k, v, None, decays)
            want = torch.autograd.grad(o, [q, k, v], dO, retain_graph=True)
            diag.fpb_debug_refuse_launch(3)
            if apart:
                with pytest.raises(RuntimeError, match="launch"):
                    torch.autograd.grad(o, [q, k, v], dO, retain_graph=True)
            else:
                got = torch.autograd.grad(o, [q, k, v], dO, retain_graph=True)
                assert all(torch.equal(a, b) for a, b in zip(got, want))
        finally:
            diag.fpb_debug_refuse_launch(-1)
    _lib.device_status()
