"""Prediction suffixes that one CTA walks back to back remain sequences of their own."""
import pytest
import torch

from oracle import retention_oracle as orc

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _case(B, M, N, P, H, dk, dv, state_dtype=BF, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda") * dk ** -0.5
    sq, sk, sv, do = (r(B, M, P, H, d).to(BF) for d in (dk, dk, dv, dv))
    return [sq, sk, sv, r(B, H, dk, dv).to(state_dtype), r(B, N, H, dk, dv).to(state_dtype)], do


def _run(tensors, do, decays):
    import flash_pop_b200 as fp
    from flash_pop_b200 import _lib
    leaves = [t.detach().clone().requires_grad_(True) for t in tensors]
    o = fp.pop_suffix_retention(*leaves, decays)
    assert _lib.last_path() == _lib.PATH_TCGEN05
    out = [o.detach(), *torch.autograd.grad(o, leaves, do)]
    _lib.device_status()
    return out


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("P,dk,dv", [(80, 64, 64), (40, 64, 64), (17, 64, 64), (80, 128, 128), (100, 64, 128)])
def test_no_suffix_sees_the_next_one(P, dk, dv, bad):
    """Infinities and NaN in one suffix, first of a batch row or not, reach the gradients of that suffix alone: what
    follows a suffix in memory is nothing to it, as it is when every suffix has a CTA to itself."""
    B, M, H = 2, 60, 3                 # 120 suffixes a head: two or more a CTA in every walk
    decays = tuple(orc.head_decays(H, (5, 12)))
    tensors, do = _case(B, M, M, P, H, dk, dv)
    clean = _run(tensors, do, decays)
    for row, m in ((1, 0), (1, 1), (0, 7)):
        spoilt = [t.clone() for t in tensors]
        for t in spoilt[:3]:
            t[row, m] = bad
        do2 = do.clone()
        do2[row, m] = bad
        got = _run(spoilt, do2, decays)
        keep = torch.ones(B, M, dtype=torch.bool, device="cuda")
        keep[row, m] = False
        for a, b in zip(got[:4], clean[:4]):           # o, dQ, dK, dV by suffix
            assert torch.equal(a[keep], b[keep])
        rows = torch.arange(B, device="cuda") != (row if m == 0 else -1)
        assert torch.equal(got[4][rows], clean[4][rows])                 # start states: suffix 0's own
        blocks = torch.ones(B, M, dtype=torch.bool, device="cuda")
        if m > 0:
            blocks[row, m - 1] = False
        assert torch.equal(got[5][blocks], clean[5][blocks])             # block states: where a later suffix starts


@pytest.mark.parametrize("state_dtype", [BF, torch.float32])
@pytest.mark.parametrize("B,M,N,P,H,dk,dv", [
    (3, 50, 50, 80, 3, 64, 64), (7, 23, 22, 17, 5, 64, 64), (2, 75, 75, 64, 4, 64, 64), (5, 40, 41, 65, 2, 128, 128), (1, 200, 199, 80, 2, 64, 128),
    (4, 40, 40, 16, 75, 64, 64), (3, 8, 8, 130, 160, 64, 64)])
def test_the_shipped_sharing_equals_one_cta_per_suffix(B, M, N, P, H, dk, dv, state_dtype):
    """Uneven pieces, pieces across batch rows, several waves of heads, both state types: bit for bit what one CTA per suffix
    gives.  (Counts of suffixes and heads that the shipped rule groups; row by row, few suffixes a call, it does not.)"""
    from flash_pop_b200 import _lib
    decays = tuple(orc.head_decays(H, (5, 12)))
    tensors, do = _case(B, M, N, P, H, dk, dv, state_dtype, seed=M)
    grouped = _run(tensors, do, decays)
    with _lib.diagnostics_build() as diag:
        try:
            diag.fpb_debug_suffix_group(1, 0)
            single = _run(tensors, do, decays)
        finally:
            diag.fpb_debug_suffix_group(1 << 20, 0)
    for a, b in zip(grouped, single):
        assert torch.equal(a, b)
    rows = orc.pop_suffix_retention(*(t[:1, :, :, :2].double().cpu() for t in tensors[:3]), tensors[3][:1, :2].double().cpu(),
                                    tensors[4][:1, :, :2].double().cpu(), decays[:2])
    assert orc.rel_rms(grouped[0][:1, :, :, :2].float().cpu(), rows) < 5e-3
