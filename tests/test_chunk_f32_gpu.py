"""The chunked fp32 kernels against the oracle in 64 bits at the edges of chunks, segments and head dimensions, and what
they must share with the token walk they stand in for: strides, missing states, partial gradients, scratch limits, decays
down to 0, and no trace of a later token in an earlier one."""
import ctypes

import pytest
import torch

from oracle import retention_oracle as orc

pytestmark = pytest.mark.gpu
# sums of some 10^2 to 10^3 products, rounded to 2^-24 each: a random walk of 2^-24 sqrt(10^3) = 1.9e-6
REL = 2e-6


def _inputs(seed, B, T, H, dk, dv, state=True):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s, scale=1.0: torch.randn(*s, generator=g) * scale
    return (r(B, T, H, dk, scale=dk ** -0.5), r(B, T, H, dk, scale=dk ** -0.5), r(B, T, H, dv, scale=dk ** -0.5),
            r(B, H, dk, dv, scale=0.1) if state else None, r(B, T, H, dv), r(B, H, dk, dv) if state else None)


def _rel(a, b):
    return float((a.detach().double().cpu() - b).norm() / b.norm())


def _check(q, k, v, s, dO, dS, decays, rel=REL):
    import flash_pop_b200 as fp
    from flash_pop_b200 import _lib
    leaves = [t.detach().cuda().requires_grad_(True) for t in (q, k, v, s) if t is not None]
    qc, kc, vc = leaves[:3]
    o, s_out = fp.fused_chunk_retention(qc, kc, vc, leaves[3] if s is not None else None, decays)
    assert _lib.last_path() == _lib.PATH_SIMT
    ends, grads = ([o, s_out], [dO.cuda(), dS.cuda()]) if dS is not None else ([o], [dO.cuda()])
    got = torch.autograd.grad(ends, leaves, grads)
    d32 = [float(torch.tensor(g, dtype=torch.float32)) for g in decays]       # the operator rounds decays to fp32
    wide = [t.double().requires_grad_(True) for t in (q, k, v, s) if t is not None]
    o_ref, s_ref = orc.retention_chunkwise(*wide[:3], wide[3] if s is not None else torch.zeros(q.shape[0], q.shape[2], q.shape[3], v.shape[3], dtype=torch.float64), d32, 64)
    ref = torch.autograd.grad([o_ref, s_ref][:len(ends)], wide, [g.double().cpu() for g in grads])
    for name, a, b in [("o", o, o_ref), ("s_out", s_out, s_ref)] + list(zip("qkvs", got, ref)):
        assert _rel(a, b.detach()) < rel, f"{name}: {_rel(a, b.detach()):.2e}"


@pytest.mark.parametrize("B,T,H,dk,dv,state", [
    (1, 16, 1, 32, 32, False), (2, 31, 3, 64, 64, True), (1, 32, 2, 64, 128, True), (2, 33, 2, 128, 64, True), (2, 256, 4, 64, 64, False),
    (4, 1024, 8, 128, 128, True), (1, 1023, 1, 32, 128, True), (3, 97, 5, 36, 20, True), (1, 300, 2, 100, 68, True), (2, 64, 2, 4, 4, True),
    (1, 2500, 1, 64, 64, True), (40, 70, 8, 32, 64, True), (1, 129, 1, 128, 32, False)])
def test_against_64_bits(B, T, H, dk, dv, state):
    _check(*_inputs(T + dk, B, T, H, dk, dv, state), orc.head_decays(H, (5, 12) if H > 1 else None))


@pytest.mark.parametrize("decays", [(1.0, 0.0), (0.25, 0.5), (0.999, 1e-30)])
def test_any_decay(decays):
    _check(*_inputs(3, 2, 90, 2, 32, 32), decays)


def test_strided_views_match_contiguous_ones_and_partial_gradients_match_full_ones():
    import flash_pop_b200 as fp
    decays = orc.head_decays(3, (5, 12))
    q, k, v, s, dO, dS = (t.cuda() for t in _inputs(5, 2, 75, 3, 64, 32))
    packed = torch.cat((q, k, v, dO), -1)
    views = [t.detach().requires_grad_(True) for t in packed.split([64, 64, 32, 32], -1)[:3]]
    turned = [t.transpose(1, 2).contiguous().transpose(1, 2).requires_grad_(True) for t in (q, k, v)]
    plain = [t.clone().requires_grad_(True) for t in (q, k, v)]
    results = []
    for x in (plain, views, turned):
        o, s_out = fp.fused_chunk_retention(*x, s, decays)
        results.append([o, s_out, *torch.autograd.grad(o, x, packed[..., 160:] if x is views else dO)])
    for other in results[1:]:
        assert all(torch.equal(a, b) for a, b in zip(results[0], other))
    for i in range(3):                               # one gradient at a time: dQ alone, dK / dV alone
        x = [t.detach().requires_grad_(j == i) for j, t in enumerate(plain)]
        o, _ = fp.fused_chunk_retention(*x, s, decays)
        (g,) = torch.autograd.grad(o, [x[i]], dO)
        assert torch.equal(g, results[0][2 + i])


def test_later_tokens_leave_no_trace():
    import flash_pop_b200 as fp
    decays = orc.head_decays(2, (5, 12))
    for bad in (float("inf"), float("nan")):
        for cut in (1, 5, 31, 32, 50):
            q, k, v, s, dO, _ = (t.cuda() for t in _inputs(9, 1, 70, 2, 32, 64))
            clean, _ = fp.fused_chunk_retention(q, k, v, s, decays)
            k2, v2 = k.clone(), v.clone()
            k2[:, cut:], v2[:, cut:] = bad, bad
            o, _ = fp.fused_chunk_retention(q, k2, v2, s, decays)
            assert torch.equal(o[:, :cut], clean[:, :cut])
            x = [t.clone().requires_grad_(True) for t in (q, k, v)]      # and the gradients of later tokens see no earlier ones
            d2 = dO.clone()
            d2[:, :cut] = bad
            ref = torch.autograd.grad(fp.fused_chunk_retention(*x, s, decays)[0], x, dO)
            got = torch.autograd.grad(fp.fused_chunk_retention(*x, s, decays)[0], x, d2)
            for a, b in zip(got, ref):
                assert torch.equal(a[:, cut:], b[:, cut:])


def test_scratch_limits_change_the_split_only():
    from flash_pop_b200 import _lib
    B, T, H, d = 2, 500, 3, 64
    decays = orc.head_decays(H, (5, 12))
    q, k, v, s, *_ = (t.cuda() for t in _inputs(11, B, T, H, d, d))
    need = _lib.lib().fpb_workspace_bytes(ctypes.byref(_lib.dims(q, d, decays)))
    assert need > 0
    ref, _ = orc.retention_chunkwise(*(t.double().cpu() for t in (q, k, v, s)), [float(torch.tensor(g, dtype=torch.float32)) for g in decays], 64)
    for nbytes in (need, need // 3, B * H * d * d * 8, 1024, 0):
        guard = torch.full((nbytes + 256,), 171, dtype=torch.uint8, device="cuda")
        o, s_out = torch.empty_like(v), torch.empty_like(s)
        dm = _lib.dims(q, d, decays)
        if nbytes:
            dm.workspace, dm.workspace_bytes = guard.data_ptr(), nbytes
        _lib.check(_lib.lib().fpb_retention_fwd(dm, _lib.seq(q), _lib.seq(k), _lib.seq(v), _lib.state(s), _lib.seq(o), _lib.state(s_out),
                                                _lib.stream_ptr(q.device)))
        assert _rel(o, ref) < REL and bool((guard[nbytes:] == 171).all())
        o2 = torch.empty_like(v)
        _lib.check(_lib.lib().fpb_retention_fwd_static(_lib.dims(q, d, decays), _lib.seq(q), _lib.seq(k), _lib.seq(v), _lib.state(s),
                                                       _lib.seq(o2), _lib.state(None), _lib.stream_ptr(q.device)))
        assert _rel(o2, ref) < REL


@pytest.mark.parametrize("T,dk,dv", [(70, 32, 64), (70, 36, 20), (33, 128, 100), (300, 20, 128)])
def test_padding_meets_no_infinity(T, dk, dv):
    """Everything positive and one infinity: every sum is finite or +inf, with no 0 x inf unless padding is multiplied.
    The token walk (which unaligned tensors take) pads nothing and says which elements are which."""
    import flash_pop_b200 as fp
    B, H = 1, 2
    decays = orc.head_decays(H, (5, 12))
    q, k, v, s, dO, dS = (t.abs().cuda() + 0.01 for t in _inputs(13, B, T, H, dk, dv))

    def unaligned(t):
        return torch.empty(t.numel() + 1, device="cuda")[1:].view(t.shape).copy_(t)

    def run(form):
        x = [form(t).requires_grad_(True) for t in (q2, k2, v2, s)]
        o, s_out = fp.fused_chunk_retention(*x, decays)
        return [o, s_out, *torch.autograd.grad((o, s_out), x, (form(dO), dS))]

    for token in (T - 1, T - 3, T // 2):
        for which in range(3):
            q2, k2, v2 = (t.clone() for t in (q, k, v))
            (q2, k2, v2)[which][0, token, 1, 3] = float("inf")
            for a, b in zip(run(lambda t: t.clone()), run(unaligned)):
                assert not torch.isnan(b).any() and torch.equal(torch.isinf(a), torch.isinf(b)) and not torch.isnan(a).any()
