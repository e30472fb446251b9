"""Column sums (alone and behind the swish backward) and the grouped linear layers built on them: against 64 bits at the edges
of rows and columns, and against the plain modules."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("rows,n", [(1, 64), (31, 64), (32, 128), (257, 192), (2047, 1024), (2049, 320), (8192, 4096), (70000, 64)])
def test_column_sums(rows, n):
    from flash_pop_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(rows)
    dy, a = (torch.randn(rows, n, generator=g, device="cuda").to(BF) * s for s in (1, 3))
    sums, none = _lib.native().column_sums(dy, None)
    assert none is None
    # one bf16 rounding of the result (2^-9) over fp32 sums of up to 10^5 terms (2^-24 sqrt(rows), relative to the terms)
    scale = dy.double().pow(2).sum(0).sqrt()
    ref = dy.double().sum(0)
    assert bool(((sums.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5 * scale).all())
    sums, da = _lib.native().column_sums(dy, a)
    sg = torch.sigmoid(a.double())
    ref_da = dy.double() * sg * (1 + a.double() * (1 - sg))
    assert bool(((da.double() - ref_da).abs() <= 2 ** -8 * ref_da.abs() + 1e-6 * dy.double().abs()).all())
    scale, ref = ref_da.pow(2).sum(0).sqrt(), ref_da.sum(0)
    assert bool(((sums.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5 * scale).all())


def _net(width=256, ffn=320):
    import flash_pop_b200 as fp
    torch.manual_seed(0)
    return fp.RetNetDecoder(fp.RetNetDecoderLayer.Config(num_heads=4, head_dim_v=width // 4, dim_feedforward=ffn, dropout=0.0, device="cuda",
                                                         dtype=BF), 1)


def _grads(net, x, dy):
    x = x.clone().requires_grad_(True)
    y, _ = net(x)
    return [y.detach(), *torch.autograd.grad(y, [x, *net.parameters()], dy)]


def test_layer_gradients_match_the_plain_modules():
    net = _net()
    x, dy = (torch.randn(2, 130, 256, device="cuda").to(BF) for _ in range(2))
    fused = _grads(net, x, dy)
    handles = [m.register_forward_hook(lambda *a: None) for m in net.modules() if type(m) is torch.nn.Linear]      # a hook: plain modules
    plain = _grads(net, x, dy)
    for h in handles:
        h.remove()
    exact = _grads_in_float(net, x, dy)
    assert torch.equal(fused[0], plain[0])           # forward: the same products
    for i, (a, b, e) in enumerate(zip(fused[1:], plain[1:], exact[1:])):
        ra, rb = (float((t.double() - e.double()).norm() / e.double().norm()) for t in (a, b))
        assert ra <= 1.1 * rb + 1e-4, (i, ra, rb)    # no further from fp32 weights and sums than the modules' own backward


def _grads_in_float(net, x, dy):
    import copy
    wide = copy.deepcopy(net).float()
    for l in wide.layers:
        l.config = copy.copy(l.config)
        l.config.dtype = torch.float32
        l.retention.config = copy.copy(l.retention.config)
        l.retention.config.use_fused_version = True
    return _grads(wide, x.float(), dy.float())


def test_calls_that_keep_the_plain_modules_and_partial_or_second_gradients():
    from flash_pop_b200 import layer_ops
    from flash_pop_b200.layer_ops import SwishFeedForward, linear_group, linears_supported
    lin = [torch.nn.Linear(128, 64, device="cuda", dtype=BF) for _ in range(2)]
    x = torch.randn(3, 9, 128, device="cuda").to(BF)
    assert linears_supported(x, *lin)
    with torch.no_grad():
        assert not linears_supported(x, *lin)
    with torch.autocast("cuda", dtype=BF):
        assert not linears_supported(x, *lin)
    lin[1].weight.requires_grad_(False)
    assert not linears_supported(x, *lin)
    lin[1].weight.requires_grad_(True)
    assert not linears_supported(x.transpose(0, 1), *lin) and not linears_supported(x, torch.nn.Linear(128, 60, device="cuda", dtype=BF))
    xg = x.clone().requires_grad_(True)
    a, b = linear_group(xg, *lin)
    (gx,) = torch.autograd.grad(b.float().sum(), [xg], retain_graph=True)          # one output only
    assert torch.allclose(gx.float(), lin[1].weight.float().sum(0).expand_as(gx), rtol=1e-2, atol=1e-2)
    # second gradients go through the framework's operations
    w1, w2 = (torch.randn(*s, device="cuda").to(BF).mul_(0.1).requires_grad_(True) for s in ((64, 128), (128, 64)))
    b1, b2 = (torch.randn(n, device="cuda").to(BF).requires_grad_(True) for n in (64, 128))
    results = []
    for f in (SwishFeedForward.apply, lambda x, w1, b1, w2, b2: F.linear(F.silu(F.linear(x, w1, b1)), w2, b2)):
        xi = x.clone().requires_grad_(True)
        (g,) = torch.autograd.grad(f(xi, w1, b1, w2, b2).float().pow(2).sum(), [xi], create_graph=True)
        results.append(torch.autograd.grad(g.float().pow(2).sum(), [xi, w1, b1, w2, b2]))
    for p, q in zip(*results):
        assert float((p.double() - q.double()).norm() / q.double().norm()) < 2e-2      # bf16, two orders
    assert layer_ops.observed() is False
