"""The operators' native host side against the Python path it stands in for, over the forms of call both can get: layouts,
dtypes, missing states, partial gradients, sub-classes, errors.  Same kernels underneath, so results agree bit for bit."""
import contextlib

import pytest
import torch

from oracle import retention_oracle as orc

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


class _Declines:
    """Stands for the extension and leaves every call to the Python path."""

    def __getattr__(self, name):
        return lambda *a: None


@contextlib.contextmanager
def python_path():
    from flash_pop_b200 import _lib
    kept = _lib.native
    _lib.native = lambda: _Declines()
    try:
        yield
    finally:
        _lib.native = kept


def _layouts(t):
    """The same values as a contiguous tensor, a slice of a packed one, a transposed one and a row-expanded one."""
    packed = torch.cat((t, t + 1), -1)[..., :t.shape[-1]]
    turned = t.transpose(1, 2).contiguous().transpose(1, 2)
    odd = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)[1:].view(t.shape).copy_(t)
    return {"plain": t, "packed": packed, "turned": turned, "odd": odd, "expanded": t[:1].expand_as(t), "inner": t.transpose(-1, -2).contiguous().transpose(-1, -2)}


def _both(f):
    """f() on the native path and on the Python path: results, or the type and text of what was raised."""
    def attempt():
        try:
            return f()
        except Exception as e:       # noqa: BLE001 - whatever it is, both sides have to raise it
            return type(e), str(e)
    a = attempt()
    with python_path():
        b = attempt()
    assert type(a) is type(b) and len(a) == len(b)
    for x, y in zip(a, b):
        if isinstance(x, torch.Tensor):
            assert x.dtype == y.dtype and x.shape == y.shape and torch.equal(x, y), (x.shape, x.dtype)
        else:
            assert x == y
    return a


@pytest.mark.parametrize("layout", ["plain", "packed", "turned", "odd", "expanded", "inner"])
@pytest.mark.parametrize("dtype,state", [(BF, BF), (BF, F32), (BF, None), (F32, F32), (F32, None)])
def test_operator_forms(layout, dtype, state):
    import flash_pop_b200 as fp
    B, T, H, d = 2, 70, 3, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    decays = tuple(orc.head_decays(H, (5, 12)))
    q, k, v, dO = ((torch.randn(B, T, H, d, generator=g, device="cuda") * 0.1).to(dtype) for _ in range(4))
    s = None if state is None else (torch.randn(B, H, d, d, generator=g, device="cuda") * 0.1).to(state)
    pick = lambda t: _layouts(t)[layout].detach().requires_grad_(True)

    def plain():
        x = [pick(t) for t in (q, k, v)]
        o, s_out = fp.fused_chunk_retention(*x, s, decays)
        return [o, s_out, *torch.autograd.grad(o, x, _layouts(dO)[layout])]

    def pop():
        x = [pick(t) for t in (q, k, v)]
        s0 = None if s is None else s.clone().requires_grad_(True)
        o, blocks = fp.flash_pop_retention(*x, s0, decays, 16)
        y = [torch.stack([pick(t)[:, :20]] * 5, 1) for t in (q, k, v)]
        so = fp.pop_suffix_retention(*y, s0, blocks, decays)
        return [o, blocks, so, *torch.autograd.grad((o, so), x + ([] if s is None else [s0]), (_layouts(dO)[layout], so.detach()))]

    def step():
        prev = s
        return [*fp.retention_step(pick(q)[:, 3], pick(k)[:, 3], pick(v)[:, 3], decays, prev)]

    for f in (plain, pop, step):
        _both(f)
    if layout == "plain":
        for need in range(3):
            x = [t.detach().requires_grad_(i == need) for i, t in enumerate((q, k, v))]
            _both(lambda: torch.autograd.grad(fp.fused_chunk_retention(*x, s, decays)[0], [x[need]], dO))
        _both(lambda: torch.autograd.grad(fp.fused_chunk_retention(*[pick(t) for t in (q, k, v)], s, list(decays))[1].sum() * 0 + pick(q).sum(),
                                          [], allow_unused=True) or [torch.zeros(1)])


def test_refusals_are_the_same():
    import flash_pop_b200 as fp
    q = torch.randn(1, 8, 2, 32, device="cuda")
    r = lambda *a, **k: (lambda: [*fp.fused_chunk_retention(*a, **k)])
    for f in (r(q, q, q, None, (0.9,)), r(q, q, q.half(), None, (0.9, 0.9)), r(q.half(), q.half(), q.half(), None, (0.9, 0.9)),
              r(q, q[:, :4], q, None, (0.9, 0.9)), r(q, q, q, None, (0.9, 1.5)), r(q, q, q, None, (0.9, float("nan"))),
              r(q, q, q, torch.zeros(1, 2, 32, 16, device="cuda"), (0.9, 0.9)), r(q, q, q, torch.zeros(1, 2, 32, 32, device="cuda").bfloat16(), (0.9, 0.9)),
              r(q.cpu(), q.cpu(), q.cpu(), None, (0.9, 0.9)), r(q[:0], q[:0], q[:0], None, (0.9, 0.9)), r(q[:, :0], q[:, :0], q[:, :0], None, (0.9, 0.9)),
              lambda: [*fp.flash_pop_retention(q, q, q, None, (0.9, 0.9), 0)], lambda: [*fp.flash_pop_retention(q, q, q, None, (0.9, 0.9), 100)],
              lambda: [*fp.retention_step(q[:, 0], q[:, 0], q[:, 0], (0.9, 0.9), torch.zeros(1, 2, 32, 32, device="cuda"), state_dtype=torch.float16)]):
        _both(f)


def test_layer_passes():
    from flash_pop_b200 import layer_ops
    g = torch.Generator(device="cuda").manual_seed(4)
    for dtype in (BF, F32):
        o, z, dy = (torch.randn(2, 9, 3, 64, generator=g, device="cuda").to(dtype) for _ in range(3))
        w, b = torch.randn(64, generator=g, device="cuda"), torch.randn(64, generator=g, device="cuda")
        ph = torch.randn(1, 9, 32, 2, generator=g, device="cuda")
        for layout in ("plain", "packed", "turned", "odd", "expanded"):
            leaf = lambda t: _layouts(t)[layout].detach().requires_grad_(True)

            def rotary():
                x = [leaf(o), leaf(z)]
                a, c = layer_ops.rotary_qk(*x, ph)
                return [a, c, *torch.autograd.grad((a, c), x, (_layouts(dy)[layout], dy))]

            def gate():
                x = [leaf(o), leaf(z)]
                y = layer_ops.groupnorm_gate(*x, 1e-6)
                return [y, *torch.autograd.grad(y, x, _layouts(dy)[layout])]

            def norm():
                x = leaf(o)
                y = layer_ops.layer_norm(x, w, b, 1e-6)
                return [y, *torch.autograd.grad(y, [x], _layouts(dy)[layout])]

            for f in (rotary, gate, norm):
                _both(f)
