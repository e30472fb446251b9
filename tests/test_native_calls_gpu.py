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


class _Recorder:
    """The extension, with a note of which of its functions took the call they were given."""

    def __init__(self, native):
        self.native, self.taken = native, {}

    def __getattr__(self, name):
        def call(*args):
            got = getattr(self.native, name)(*args)
            self.taken.setdefault(name, []).append(got is not None)
            return got
        return call


@contextlib.contextmanager
def recorded():
    from flash_pop_b200 import _lib
    kept = _lib.native
    recorder = _Recorder(kept())
    _lib.native = lambda: recorder
    try:
        yield recorder.taken
    finally:
        _lib.native = kept


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


@pytest.mark.parametrize("layout", ["plain", "packed", "turned", "odd", "expanded", "inner"])
@pytest.mark.parametrize("dtype,state", [(BF, BF), (BF, F32), (BF, None), (F32, F32), (F32, None)])
def test_the_extension_takes_the_ordinary_call(layout, dtype, state):
    """Which calls go through the extension at all: layouts that the kernels read in place do, others do not."""
    import flash_pop_b200 as fp
    from flash_pop_b200 import layer_ops
    B, T, H, d = 2, 24, 3, 64
    decays = tuple(orc.head_decays(H, (5, 12)))
    pick = lambda: _layouts(torch.randn(B, T, H, d, device="cuda").to(dtype))[layout].detach().requires_grad_(True)
    s = None if state is None else torch.randn(B, H, d, d, device="cuda").to(state)
    x, dy = [pick() for _ in range(3)], pick().detach()
    in_place = layout not in ("expanded", "inner")
    with recorded() as taken:
        o, _ = fp.fused_chunk_retention(*x, s, decays)
        torch.autograd.grad(o, x, dy)
        _, blocks = fp.flash_pop_retention(*x, s, decays, 8)
        y = [t.detach().unsqueeze(1).requires_grad_(True) for t in x]
        so = fp.pop_suffix_retention(*y, s, blocks.detach(), decays)
        torch.autograd.grad(so, y, dy.unsqueeze(1))
        fp.retention_step(*(t.detach()[:, 0] for t in x), decays, s)
    assert taken == {"forward": [in_place] * 2, "backward": [in_place], "suffix_forward": [in_place], "suffix_backward": [in_place],
                     "step": [in_place]}
    if layout == "odd":                # (the layer passes refuse what 16-byte accesses cannot read)
        return
    with recorded() as taken:
        torch.autograd.grad(layer_ops.rotary_qk(x[0], x[1], torch.randn(1, T, d // 2, 2, device="cuda")), x[:2], (dy, dy))
        torch.autograd.grad(layer_ops.groupnorm_gate(x[0], x[1], 1e-6), x[:2], dy)
        w = torch.randn(d, device="cuda")
        torch.autograd.grad(layer_ops.layer_norm(x[0], w, w, 1e-6), x[:1], dy)
    assert taken == {"rotary": [in_place] * 2, "gate_forward": [in_place], "gate_backward": [in_place], "norm_forward": [layout == "plain"],
                     "norm_backward": [layout == "plain"]}


def test_streams_and_threads():
    """The extension releases the interpreter lock around the C ABI: threads on streams of their own, and a side stream of
    the main thread, get what the main thread gets on its stream."""
    import threading
    import flash_pop_b200 as fp
    decays = tuple(orc.head_decays(4, (5, 12)))
    cases = []
    for B, T, d, dtype in ((2, 300, 64, BF), (1, 2000, 128, BF), (2, 100, 32, F32)):
        x = [(torch.randn(B, T, 4, d, device="cuda") * 0.1).to(dtype) for _ in range(4)]
        cases.append((x, torch.randn(B, 4, d, d, device="cuda").to(dtype)))

    def once(x, s):
        leaves = [t.detach().requires_grad_(True) for t in x[:3]]
        o, s_out = fp.fused_chunk_retention(*leaves, s, decays)
        p, blocks = fp.flash_pop_retention(*leaves, s, decays, 16)
        grads = torch.autograd.grad((o, p), leaves, (x[3], x[3]))
        return [o.detach(), s_out.detach(), p.detach(), blocks.detach(), *grads, *fp.retention_step(*(t[:, 0] for t in x[:3]), decays, s)]

    want = [once(*c) for c in cases]
    torch.cuda.synchronize()
    failures = []

    def work(case, stream):
        try:
            with torch.cuda.stream(stream):
                for _ in range(20):
                    got = once(*cases[case])
                    stream.synchronize()
                    assert all(torch.equal(a, b) for a, b in zip(got, want[case]))
        except BaseException as e:       # noqa: BLE001 - reported by the main thread
            failures.append(e)

    threads = [threading.Thread(target=work, args=(i % len(cases), torch.cuda.Stream())) for i in range(6)]
    for t in threads:
        t.start()
    work(0, torch.cuda.Stream())
    for t in threads:
        t.join(120)
    assert not failures, failures[0]
