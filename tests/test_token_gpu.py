"""One token through a decoder stack in one launch (fpb_decoder_token) against the same stack in 64 bits and against
the layer-by-layer path, over the edges of its ranges; and the calls that must keep taking the layer-by-layer path."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
BF, F32 = torch.bfloat16, torch.float32


def _net(layers, H, dk, dv, ffn, seed=0, act="swish", **kw):
    import flash_pop_b200 as fp
    torch.manual_seed(seed)
    cfg = fp.RetNetDecoderLayer.Config(num_heads=H, head_dim_v=dv, head_dim_qk=dk, dim_feedforward=ffn, dropout=0.0, device="cuda",
                                       dtype=BF, activation=act, head_decays_range=(5, 12), **kw)
    net = fp.RetNetDecoder(cfg, layers).eval().requires_grad_(False)
    for p in net.parameters():                       # biases and norm parameters away from their 0 and 1
        if p.dim() == 1:
            p.add_(torch.randn_like(p) * 0.1)
    return net


def _exact(net, x, states, index, act):
    x, out = x.double(), []
    fn = {"swish": F.silu, "gelu": F.gelu, "relu": F.relu}[act]
    for n, l in enumerate(net.layers):
        r = l.retention
        lin = lambda m, t: F.linear(t, m.weight.double(), m.bias.double())
        norm = lambda m, t: F.layer_norm(t, t.shape[-1:], m.weight.double(), m.bias.double(), m.eps)
        h = norm(l.norm1, x)
        q, k, v = (lin(m, h).unflatten(-1, (r.num_heads, -1)) for m in (r.q_proj, r.k_proj, r.v_proj))
        ph = r.xpos_embedder._rotation(1, index)[0, 0].to(torch.complex128)
        rot = lambda t: torch.view_as_real(torch.view_as_complex(t.unflatten(-1, (-1, 2)).contiguous()) * ph).flatten(-2)
        q, k = rot(q), rot(k) * r.head_dim_qk ** -0.5
        s = k.unsqueeze(-1) * v.unsqueeze(-2)
        if states is not None:
            s = s + states[n].double() * torch.tensor(r.head_decays, device=x.device).float().double().view(-1, 1, 1)
        out.append(s)
        o = F.layer_norm((q.unsqueeze(-2) @ s).squeeze(-2), (r.head_dim_v,), None, None, 1e-6).flatten(1)
        x = x + lin(r.out_proj, o * fn(lin(r.g_proj, h)))
        x = x + lin(l.linear2, fn(lin(l.linear1, norm(l.norm2, x))))
    return x, torch.stack(out)


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("layers,B,H,dk,dv,ffn,act,state", [
    (2, 1, 8, 128, 128, 4096, "swish", F32), (3, 16, 8, 128, 128, 4096, "swish", F32), (2, 17, 4, 64, 64, 1024, "gelu", BF),
    (1, 33, 8, 64, 64, 2048, "relu", None), (2, 64, 8, 128, 128, 1024, "swish", F32), (2, 32, 4, 64, 128, 96, "swish", F32),
    (2, 5, 3, 48, 32, 160, "gelu", BF), (1, 3, 1, 40, 32, 32, "relu", None), (1, 2, 4, 256, 256, 8192, "swish", F32),
    (17, 4, 2, 32, 32, 64, "gelu", F32), (33, 2, 4, 64, 64, 128, "swish", F32)])
def test_token_matches_the_stack_in_64_bits(layers, B, H, dk, dv, ffn, act, state):
    import flash_pop_b200 as fp
    from flash_pop_b200 import _lib
    net = _net(layers, H, dk, dv, ffn, act=act)
    g = torch.Generator(device="cuda").manual_seed(B)
    x = torch.randn(B, H * dv, generator=g, device="cuda").to(BF)
    s = None if state is None else (torch.randn(layers, B, H, dk, dv, generator=g, device="cuda") * 0.1).to(state)
    rs = None if s is None else fp.RecurrentState(s, 77)
    n0 = _lib.launch_count()
    with torch.no_grad():
        y, new = net.forward_recurrent(x, rs)
    assert _lib.launch_count() - n0 == (layers + 15) // 16
    _lib.device_status()
    with torch.enable_grad():                        # the layer-by-layer path (no parameter asks for a gradient)
        y1, new1 = net.forward_recurrent(x, rs)
    assert y.dtype == y1.dtype and new.state.dtype == new1.state.dtype and new.state.shape == new1.state.shape and new.index == new1.index
    ye, se = _exact(net, x, s, 0 if rs is None else 77, act)
    # no further from the exact result than the path it stands in for.  Both errors are independent samples of the same bf16
    # roundings: a tenth of slack.  In a deep stack they grow along a few directions (of 33 layers, some ten): the ratio of
    # two norms with ten degrees of freedom each stays below 1.7 nine times in ten, and the sizes here are fixed by the seed
    slack = 1.1 if layers < 8 else 1.7
    assert _rel(y, ye) <= slack * _rel(y1, ye) + 1e-4 and _rel(new.state, se) <= slack * _rel(new1.state, se) + 1e-4
    # about ten bf16 roundings of 2^-9 a layer.  (From a zero state o = (q . k) v: GroupNorm scales a head whose q . k is
    # close to zero up by orders of magnitude, rounding errors with it, so only the comparison above binds there.)
    assert state is None or _rel(y, ye) < 1e-2 * layers


def test_strided_states_lists_and_graphs():
    import flash_pop_b200 as fp
    net = _net(2, 4, 64, 64, 256)
    x = torch.randn(6, 256, device="cuda").to(BF)
    wide = torch.randn(2, 12, 4, 64, 64, device="cuda") * 0.1
    s = wide[:, ::2]
    with torch.no_grad():
        y, new = net.forward_recurrent(x, fp.RecurrentState(s, 3))
        y1, new1 = net.forward_recurrent(x, fp.RecurrentState(s.contiguous(), 3))
        y2, new2 = net.forward_recurrent(x, fp.RecurrentState([s[0], s[1]], 3))
        assert torch.equal(y, y1) and torch.equal(y, y2) and torch.equal(new.state, new1.state) and torch.equal(new.state, new2.state)
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        xin = x.clone()
        with torch.cuda.graph(graph, stream=side):
            yg, newg = net.forward_recurrent(xin, fp.RecurrentState(s, 3))
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(yg, y) and torch.equal(newg.state, new.state)
        xin.copy_(x.flip(0))
        graph.replay()
        assert torch.equal(yg, net.forward_recurrent(x.flip(0), fp.RecurrentState(s, 3))[0])


def test_calls_that_keep_the_layer_by_layer_path():
    import flash_pop_b200 as fp
    from flash_pop_b200.retnet import MultiScaleRetention, RetNetDecoderLayer
    from flash_pop_b200.token_stack import decoder_token
    x = torch.randn(2, 256, device="cuda").to(BF)
    taken = lambda net, x=x, rs=None: decoder_token(net, x, rs, RetNetDecoderLayer, MultiScaleRetention) is not None
    with torch.no_grad():
        net = _net(2, 4, 64, 64, 256)
        assert taken(net)
        seen = []
        handle = net.layers[1].linear1.register_forward_hook(lambda *a: seen.append(1))
        assert not taken(net)
        net.forward_recurrent(x)
        assert seen
        handle.remove()
        assert taken(net) and not taken(net, torch.randn(65, 256, device="cuda").to(BF)) and not taken(net, x.float())
        assert not taken(net, rs=fp.RecurrentState(None, torch.zeros(2, dtype=torch.long, device="cuda")))
        with torch.autocast("cuda", dtype=BF):
            assert not taken(net)
        net.layers[0].linear2 = torch.nn.Sequential(net.layers[0].linear2)
        assert not taken(net)
        assert not taken(_net(1, 4, 64, 64, 256, norm_first=False)) and not taken(_net(1, 4, 64, 64, 250))
        dropping = _net(1, 4, 64, 64, 256)
        dropping.layers[0].dropout.p = 0.5
        assert taken(dropping)
        dropping.train()
        assert not taken(dropping)
    assert not taken(_net(1, 4, 64, 64, 256))        # gradients on


def test_what_the_launch_reads_is_alive_until_it_is_made(monkeypatch):
    """Another thread may replace a parameter or grow the rotation table while the addresses are collected."""
    import weakref
    import flash_pop_b200 as fp
    from flash_pop_b200 import _lib
    net = _net(2, 4, 64, 64, 256)
    x = torch.randn(3, 256, device="cuda").to(BF)
    real, refs, alive = _lib.lib(), [], []
    xpos, q_proj = net.xpos_embedder, net.layers[0].retention.q_proj
    table_row = xpos._rotation

    def rotation(length, index):
        row = table_row(length, index).clone()                  # (as a table that is replaced at once)
        if refs:
            refs.append(weakref.ref(q_proj.weight))
            q_proj.weight = torch.nn.Parameter(q_proj.weight.clone(), requires_grad=False)
        refs.append(weakref.ref(row))
        return row

    class Lib:
        def __getattr__(self, name):
            return getattr(real, name)

        def fpb_decoder_token(self, *args):
            alive.extend(r() is not None for r in refs)
            return real.fpb_decoder_token(*args)

    with torch.no_grad():
        want, _ = net.forward_recurrent(x, fp.RecurrentState(None, 5))
        monkeypatch.setattr(xpos, "_rotation", rotation)
        monkeypatch.setattr(_lib, "lib", lambda handle=Lib(): handle)
        got, _ = net.forward_recurrent(x, fp.RecurrentState(None, 5))
    assert alive == [True] * 3 and torch.equal(got, want)


def test_an_overridden_walk_over_the_layers_is_taken():
    """A decoder class, or one decoder, that walks its layers in its own way does so for a token as for a chunk."""
    import flash_pop_b200 as fp
    net = _net(2, 4, 64, 64, 256)
    x = torch.randn(3, 256, device="cuda").to(BF)
    walked = []

    class Own(fp.RetNetDecoder):
        def _walk_layers(self, *args):
            walked.append(self)
            return super()._walk_layers(*args)

    with torch.no_grad():
        net.forward_recurrent(x)
        net.__class__ = Own
        net.forward_recurrent(x)
        assert len(walked) == 1
        net.__class__ = fp.RetNetDecoder
        plain = net._walk_layers
        net._walk_layers = lambda *args: walked.append(net) or plain(*args)
        net.forward_recurrent(x)
        assert len(walked) == 2
