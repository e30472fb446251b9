"""The work that programs built on this package have it do, as cases to time.

A case is a dict of plain values.  `listed()` gives the fixed ones, `draw(rng)` more of the same ranges; `prepare` makes
what a program holds before the call, `run` makes one pass through the public entry points, `work` says what the pass
cannot do without, `tolerance` how far another correct implementation may be off, and `exact` the result in 64 bits.

Kinds of case:
  step     one recurrent decoding step of one layer              flash_pop_b200.retention_step
  token    one token through a whole decoder stack               RetNetDecoder.forward_recurrent
  op       the chunked retention operator                        fused_chunk_retention (forward, or forward + gradients)
  pop      the observation stream and the prediction suffixes    flash_pop_retention + pop_suffix_retention
  decoder  a stack of decoder layers, forward and gradients      RetNetDecoder
"""
import math

import torch

import flash_pop_b200 as fp
from flash_pop_b200.retnet import get_decays

CHUNK = 64                     # tokens per chunk: what the operation counts are stated for
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
SIZES = {"bf16": 2, "f32": 4}


def listed():
    return [
        # A single user's generation loop, one layer: nothing but latency.  fp32 state, as the decoder layers carry it.
        dict(name="step_one_row", kind="step", B=1, H=8, dk=128, dv=128, dtype="bf16", state="f32", in_place=False),
        # A serving batch: 256 rows, the state (67 MB, updated in place) is read and written once.
        dict(name="step_serving", kind="step", B=256, H=8, dk=128, dv=128, dtype="bf16", state="bf16", in_place=True),
        # A token through the 12-layer stack of the training configuration (d_model 1024), a small serving batch.
        dict(name="token_12_layers", kind="token", layers=12, B=16, H=8, d=128, ffn=4096, dtype="bf16"),
        # The fp32 operator with its gradients at the size of the smallest configuration: tests, notebooks, toy models.
        dict(name="op_small_f32", kind="op", train=True, B=2, H=4, T=256, dk=64, dv=64, dtype="f32", state=False),
        # A short ragged training batch of small heads that carries a state in and out, as truncated sequences do.
        dict(name="op_ragged_d64", kind="op", train=True, B=4, H=8, T=777, dk=64, dv=64, dtype="bf16", state=True),
        # A prompt of odd length appended to an existing context, one row: few sequences, so most of the GPU would idle.
        dict(name="prefill_ragged", kind="op", train=False, B=1, H=16, T=5003, dk=128, dv=128, dtype="bf16", state=True),
        # Forward over a full batch (scoring, or the forward half of training).
        dict(name="forward_full", kind="op", train=False, B=8, H=16, T=8192, dk=128, dv=128, dtype="bf16", state=False),
        # The training step of the operator at the benchmark's headline size.
        dict(name="train_full", kind="op", train=True, B=8, H=16, T=8192, dk=128, dv=128, dtype="bf16", state=False),
        # Values twice as wide as the keys (the usual RetNet ratio), long sequences: the largest case.
        dict(name="train_wide_values", kind="op", train=True, B=4, H=32, T=16384, dk=128, dv=256, dtype="bf16", state=False),
        # World-model training: 64 blocks of 80 observation tokens with 80 prediction tokens each, all gradients.
        dict(name="pop_train", kind="pop", train=True, B=16, H=8, d=64, blocks=64, block=80, tail=0, suffixes=64, P=80, state=False),
        # World-model rollout: a few rows, odd block size, a ragged tail, suffixes from the carried state; forward only.
        dict(name="pop_rollout", kind="pop", train=False, B=4, H=4, d=64, blocks=12, block=40, tail=7, suffixes=13, P=15, state=True),
        # Two layers of the training stack with all their gradients: projections, norms, rotation, gate around the operator.
        dict(name="decoder_train", kind="decoder", layers=2, B=4, T=2048, H=8, d=128, ffn=4096, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    """An integer of [lo, hi], evenly spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "op", "op", "op", "op", "f32", "pop", "pop", "token", "decoder"])
    if kind == "step":
        dk, dv = rng.choice([(64, 64), (64, 128), (128, 128), (128, 256)])
        return dict(kind="step", B=_log(rng, 1, 384), H=rng.choice([4, 8, 12, 16]), dk=dk, dv=dv, dtype="bf16",
                    state=rng.choice(["bf16", "f32"]), in_place=rng.random() < 0.5)
    if kind == "token":
        return dict(kind="token", layers=rng.randint(2, 12), B=_log(rng, 1, 64), H=rng.choice([4, 8]), d=rng.choice([64, 128]),
                    ffn=rng.choice([1024, 2048, 4096]), dtype="bf16")
    if kind == "f32":
        dk, dv = rng.choice([(32, 32), (64, 64), (64, 128), (128, 128)])
        return dict(kind="op", train=rng.random() < 0.7, B=rng.randint(1, 4), H=rng.randint(1, 8), T=_log(rng, 32, 1024), dk=dk, dv=dv,
                    dtype="f32", state=rng.random() < 0.5)
    if kind == "pop":
        d, block = 64, _log(rng, 8, 160)
        B, H, P = _log(rng, 1, 16), rng.choice([4, 8]), _log(rng, 4, 100)
        blocks = max(2, min(96, _log(rng, 256, 6000) // block))
        return dict(kind="pop", train=rng.random() < 0.6, B=B, H=H, d=d, blocks=blocks, block=block, tail=rng.choice([0, rng.randrange(block)]),
                    suffixes=blocks + rng.choice([0, 1]), P=P, state=rng.random() < 0.5)
    if kind == "decoder":
        return dict(kind="decoder", layers=rng.randint(1, 2), B=rng.randint(1, 4), T=_log(rng, 200, 2048), H=rng.choice([4, 8]),
                    d=rng.choice([64, 128]), ffn=rng.choice([1024, 2048, 4096]), dtype="bf16")
    dk, dv = rng.choice([(64, 64), (64, 128), (128, 128), (128, 128), (128, 256)])
    H = rng.choice([3, 4, 8, 12, 16, 32])
    T = _log(rng, 100, 16384)
    most = max(1, min(32, (1 << 28) // (T * H * max(dk, dv))))
    return dict(kind="op", train=rng.random() < 0.6, B=_log(rng, 1, most), H=H, T=T, dk=dk, dv=dv, dtype="bf16", state=rng.random() < 0.5)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=gen, device="cuda") * scale).to(dtype)

    c, kind = case, case["kind"]
    st = dict(case=case, decays=tuple(get_decays(c["H"], (5, 12)).tolist()))
    if kind == "step":
        B, H, dk, dv = c["B"], c["H"], c["dk"], c["dv"]
        st.update(q=normal(B, H, dk, scale=dk ** -0.5), k=normal(B, H, dk, scale=dk ** -0.5), v=normal(B, H, dv, scale=dk ** -0.5),
                  s=normal(B, H, dk, dv, scale=0.1, dtype=DTYPES[c["state"]]))
    elif kind == "op":
        B, H, T, dk, dv, dt = c["B"], c["H"], c["T"], c["dk"], c["dv"], DTYPES[c["dtype"]]
        s = normal(B, H, dk, dv, scale=0.1, dtype=dt) if c["state"] else None
        st.update(q=normal(B, T, H, dk, scale=dk ** -0.5, dtype=dt), k=normal(B, T, H, dk, scale=dk ** -0.5, dtype=dt),
                  v=normal(B, T, H, dv, scale=dk ** -0.5, dtype=dt), s=s)
        if c["train"]:
            st["leaves"] = [t.requires_grad_(True) for t in (st["q"], st["k"], st["v"], s) if t is not None]
            st["do"] = normal(B, T, H, dv, dtype=dt)
            st["ds"] = normal(B, H, dk, dv, dtype=dt) if c["state"] else None
    elif kind == "pop":
        B, H, d, P = c["B"], c["H"], c["d"], c["P"]
        T = c["blocks"] * c["block"] + c["tail"]
        x = [normal(B, T, H, d, scale=d ** -0.5) for _ in range(3)]
        y = [normal(B, c["suffixes"], P, H, d, scale=d ** -0.5) for _ in range(3)]
        s = normal(B, H, d, d, scale=0.1) if c["state"] else None
        st.update(x=x, y=y, s=s)
        if c["train"]:
            st["leaves"] = [t.requires_grad_(True) for t in (*x, *y, s) if t is not None]
            st["do"], st["dso"] = normal(B, T, H, d), normal(B, c["suffixes"], P, H, d)
    else:
        torch.manual_seed(seed)
        dt, width = DTYPES[c["dtype"]], c["H"] * c["d"]
        cfg = fp.RetNetDecoderLayer.Config(num_heads=c["H"], head_dim_v=c["d"], head_dim_qk=c["d"], dim_feedforward=c["ffn"], dropout=0.0,
                                           device="cuda", dtype=dt)
        net = fp.RetNetDecoder(cfg, c["layers"])
        st["net"] = net
        if kind == "token":
            net.eval().requires_grad_(False)
            st["x"] = normal(c["B"], width, dtype=dt)
            state = normal(c["layers"], c["B"], c["H"], c["d"], c["d"], scale=0.1, dtype=torch.float32)
            st["rs"] = fp.RecurrentState(state, 100)
        else:
            st["x"] = normal(c["B"], c["T"], width, dtype=dt).requires_grad_(True)
            st["dy"] = normal(c["B"], c["T"], width, dtype=dt)
            st["leaves"] = [st["x"], *net.parameters()]
    return st


def run(state):
    st, c = state, state["case"]
    kind = c["kind"]
    if kind == "step":
        return fp.retention_step(st["q"], st["k"], st["v"], st["decays"], st["s"], in_place=c["in_place"])
    if kind == "op":
        if not c["train"]:
            with torch.no_grad():
                return fp.fused_chunk_retention(st["q"], st["k"], st["v"], st["s"], st["decays"])
        o, s_out = fp.fused_chunk_retention(st["q"], st["k"], st["v"], st["s"], st["decays"])
        if st["ds"] is None:
            grads = torch.autograd.grad(o, st["leaves"], st["do"])
        else:
            grads = torch.autograd.grad((o, s_out), st["leaves"], (st["do"], st["ds"]))
        return [o.detach(), s_out.detach(), *grads]
    if kind == "pop":
        with torch.set_grad_enabled(c["train"]):
            o, blocks = fp.flash_pop_retention(*st["x"], st["s"], st["decays"], c["block"])
            so = fp.pop_suffix_retention(*st["y"], st["s"], blocks, st["decays"])
        if not c["train"]:
            return o, blocks, so
        grads = torch.autograd.grad((o, so), st["leaves"], (st["do"], st["dso"]))
        return [o.detach(), blocks.detach(), so.detach(), *grads]
    if kind == "token":
        with torch.no_grad():
            y, rs = st["net"].forward_recurrent(st["x"], st["rs"])
        return y, rs.state
    y, rs = st["net"](st["x"])
    return [y.detach(), rs.state.detach(), *torch.autograd.grad(y, st["leaves"], st["dy"])]


def _retention_flops(dk, dv, train):
    """Per (token, head), the causal half of a chunk's own tile: forward, and with `train` the gradients too."""
    half = (CHUNK + 1) / 2
    fwd = 2 * half * (dk + dv) + 4 * dk * dv
    return fwd + (2 * half * (3 * dk + 2 * dv) + 8 * dk * dv if train else 0)


def work(case):
    c, kind = case, case["kind"]
    if kind == "step":
        B, H, dk, dv = c["B"], c["H"], c["dk"], c["dv"]
        return {"bytes": B * H * (2 * dk * dv * SIZES[c["state"]] + (2 * dk + 2 * dv) * SIZES[c["dtype"]]), "flops": B * H * 5 * dk * dv}
    if kind == "op":
        e, n, dk, dv = SIZES[c["dtype"]], c["B"] * c["H"], c["dk"], c["dv"]
        moved = n * c["T"] * (2 * dk + 2 * dv) * (2 if c["train"] else 1)          # q, k, v, o; and dO, dQ, dK, dV
        states = n * dk * dv * (1 + (1 if c["state"] else 0)) + (n * dk * dv * 2 if c["train"] and c["state"] else 0)
        return {"bytes": e * (moved + states), "flops": n * c["T"] * _retention_flops(dk, dv, c["train"])}
    if kind == "pop":
        n, d = c["B"] * c["H"], c["d"]
        tokens = c["blocks"] * c["block"] + c["tail"] + c["suffixes"] * c["P"]
        moved = n * tokens * 4 * d * (2 if c["train"] else 1)
        states = n * d * d * c["blocks"] + (n * d * d * (2 if c["train"] else 1) if c["state"] else 0)
        return {"bytes": 2 * (moved + states), "flops": n * tokens * _retention_flops(d, d, c["train"])}
    width, e = c["H"] * c["d"], SIZES[c["dtype"]]
    weights = c["layers"] * (5 * width * width + 2 * width * c["ffn"])
    if kind == "token":
        states = c["layers"] * c["B"] * c["H"] * c["d"] * c["d"]
        return {"bytes": e * (weights + 2 * c["B"] * width) + 2 * 4 * states, "flops": 2 * c["B"] * weights + 5 * states}
    tokens = c["B"] * c["T"]
    return {"bytes": e * (2 * weights + 4 * tokens * width),
            "flops": 6 * tokens * weights + c["layers"] * tokens * c["H"] * _retention_flops(c["d"], c["d"], True)}


def tolerance(case):
    """Up to four times what these cases differ by from the result in 64 bits (the step 1.7e-3, the fp32 operator 3e-7,
    more for other orders of its sums; the bf16 operators 2.9e-3; a training stack of two layers 1.1e-2, a token's
    twelve 1.8e-2), and from the same path with its retention or its weights in fp32."""
    if case["kind"] == "step":
        return {"rel": 6e-3, "max": 1.6e-2}
    if case["kind"] == "op" and case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 1e-4}
    if case["kind"] in ("op", "pop"):
        return {"rel": 1e-2, "max": 0.12}
    if case["kind"] == "token":
        return {"rel": 5e-2, "max": 0.8}
    return {"rel": 3e-2, "max": 0.5}


# ---- the same passes in 64 bits, in plain torch ---------------------------------------------------------------------

def _gammas(case, device):
    """Head decays as the operators round them: to 32 bits before any power is taken."""
    return torch.tensor(get_decays(case["H"], (5, 12)), device=device).float().double()


def _retention64(q, k, v, s, gamma, block=0):
    """Retention of (B, T, H, d) doubles in chunks; returns the outputs, the last state and the states after full blocks."""
    B, T, H, dk = q.shape
    state = s if s is not None else q.new_zeros(B, H, dk, v.shape[-1])
    outs, blocks, a = [], [], 0
    lg = gamma.log()
    k = k * dk ** -0.5
    while a < T:
        e = min(a + 128, T)
        if block:
            e = min(e, (a // block + 1) * block)
        n = e - a
        i = torch.arange(n, device=q.device, dtype=q.dtype)
        gap = i[:, None] - i[None, :]
        mask = torch.where(gap >= 0, (gap.clamp(min=0)[None] * lg[:, None, None]).exp(), 0.0)
        qc, kc, vc = (t[:, a:e].transpose(1, 2) for t in (q, k, v))
        row = ((i + 1)[None, :, None] * lg[:, None, None]).exp()
        col = ((n - 1 - i)[None, :, None] * lg[:, None, None]).exp()
        outs.append((((qc @ kc.transpose(2, 3)) * mask) @ vc + (qc * row) @ state).transpose(1, 2))
        state = state * (n * lg).exp()[:, None, None] + (kc * col).transpose(2, 3) @ vc
        if block and e % block == 0:
            blocks.append(state)
        a = e
    return torch.cat(outs, 1), state, blocks


def _rotate64(x, start):
    """Rotate the channel pairs of (B, T, H, d) at positions start, start + 1, ..."""
    half = x.shape[-1] // 2
    theta = 10000.0 ** -torch.linspace(0, 1, half, device=x.device, dtype=torch.float64)
    angle = torch.arange(start, start + x.shape[1], device=x.device, dtype=torch.float64)[:, None] * theta
    c, sn = angle.cos()[:, None, :], angle.sin()[:, None, :]
    a, b = x[..., 0::2], x[..., 1::2]
    return torch.stack((a * c - b * sn, a * sn + b * c), -1).flatten(-2)


def _stack64(case, net, params, x, states, start):
    """The decoder stack on (B, T, width) doubles; `params` maps the names of the parameters to doubles."""
    F = torch.nn.functional
    H, width = case["H"], x.shape[-1]
    gamma = torch.tensor(net.layers[0].retention.head_decays, device=x.device).float().double()
    last = []
    for n in range(case["layers"]):
        p = {k[len("layers.%d." % n):]: t for k, t in params.items() if k.startswith("layers.%d." % n)}
        lin = lambda name, t: F.linear(t, p[name + ".weight"], p[name + ".bias"])
        h = F.layer_norm(x, (width,), p["norm1.weight"], p["norm1.bias"], 1e-6)
        q, k, v = (lin("retention.%s_proj" % w, h).unflatten(-1, (H, -1)) for w in "qkv")
        o, s, _ = _retention64(_rotate64(q, start), _rotate64(k, start), v, None if states is None else states[n], gamma)
        last.append(s)
        o = F.layer_norm(o, o.shape[-1:], None, None, 1e-6).flatten(-2)
        x = x + lin("retention.out_proj", o * F.silu(lin("retention.g_proj", h)))
        h = F.layer_norm(x, (width,), p["norm2.weight"], p["norm2.bias"], 1e-6)
        x = x + lin("linear2", F.silu(lin("linear1", h)))
    return x, torch.stack(last)


def exact(case, seed):
    """What `run` returns for these inputs, computed in 64 bits."""
    c, st = case, prepare(case, seed)
    wide = lambda t: None if t is None else t.detach().double()
    if c["kind"] == "step":
        gamma, k = _gammas(c, "cuda"), wide(st["k"]) * c["dk"] ** -0.5
        s = wide(st["s"]) * gamma[:, None, None] + k.unsqueeze(-1) * wide(st["v"]).unsqueeze(-2)
        return (wide(st["q"]).unsqueeze(-2) @ s).squeeze(-2), s
    if c["kind"] == "token":
        with torch.no_grad():
            params = {k: p.double() for k, p in st["net"].named_parameters()}
            y, s = _stack64(c, st["net"], params, wide(st["x"]).unsqueeze(1), wide(st["rs"].state), st["rs"].index)
        return y.squeeze(1), s
    if c["kind"] == "decoder":
        x = wide(st["x"]).requires_grad_(True)
        params = {k: p.detach().double().requires_grad_(True) for k, p in st["net"].named_parameters()}
        y, s = _stack64(c, st["net"], params, x, None, 0)
        return [y.detach(), s.detach(), *torch.autograd.grad(y, [x, *params.values()], wide(st["dy"]))]
    train, gamma = c["train"], _gammas(c, "cuda")
    leaf = lambda t: None if t is None else wide(t).requires_grad_(train)
    if c["kind"] == "op":
        q, k, v, s = (leaf(st[n]) for n in ("q", "k", "v", "s"))
        o, s_out, _ = _retention64(q, k, v, s, gamma)
        if not train:
            return o, s_out
        ends, weights = ([o], [wide(st["do"])]) if st["ds"] is None else ([o, s_out], [wide(st["do"]), wide(st["ds"])])
        return [o.detach(), s_out.detach(), *torch.autograd.grad(ends, [t for t in (q, k, v, s) if t is not None], weights)]
    x, y, s = [leaf(t) for t in st["x"]], [leaf(t) for t in st["y"]], leaf(st["s"])
    o, _, blocks = _retention64(*x, s, gamma, c["block"])
    first = s if s is not None else torch.zeros_like(blocks[0])
    starts = torch.stack([first, *blocks][:c["suffixes"]], 1)
    so = _retention64(*(t.flatten(0, 1) for t in y), starts.flatten(0, 1), gamma)[0].unflatten(0, (c["B"], c["suffixes"]))
    blocks = torch.stack(blocks, 1)
    if not train:
        return o, blocks, so
    grads = torch.autograd.grad((o, so), [t for t in (*x, *y, s) if t is not None], (wide(st["do"]), wide(st["dso"])))
    return [o.detach(), blocks.detach(), so.detach(), *grads]
