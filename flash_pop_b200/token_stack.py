"""One token through a stack of pre-norm decoder layers in one cooperative launch (``fpb_decoder_token``): what
``RetNetDecoder.forward_recurrent`` (flash_pop/retnet.py:535-546) runs when every layer is the plain one and nothing is
watching - no gradient, no hook on a sub-module, no replaced sub-module, no autocast or dispatch mode, bf16 weights and
activations, at most 64 rows.  Everything else takes the layer-by-layer path.  Nothing is remembered between calls: the
parameters' addresses and the conditions are read anew for every token."""
from __future__ import annotations

import ctypes
from typing import Optional

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch import Tensor

from flash_pop_b200 import _lib
from flash_pop_b200.layer_ops import observed, plain_linear
from flash_pop_b200.recurrent_state import RecurrentState
from flash_pop_b200.xpos_emb import XPos

MAX_ROWS = 64
_BF, _F32 = torch.bfloat16, torch.float32
_ACTS = {F.silu: _lib.ACT_SWISH, F.gelu: _lib.ACT_GELU, F.relu: _lib.ACT_RELU}


# `kept` holds every tensor whose address goes into the launch until it is made: between the two another thread may replace
# a parameter or grow a table, and what it lets go would be handed out again.
def _linear(m, n_out, n_in, device, out: list, kept: list) -> bool:
    if not plain_linear(m):
        return False
    p = m.__dict__["_parameters"]
    address = _lib.native().address           # of a parameter that the kernels can read in place, or None
    weight = p.get("weight")
    w = address(weight, _BF, 16, device, n_out, n_in)
    if w is None:
        return False
    bias = p.get("bias", p)                   # (a parametrised or deleted bias is not in the table at all)
    if bias is p:
        return False
    b = 0 if bias is None else address(bias, _BF, 4, device, n_out, 0)
    if b is None:
        return False
    out += (w, b)
    kept += (weight, bias)
    return True


def _norm(m, width, device, out: list, kept: list) -> bool:
    if type(m) is not nn.LayerNorm or m.normalized_shape != (width,) or "forward" in m.__dict__:
        return False
    d = m.__dict__["_parameters"]
    for name in ("weight", "bias"):
        t = d.get(name, m)
        if t is m:
            return False
        at = 0 if t is None else _lib.native().address(t, _F32, 16, device, width, 0)
        if at is None:
            return False
        out.append(at)
        kept.append(t)
    return True


def _layer(layer, first, shape, x_device, index, layer_cls, retention_cls, kept: list):
    """(pointers, phasor address, tail of the layer's record) of a layer the kernels can run as it stands, else None."""
    H, dk, dv, ffn = shape
    width, device = H * dv, x_device.index
    cls, own = type(layer), layer.__dict__
    mods = own["_modules"]
    ret = mods["retention"]
    if (cls.forward_recurrent is not layer_cls.forward_recurrent or cls._residual_blocks is not layer_cls._residual_blocks
            or cls._feedforward_block is not layer_cls._feedforward_block or not own["norm_first"] or own["config"].dtype != _BF
            or not own.keys().isdisjoint(("forward_recurrent", "_residual_blocks", "_feedforward_block"))):
        return None
    rcls, rown = type(ret), ret.__dict__
    if (not issubclass(rcls, retention_cls) or rcls.forward_recurrent is not retention_cls.forward_recurrent
            or rcls._gate_and_project is not retention_cls._gate_and_project
            or not rown.keys().isdisjoint(("forward_recurrent", "_gate_and_project"))):
        return None
    drop = mods["dropout"]
    dd = drop.__dict__
    if type(drop) is not nn.Dropout or dd["_forward_hooks"] or dd["_forward_pre_hooks"] or (drop.p > 0 and drop.training):
        return None
    if (ret.dropout > 0 and ret.training) or (ret.num_heads, ret.head_dim_qk, ret.head_dim_v) != (H, dk, dv) or ret.head_decays != first.head_decays:
        return None
    decays_t = rown["_buffers"].get("head_decays_torch")
    act_gate, act_ffn = _ACTS.get(ret.activation), _ACTS.get(layer.activation)
    if decays_t is None or decays_t.dtype != _F32 or act_gate is None or act_ffn is None:
        return None
    rm = rown["_modules"]
    ptrs: list = []
    n1, n2 = mods["norm1"], mods["norm2"]
    if not (_norm(n1, width, device, ptrs, kept) and _norm(n2, width, device, ptrs, kept)
            and _linear(rm["q_proj"], H * dk, width, device, ptrs, kept) and _linear(rm["k_proj"], H * dk, width, device, ptrs, kept)
            and _linear(rm["v_proj"], width, width, device, ptrs, kept) and _linear(rm["g_proj"], width, width, device, ptrs, kept)
            and _linear(rm["out_proj"], width, width, device, ptrs, kept) and _linear(mods["linear1"], ffn, width, device, ptrs, kept)
            and _linear(mods["linear2"], width, ffn, device, ptrs, kept)):
        return None
    if ret.relative_position:
        xpos = ret.xpos_embedder
        if type(xpos) is not XPos or xpos.head_dim != dk:
            return None
        xpos._move(x_device)
        row = xpos._rotation(1, index)
        ptrs.append(row.data_ptr())
        kept.append(row)
    else:
        ptrs.append(0)
    return ptrs, (act_gate, act_ffn, n1.eps, n2.eps, rm["group_norm"].eps)


def decoder_token(net, x: Tensor, recurrent_state: Optional[RecurrentState], layer_cls, retention_cls):
    """``net.forward_recurrent(x, recurrent_state)`` through the fused launch, or None when the call is not one of theirs."""
    if torch.is_grad_enabled() or observed() or type(x) is not Tensor or not x.is_cuda or x.dtype != _BF or x.dim() != 2 or not x.is_contiguous():
        return None
    B, device = x.shape[0], x.device
    layers = list(net.layers)
    if not 0 < B <= MAX_ROWS or not layers or x.data_ptr() % 16 or not all(issubclass(type(l), layer_cls) for l in layers):
        return None
    first = layers[0].retention
    if not isinstance(first, retention_cls) or type(layers[0].linear1) is not nn.Linear:
        return None
    H, dk, dv, ffn = first.num_heads, first.head_dim_qk, first.head_dim_v, layers[0].linear1.out_features
    if x.shape[1] != H * dv:
        return None
    n = len(layers)
    rs = net._validate_and_init_state(recurrent_state)
    index, states = rs.index, rs.state
    if type(index) is not int or index < 0:
        return None
    # the carried states: one (layers, B, H, dk, dv) tensor or a list of (B, H, dk, dv), or none yet
    if isinstance(states, Tensor):
        if type(states) is not Tensor or states.dim() != 5:
            return None
        base, step = states.data_ptr(), states.stride(0) * states.element_size()
        prev = states[0]
        addresses = [base + i * step for i in range(n)]
    else:
        states = list(states)
        if any(s is None for s in states):
            if any(s is not None for s in states):
                return None
            prev, addresses = None, [0] * n
        else:
            prev = states[0]
            if any(type(s) is not Tensor or s.dtype != prev.dtype or s.stride() != prev.stride() or s.shape != prev.shape
                   or s.device != device for s in states):
                return None
            addresses = [s.data_ptr() for s in states]
    sb = sh = 0
    if prev is not None:
        if (prev.shape != (B, H, dk, dv) or prev.dtype not in (_BF, _F32) or prev.device != device or prev.stride(3) != 1
                or prev.stride(2) != dv):
            return None
        sb, sh = prev.stride(0), prev.stride(1)
        align = 4 * prev.element_size()
        if sb % 4 or sh % 4 or (B > 1 and sb < dk * dv) or (H > 1 and sh < dk * dv) or any(a % align for a in addresses):
            return None
    # as the step operator types it: fp32 decays promote a carried state to fp32, a first state has the activations' type
    out_dtype = _BF if prev is None else _F32
    d = _lib._TokenDims(n, B, H, dk, dv, ffn, _lib.FPB_F32 if prev is not None and prev.dtype == _F32 else _lib.FPB_BF16,
                        _lib.FPB_F32 if out_dtype == _F32 else _lib.FPB_BF16, None, None, 0)
    need = _lib.lib().fpb_decoder_token_workspace(ctypes.byref(d))
    if need <= 0:
        return None
    record, size = _lib.DECODER_LAYER, _lib.DECODER_LAYER.size
    table = bytearray(n * size)
    out = torch.empty((n, B, H, dk, dv), device=device, dtype=out_dtype)
    out_base, out_step = out.data_ptr(), out.stride(0) * out.element_size()
    kept = [states]
    for i, layer in enumerate(layers):
        got = _layer(layer, first, (H, dk, dv, ffn), device, index, layer_cls, retention_cls, kept)
        if got is None:
            return None
        record.pack_into(table, i * size, *got[0], addresses[i], sb, sh, out_base + i * out_step, out.stride(1), out.stride(2), *got[1])
    y = torch.empty_like(x)
    with torch.cuda.device(device):
        scratch = torch.empty(need, dtype=torch.uint8, device=device)
        decays = (ctypes.c_double * H)(*first.head_decays)
        d.head_decays = ctypes.cast(decays, ctypes.POINTER(ctypes.c_double))
        d.workspace, d.workspace_bytes = scratch.data_ptr(), need
        records = (ctypes.c_char * len(table)).from_buffer(table)
        _lib.check(_lib.lib().fpb_decoder_token(ctypes.byref(d), records, x.data_ptr(), x.stride(0), y.data_ptr(), y.stride(0),
                                                _lib.stream_ptr(device)))
    return y, RecurrentState(out, index + 1)
