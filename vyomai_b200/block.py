"""Whole sublayers of a transformer layer as one call into the library (vy_attn_block_*, vy_ffn_block_*).

The functions here take over from functional.py / autograd_train.py where a sublayer's tensors are what those calls take: one dtype, contiguous, on the device,
no dropout, head_dim 64, tilings settled. Everything else, and a sublayer's first call of each shape (whose products time their tilings), goes the
general way, launch by launch. Nothing is kept from a call but the tilings, by the values that they depend on; addresses are read anew each time.

Where the one call applies, both ways save the same for the backward pass: the input and one buffer as the library lays it out (`pack`, `attention_saved`, `ffn_saved`).
So either direction goes its own way, and a forward pass that is computed again (torch.utils.checkpoint) saves what the first one did, whatever has been settled in between.
With the same tilings the two ways give the same results to the bit; tilings are chosen by timing, and another split of a weight gradient's sum rounds otherwise.
"""
from __future__ import annotations

import math
from ctypes import byref
from typing import Optional

import torch

from . import _lib, gemm_tune, ops
from .functional import pack_linears

C = _lib.CONSTS
_ATTN, _FFN = _lib.STRUCTS["VyAttnBlock"], _lib.STRUCTS["VyFfnBlock"]
_DT = {torch.float32: C["VY_F32"], torch.bfloat16: C["VY_BF16"]}
_ACT = {"gelu": (C["VY_ACT_GELU_ERF"], C["VY_ACT_DGELU_ERF"])}


def _plain(T: torch.dtype, *ts: Optional[torch.Tensor]) -> bool:
    for t in ts:
        if t is not None and (t.dtype is not T or not t.is_cuda or not t.is_contiguous()):
            return False
    return True


def _stacked(ts) -> bool:
    """Do the tensors' rows follow one another in memory?"""
    at = ts[0].data_ptr()
    for t in ts:
        if t.data_ptr() != at:
            return False
        at += t.numel() * t.element_size()
    return True


def _direct(ps) -> bool:   # a trainer's own gradient buffers (autograd_train.py): the general way writes those
    return any(getattr(p, "_vy_direct_grad", False) or getattr(p, "_vy_grad_ready", None) is not None for p in ps if p is not None)


def _param(module, name: str):
    """module.<name>, past nn.Module's attribute look-up where it is a parameter (this runs several times per launch)."""
    p = module._parameters.get(name)
    return getattr(module, name) if p is None else p


def _buffer(nbytes: int, like: torch.Tensor) -> torch.Tensor:
    return torch.empty(nbytes, device=like.device, dtype=torch.uint8)


def _pieces(buf: torch.Tensor, specs) -> list:
    """Views of `buf`, one per (shape, dtype), one after the other on boundaries of 256 bytes: the library's layout of what a forward call leaves."""
    out, at = [], 0
    for shape, dt in specs:
        n = math.prod(shape) * dt.itemsize
        out.append(buf[at:at + n].view(dt).view(shape))
        at += (n + 255) // 256 * 256
    return out


def pack(ts) -> torch.Tensor:
    """The buffer that the one call would have left, from the tensors of the general way."""
    buf = _buffer(sum((t.numel() * t.element_size() + 255) // 256 * 256 for t in ts), ts[0])
    for view, t in zip(_pieces(buf, [(tuple(t.shape), t.dtype) for t in ts]), ts):
        view.copy_(t)
    return buf


# ---- attention block ----
class AttentionParts:
    """The parameters of one attention block as they are now."""

    __slots__ = ("mod", "lin", "ws", "bs", "dense", "wo", "bo", "ln", "gamma", "beta", "drops")

    def __init__(self, mod):
        m = mod._modules
        self.mod, out = mod, m["out"]
        self.lin = [m["qkv"]] if "qkv" in m else [m["query"], m["key"], m["value"]]
        self.ws, self.bs = [_param(l, "weight") for l in self.lin], [_param(l, "bias") for l in self.lin]
        inner = out._modules
        self.dense, self.ln, drop = inner["dense"], inner["layernorm"], inner["dropout"]
        self.wo, self.bo, self.gamma, self.beta = _param(self.dense, "weight"), _param(self.dense, "bias"), _param(self.ln, "weight"), _param(self.ln, "bias")
        self.drops = out.training and drop.p > 0.0


def attention_key(a: AttentionParts, x2d, B, S, mask, rope, kv, decode_no_mask, train: bool) -> Optional[tuple]:
    """What the sublayer's tilings depend on; None where the one call does not apply."""
    T, ws, bs = x2d.dtype, a.ws, a.bs
    if T not in _DT or _lib.TIMER is not None or ops._SIDE_ON or a.drops or type(a.ln) is not torch.nn.LayerNorm or a.gamma is None or a.beta is None:
        return None
    if not _plain(T, x2d, *ws, *bs, a.wo, a.bo, a.gamma, a.beta) or any((b is None) != (bs[0] is None) for b in bs):
        return None
    (rows, H), Hq, Hkv = x2d.shape, a.mod.num_attention_heads, a.mod._kv_heads
    if sum(w.shape[0] for w in ws) != (Hq + 2 * Hkv) * 64 or ws[0].shape[1] != H or a.wo.shape != (H, Hq * 64) or a.gamma.numel() != H or rows != B * S:
        return None
    if train and (H >= 4096 or (Hq + 2 * Hkv) * 64 >= 4096 or _direct((*ws, *bs, a.wo, a.bo, a.gamma, a.beta))):
        return None
    if not _stacked(ws) or (bs[0] is not None and not _stacked(bs)):
        pack_linears(a.lin)
    if rope is not None and not (_plain(torch.float32, rope[0], rope[1]) and rope[0].shape[1] == 32):
        return None
    pad = mask.key_padding
    if pad is not None and (pad.dtype is not torch.uint8 or not pad.is_cuda or pad.stride(1) != 1):
        return None
    kind = 0
    if kv is not None:
        k, v = kv.k_buf, kv.v_buf
        kind = 2 if S == 1 and decode_no_mask else 1
        if train or k.stride() != v.stride() or k.dtype is not v.dtype or not k.is_cuda or not v.is_cuda or k.shape[3] != 64 or k.stride(3) != 1 or k.shape[1] != Hkv or k.shape[0] < B:
            return None
        if k.dtype is not torch.bfloat16 and (kind == 1 or k.dtype not in _DT):
            return None
    return ("attention", train, B, S, H, T, Hq, Hkv, bs[0] is not None, a.bo is not None, rope is not None, kind, gemm_tune.ENABLED, x2d.device)


def attention_weights_fit(a: AttentionParts, x2d) -> bool:
    """Are the parameters still what `attention_key` found? What was put into their `.data` since the forward pass may lie elsewhere or be of another type."""
    ws, bs, H, n = a.ws, a.bs, x2d.shape[1], (a.mod.num_attention_heads + 2 * a.mod._kv_heads) * 64
    if not _plain(x2d.dtype, *ws, *bs, a.wo, a.bo, a.gamma, a.beta) or sum([w.numel() for w in ws]) != n * H or a.wo.numel() != a.mod.num_attention_heads * 64 * H:
        return False
    if a.gamma.numel() != H or a.beta.numel() != H or (a.bo is not None and a.bo.numel() != H) or (bs[0] is not None and sum([b.numel() for b in bs]) != n):
        return False
    stacked = lambda: _stacked(ws) and (bs[0] is None or _stacked(bs))  # noqa: E731
    if not stacked():
        pack_linears(a.lin)
        return stacked()   # the module may hold other parameters by now
    return True


def _attention_args(a: AttentionParts, x2d, B, S, mask, rope, kv, start_pos, kind: int, save: bool):
    mod = a.mod
    st = _ATTN(seqs=B, tokens=S, width=x2d.shape[1], heads=mod.num_attention_heads, kv_heads=mod._kv_heads, dtype=_DT[x2d.dtype], x=x2d.data_ptr(),
               w_qkv=a.ws[0].data_ptr(), b_qkv=ops._ptr(a.bs[0]), w_out=a.wo.data_ptr(), b_out=ops._ptr(a.bo), gamma=a.gamma.data_ptr(),
               beta=a.beta.data_ptr(), eps=a.ln.eps, causal=int(mask.causal), q_pos0=mask.q_pos0, weights_static=0 if torch.is_grad_enabled() else 1, save=int(save),
               stream=ops._stream())
    if rope is not None:
        cos, sin, base = rope
        st.rope_cos, st.rope_sin, st.rope_rows, st.rope_pos = cos.data_ptr(), sin.data_ptr(), cos.shape[0], 0 if base is None else start_pos - base
    if mask.key_padding is not None:
        st.key_padding, st.kpm_stride = mask.key_padding.data_ptr(), mask.key_padding.stride(0)
    if kv is not None:
        k = kv.k_buf
        st.k_cache, st.v_cache, st.cache_dtype, st.cache_len, st.start = k.data_ptr(), kv.v_buf.data_ptr(), _DT[k.dtype], k.shape[2], kv.start_pos
        st.c_sb, st.c_sh, st.c_sl, _ = k.stride()
        if kind == 2:
            st.decode, st.tickets = 1, ops._tickets(x2d.device, B * mod._kv_heads).data_ptr()
    return st


def attention_forward(a: AttentionParts, x2d, B, S, mask, rope, kv, start_pos, key: tuple, hints: tuple, save: bool = False):
    """(y, scratch) of the block under `key`."""
    st = _attention_args(a, x2d, B, S, mask, rope, kv, start_pos, key[11], save)
    st.hint_qkv, st.hint_out = hints
    nbytes = _lib.lib().vy_attn_block_bytes(byref(st))
    y, scratch = torch.empty_like(x2d), _buffer(nbytes, x2d)
    st.y, st.scratch, st.scratch_bytes = y.data_ptr(), scratch.data_ptr(), nbytes
    _lib.run("vy_attn_block_fwd", st)
    return y, scratch


def attention_backward(a: AttentionParts, x2d, scratch, dy, B, S, mask, rope, start_pos, hints: tuple):
    """[dx, the projections' weight and bias gradients, d dense.weight (, .bias), d gamma, d beta] as AttentionBlockFn returns them."""
    st = _attention_args(a, x2d, B, S, mask, rope, None, start_pos, 0, True)
    new = lambda *s: torch.empty(s, device=dy.device, dtype=x2d.dtype)  # noqa: E731
    rows = [w.shape[0] for w in a.ws]
    dx, dw, dwo, dg, db = torch.empty_like(x2d), new(sum(rows), x2d.shape[1]), torch.empty_like(a.wo), torch.empty_like(a.gamma), torch.empty_like(a.beta)
    dbq = new(sum(rows)) if a.bs[0] is not None else None
    dbo = torch.empty_like(a.bo) if a.bo is not None else None
    L = _lib.lib()
    nbytes = L.vy_attn_block_work_bytes(byref(st))
    work, split = _buffer(nbytes, x2d), ops._splitk_workspace(dy.device)
    st.scratch, st.scratch_bytes, st.work, st.work_bytes = scratch.data_ptr(), scratch.numel(), work.data_ptr(), nbytes
    st.split_ws, st.split_bytes = split.data_ptr(), split.numel() * 4
    st.dy, st.dx, st.dw_qkv, st.db_qkv, st.dw_out, st.db_out = dy.data_ptr(), dx.data_ptr(), dw.data_ptr(), ops._ptr(dbq), dwo.data_ptr(), ops._ptr(dbo)
    st.dgamma, st.dbeta = dg.data_ptr(), db.data_ptr()
    st.hint_dw_out, st.hint_d_out, st.hint_d_qkv, st.hint_dw_qkv = hints
    _lib.run("vy_attn_block_bwd", st)
    grads = [dx, *dw.split(rows)]
    if dbq is not None:
        grads += dbq.split(rows)
    grads.append(dwo)
    if dbo is not None:
        grads.append(dbo)
    return grads + [dg, db]


def attention_saved(buf, x2d, B, S, heads, kv_heads) -> list:
    """[q, k, v, attn, s, lse, mean, rstd] of a forward call with `save`."""
    bf, f32, (rows, H) = torch.bfloat16, torch.float32, x2d.shape
    return _pieces(buf, [((B, heads, S, 64), bf), ((B, kv_heads, S, 64), bf), ((B, kv_heads, S, 64), bf), ((rows, heads * 64), x2d.dtype), ((rows, H), x2d.dtype),
                         ((B, heads, S), f32), ((rows,), f32), ((rows,), f32)])


# ---- feed-forward block ----
def ffn_key(act, h2d, input2d, w1, b1, w2, b2, ln, gamma, beta, drops: bool, train: bool) -> Optional[tuple]:
    T = h2d.dtype
    if T not in _DT or act not in _ACT or drops or _lib.TIMER is not None or ops._SIDE_ON or type(ln) is not torch.nn.LayerNorm or gamma is None or beta is None:
        return None
    if not _plain(T, h2d, input2d, w1, b1, w2, b2, gamma, beta):
        return None
    (rows, H), F = h2d.shape, w1.shape[0]
    if w1.shape[1] != H or w2.shape != (H, F) or input2d.shape != (rows, H) or gamma.numel() != H:
        return None
    if train and (H >= 4096 or F >= 4096 or _direct((w1, b1, w2, b2, gamma, beta))):
        return None
    return ("ffn", train, rows, H, F, T, act, b1 is not None, b2 is not None, gemm_tune.ENABLED, h2d.device)


def ffn_weights_fit(h2d, w1, b1, w2, b2, gamma, beta, inner: int) -> bool:
    """As attention_weights_fit."""
    H = h2d.shape[1]
    return (_plain(h2d.dtype, w1, b1, w2, b2, gamma, beta) and w1.numel() == w2.numel() == inner * H and gamma.numel() == beta.numel() == H and
            (b1 is None or b1.numel() == inner) and (b2 is None or b2.numel() == H))


def _ffn_args(act, h2d, input2d, w1, b1, w2, b2, gamma, beta, eps, save: bool):
    fwd, bwd = _ACT[act]
    return _FFN(rows=h2d.shape[0], width=h2d.shape[1], inner=w1.shape[0], dtype=_DT[h2d.dtype], act=fwd, dact=bwd, h=h2d.data_ptr(),
                input=input2d.data_ptr() if input2d is not None else h2d.data_ptr(), w1=w1.data_ptr(), b1=ops._ptr(b1), w2=w2.data_ptr(), b2=ops._ptr(b2),
                gamma=gamma.data_ptr(), beta=beta.data_ptr(), eps=eps, weights_static=0 if torch.is_grad_enabled() else 1, save=int(save), stream=ops._stream())


def ffn_saved(buf, h2d, inner: int) -> list:
    """[z, a, s, mean, rstd] of a forward call with `save`."""
    (rows, H), T = h2d.shape, h2d.dtype
    return _pieces(buf, [((rows, inner), T), ((rows, inner), T), ((rows, H), T), ((rows,), torch.float32), ((rows,), torch.float32)])


def ffn_forward(act, h2d, input2d, w1, b1, w2, b2, gamma, beta, eps, hints: tuple, save: bool = False):
    st = _ffn_args(act, h2d, input2d, w1, b1, w2, b2, gamma, beta, eps, save)
    st.hint_1, st.hint_2 = hints
    nbytes = _lib.lib().vy_ffn_block_bytes(byref(st))
    y, scratch = torch.empty_like(h2d), _buffer(nbytes, h2d)
    st.y, st.scratch, st.scratch_bytes = y.data_ptr(), scratch.data_ptr(), nbytes
    _lib.run("vy_ffn_block_fwd", st)
    return y, scratch


def ffn_backward(act, h2d, scratch, dy, w1, b1, w2, b2, gamma, beta, eps, hints: tuple):
    """(dh, d input, dW1, db1, dW2, db2, d gamma, d beta)"""
    st = _ffn_args(act, h2d, None, w1, b1, w2, b2, gamma, beta, eps, True)
    like = torch.empty_like
    dh, ds, dw1, dw2, dg, db = like(h2d), like(h2d), like(w1), like(w2), like(gamma), like(beta)
    db1, db2 = (None if b is None else like(b) for b in (b1, b2))
    nbytes = _lib.lib().vy_ffn_block_work_bytes(byref(st))
    work, split = _buffer(nbytes, h2d), ops._splitk_workspace(dy.device)
    st.scratch, st.scratch_bytes, st.work, st.work_bytes = scratch.data_ptr(), scratch.numel(), work.data_ptr(), nbytes
    st.split_ws, st.split_bytes = split.data_ptr(), split.numel() * 4
    st.dy, st.dh, st.d_input, st.dw1, st.db1, st.dw2, st.db2 = dy.data_ptr(), dh.data_ptr(), ds.data_ptr(), dw1.data_ptr(), ops._ptr(db1), dw2.data_ptr(), ops._ptr(db2)
    st.dgamma, st.dbeta = dg.data_ptr(), db.data_ptr()
    st.hint_dw2, st.hint_d2, st.hint_dw1, st.hint_d1 = hints
    _lib.run("vy_ffn_block_bwd", st)
    return dh, ds, dw1, db1, dw2, db2, dg, db
