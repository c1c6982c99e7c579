"""Inference through the whole model in one native call: a few tokens (``csrc/decode.cu``) or
whole sequences (``csrc/forward.cu``).

``decode_tokens`` and ``forward_hidden`` walk the model's parameters, hand their addresses to
the host loop in C++ and return its result; ``None`` means the model or the call has a form that
loop does not cover (PRISM, LayerNorm, another activation, FP8 or sharded weights, hooks or
replaced methods on a submodule, states that are not dense fp32 ...) and the caller runs its
layer-by-layer path.  Nothing is kept between calls.
"""
from __future__ import annotations

import ctypes

import torch
from torch.nn.modules import module as _nn_module

from . import _lib
from . import efla as efla_ops
from . import matmul as matmul_ops

MAX_ROWS = 128  # rows of one decode call (sequences, or tokens of one prompt)


def _hooked(*mods) -> bool:
    return any(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks
               or m._backward_pre_hooks or "forward" in m.__dict__ or "decode_step" in m.__dict__
               for m in mods)


def _dense(w, shape, dev) -> bool:
    return (w is not None and w.dtype is torch.bfloat16 and w.shape == shape and w.device == dev
            and w.is_contiguous() and not w.data_ptr() & 15 and not hasattr(w, "fsdp_gather"))


def _state_ok(st, shape, dev) -> bool:
    return (st.dtype is torch.float32 and st.shape == shape and st.device == dev
            and st.is_contiguous() and not st.data_ptr() & 15)


class _Form:
    """Addresses and sizes of a model the native loops cover."""
    __slots__ = ("weights", "P", "n_proj", "normalize", "eps")


def _form(model):
    from ..models import model as M
    c = model.cfg
    dev = model.embed_tokens.device
    if (dev.type != "cuda" or torch.cuda.current_device() != dev.index
            or not matmul_ops.FUSED_SWIGLU or c.activation != "swiglu"
            or _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks
            or torch.autograd.forward_ad._current_level >= 0):  # tangents: refused further down
        return None
    D, V, F = c.hidden_dim, c.vocab_size, c.intermediate_dim
    H, d = c.num_heads, c.head_dim
    hd = H * d
    norm = model.final_norm
    if (d not in (64, 128) or D % 8 or D > 8192 or F % 32 or type(norm) is not M.Norm
            or norm.kind != "rmsnorm" or _hooked(norm) or not _dense(norm.weight, (D,), dev)
            or not _dense(model.embed_tokens, (V, D), dev)):
        return None
    f = _Form()
    f.weights, f.eps, form = [], norm.eps, None
    for blk in model.blocks:
        if type(blk) is not M.Block:  # a wrapper, or anything else that takes a block's place
            return None
        mods = blk._modules
        ln1, ln2, efla, mlp = (mods.get(k) for k in ("ln1", "ln2", "efla", "mlp"))
        if (type(efla) is not M.EflaLayer or type(mlp) is not M.MLP
                or type(ln1) is not M.Norm or type(ln2) is not M.Norm
                or mods.get("prism") is not None or mlp.fp8 is not None or efla.fp8 is not None
                or mlp.act != "swiglu" or _hooked(blk, ln1, ln2, efla, mlp)
                or ln1.kind != "rmsnorm" or ln2.kind != "rmsnorm" or ln1.eps != f.eps
                or ln2.eps != f.eps):
            return None
        ep, mp = efla._parameters, mlp._parameters
        n1, n2 = ln1._parameters.get("weight"), ln2._parameters.get("weight")
        w_qkv, w_o = ep.get("w_qkv"), ep.get("w_o")
        w_up, w_down = mp.get("w_up"), mp.get("w_down")
        if w_qkv is None:
            return None
        this = (efla.P, efla.normalize, efla.per_token_beta, w_qkv.shape[0], efla.H, efla.d)
        if form is None:
            form = this
            f.P, f.normalize, f.n_proj = efla.P, int(efla.normalize), w_qkv.shape[0]
            if (f.n_proj % 8 or f.n_proj < f.P * hd + (H if efla.per_token_beta else 0)
                    or (efla.H, efla.d) != (H, d)):
                return None
        if (this != form or not _dense(n1, (D,), dev) or not _dense(n2, (D,), dev)
                or not _dense(w_qkv, (f.n_proj, D), dev) or not _dense(w_o, (D, hd), dev)
                or not _dense(w_up, (2 * F, D), dev) or not _dense(w_down, (D, F), dev)):
            return None
        beta = 0
        if not efla.per_token_beta:
            bp = ep.get("beta_param")
            if bp is None or bp.dtype is not torch.float32 or bp.numel() != 1 or bp.device != dev:
                return None
            beta = bp.data_ptr()
        f.weights.append([n1.data_ptr(), w_qkv.data_ptr(), w_o.data_ptr(), n2.data_ptr(),
                          w_up.data_ptr(), w_down.data_ptr(), beta])
    return f if f.weights else None


def decode_tokens(model, tokens: torch.Tensor, states, want_logits: bool = True):
    """tokens: (B, T) ids with T = 1 or B = 1 and B * T <= 128; states: one (B,H,d,d) fp32 tensor
    per block, updated in place.  Returns (B, V) fp32 logits (True when not wanted), or None."""
    c = model.cfg
    B, T = tokens.shape
    if not 1 <= B * T <= MAX_ROWS or (B > 1 and T > 1) or len(states) != len(model.blocks):
        return None
    f = _form(model)
    if f is None:
        return None
    D, V, F, H, d = c.hidden_dim, c.vocab_size, c.intermediate_dim, c.num_heads, c.head_dim
    dev = model.embed_tokens.device
    head = model.head_weight()
    if (tokens.device != dev or V % 4 or B * H > 65535 or not _dense(head, (V, D), dev)
            or any(st.requires_grad or not _state_ok(st, (B, H, d, d), dev) for st in states)):
        return None
    n = len(f.weights)
    table = (ctypes.c_void_p * (8 * n))()
    for i, (w, st) in enumerate(zip(f.weights, states)):
        table[8 * i:8 * i + 8] = w[:6] + [st.data_ptr(), w[6]]
    rows = B * T
    ids = tokens.reshape(-1).to(torch.int64).contiguous()
    ws = torch.empty(sum(-(-rows * k // 128) * 128 for k in (D, D, f.n_proj, H * d, F)),
                     dtype=torch.bfloat16, device=dev)
    logits = torch.empty(B, V, dtype=torch.float32, device=dev) if want_logits else None
    _lib.check(_lib.lib().ceo_decode_tokens(
        ids.data_ptr(), model.embed_tokens.data_ptr(), V, ctypes.addressof(table), n,
        model.final_norm.weight.data_ptr(), head.data_ptr(), _lib.ptr(logits), ws.data_ptr(), B, T,
        D, H, d, f.P, f.n_proj, F, f.normalize, float(f.eps), _lib.status_word(dev).data_ptr(),
        _lib.stream()), "ceo_decode_tokens")
    _lib.launch_count += 1 + 7 * n + (2 if want_logits else 0)
    for st in states:
        if not st.is_inference():
            torch.autograd.graph.increment_version(st)  # as an in-place op would
    return logits if want_logits else True


def forward_hidden(model, tokens: torch.Tensor, states=None, resets=None):
    """The rows after the final norm (B,T,D) and the final states of every block, without
    gradients, for tokens (B,T) with T a multiple of the chunk; or None."""
    c = model.cfg
    if tokens.dim() != 2 or tokens.shape[0] < 1 or tokens.shape[1] < 1 \
            or tokens.shape[1] % efla_ops.CHUNK or (model.training and c.dropout > 0.0):
        return None
    f = _form(model)
    if f is None:
        return None
    B, T = tokens.shape
    D, V, F, H, d = c.hidden_dim, c.vocab_size, c.intermediate_dim, c.num_heads, c.head_dim
    dev = model.embed_tokens.device
    n, nc = len(f.weights), T // efla_ops.CHUNK
    if tokens.device != dev or any(b.dropout > 0.0 and b.training for b in model.blocks):
        return None
    if states is not None and (len(states) < n or any(
            s is not None and not _state_ok(s, (B, H, d, d), dev) for s in states[:n])):
        return None
    resets = efla_ops._resets_u8(resets, B, nc, dev)
    L = _lib.lib()
    finals = [torch.empty(B, H, d, d, dtype=torch.float32, device=dev) for _ in range(n)]
    table = (ctypes.c_void_p * (9 * n))()
    for i, w in enumerate(f.weights):
        s0 = states[i] if states is not None else None
        table[9 * i:9 * i + 9] = w + [_lib.ptr(s0), finals[i].data_ptr()]
    rows, hd = B * T, H * d
    segs = L.ceo_efla_fwd_segments(B, T, H, d)
    parts = [rows * D * 2] * 2 + [rows * f.n_proj * 2] + [rows * hd * 2] * (5 if f.P == 3 else 4) \
        + [rows * H * 4] * 3 + [B * H * nc * d * d * 2, rows * F * 2] \
        + ([3 * B * H * segs * d * d * 4] if segs > 1 else [])
    size = sum(-(-p // 256) * 256 for p in parts)
    ws = torch.empty(size, dtype=torch.uint8, device=dev)
    ids = tokens.reshape(-1).to(torch.int64).contiguous()
    out = torch.empty(B, T, D, dtype=torch.bfloat16, device=dev)
    _lib.check(L.ceo_forward_tokens(
        ids.data_ptr(), model.embed_tokens.data_ptr(), V, ctypes.addressof(table), n,
        model.final_norm.weight.data_ptr(), out.data_ptr(), ws.data_ptr(), size, _lib.ptr(resets),
        B, T, D, H, d, f.P, f.n_proj, F, f.normalize, float(f.eps),
        _lib.status_word(dev).data_ptr(), _lib.stream()), "ceo_forward_tokens")
    _lib.launch_count += 2 + n * (12 if segs > 1 else 10)  # spans: a map pass and a fold more
    return out, finals
