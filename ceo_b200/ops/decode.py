"""A few tokens through the whole model in one native call (``csrc/decode.cu``).

``decode_tokens`` walks the model's parameters, hands their addresses to the host loop in C++
and returns the logits of each sequence's last token; ``None`` means the model or the call has a
form that loop does not cover (PRISM, LayerNorm, another activation, FP8 or sharded weights,
hooks on a submodule, states that are not dense fp32 ...) and the caller runs its layer-by-layer
path.  Nothing is kept between calls.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib
from . import matmul as matmul_ops

MAX_ROWS = 128  # rows of one call (sequences, or tokens of one prompt)


def _hooked(m) -> bool:
    return bool(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks
                or m._backward_pre_hooks)


def _dense(w, shape, dev) -> bool:
    return (w.dtype is torch.bfloat16 and w.shape == shape and w.device == dev
            and w.is_contiguous() and not w.data_ptr() & 15 and not hasattr(w, "fsdp_gather"))


def decode_tokens(model, tokens: torch.Tensor, states, want_logits: bool = True):
    """tokens: (B, T) ids with T = 1 or B = 1 and B * T <= 128; states: one (B,H,d,d) fp32 tensor
    per block, updated in place.  Returns (B, V) fp32 logits (True when not wanted), or None."""
    c = model.cfg
    B, T = tokens.shape
    dev = model.embed_tokens.device
    if (dev.type != "cuda" or tokens.device != dev or B * T < 1 or B * T > MAX_ROWS
            or (B > 1 and T > 1) or not matmul_ops.FUSED_SWIGLU or c.activation != "swiglu"
            or len(states) != len(model.blocks) or torch.cuda.current_device() != dev.index):
        return None
    D, V, F = c.hidden_dim, c.vocab_size, c.intermediate_dim
    H, d = c.num_heads, c.head_dim
    head = model.head_weight()
    norm = model.final_norm
    if (d not in (64, 128) or D % 8 or D > 8192 or F % 32 or V % 4 or B * H > 65535
            or norm.kind != "rmsnorm" or _hooked(norm) or not _dense(norm.weight, (D,), dev)
            or not _dense(model.embed_tokens, (V, D), dev) or not _dense(head, (V, D), dev)):
        return None
    hd, eps = H * d, norm.eps
    table = (ctypes.c_void_p * (8 * len(model.blocks)))()
    first = None
    for i, (blk, st) in enumerate(zip(model.blocks, states)):
        mods = blk._modules
        ln1, ln2, efla, mlp = mods["ln1"], mods["ln2"], mods["efla"], mods["mlp"]
        if (mods.get("prism") is not None or mlp.fp8 is not None or mlp.act != "swiglu"
                or _hooked(ln1) or _hooked(ln2) or _hooked(mlp)
                or ln1.kind != "rmsnorm" or ln2.kind != "rmsnorm" or ln1.eps != eps
                or ln2.eps != eps):
            return None
        ep, mp = efla._parameters, mlp._parameters
        n1, n2 = ln1._parameters["weight"], ln2._parameters["weight"]
        w_qkv, w_o, w_up, w_down = ep["w_qkv"], ep["w_o"], mp["w_up"], mp["w_down"]
        form = (efla.P, efla.normalize, efla.per_token_beta, w_qkv.shape[0])
        if first is None:
            first = form
            P, n_proj = efla.P, w_qkv.shape[0]
            if n_proj % 8 or n_proj < P * hd + (H if efla.per_token_beta else 0):
                return None
        if (form != first or not _dense(n1, (D,), dev) or not _dense(n2, (D,), dev)
                or not _dense(w_qkv, (n_proj, D), dev) or not _dense(w_o, (D, hd), dev)
                or not _dense(w_up, (2 * F, D), dev) or not _dense(w_down, (D, F), dev)
                or st.dtype is not torch.float32 or st.shape != (B, H, d, d)
                or st.device != dev or not st.is_contiguous() or st.requires_grad):
            return None
        beta = 0
        if not efla.per_token_beta:
            bp = ep["beta_param"]
            if bp.dtype is not torch.float32 or bp.numel() != 1 or bp.device != dev:
                return None
            beta = bp.data_ptr()
        table[8 * i:8 * i + 8] = [n1.data_ptr(), w_qkv.data_ptr(), w_o.data_ptr(), n2.data_ptr(),
                                  w_up.data_ptr(), w_down.data_ptr(), st.data_ptr(), beta]
    rows = B * T
    ids = tokens.reshape(-1).to(torch.int64).contiguous()
    ws = torch.empty(sum(-(-rows * n // 128) * 128 for n in (D, D, n_proj, hd, F)),
                     dtype=torch.bfloat16, device=dev)
    logits = torch.empty(B, V, dtype=torch.float32, device=dev) if want_logits else None
    _lib.check(_lib.lib().ceo_decode_tokens(
        ids.data_ptr(), model.embed_tokens.data_ptr(), V, ctypes.addressof(table),
        len(model.blocks), norm.weight.data_ptr(), head.data_ptr(), _lib.ptr(logits),
        ws.data_ptr(), B, T, D, H, d, P, n_proj, F, int(first[1]), float(eps),
        _lib.status_word(dev).data_ptr(), _lib.stream()), "ceo_decode_tokens")
    _lib.launch_count += 1 + 7 * len(model.blocks) + (2 if want_logits else 0)
    for st in states:
        if not st.is_inference():
            torch.autograd.graph.increment_version(st)  # as an in-place op would
    return logits if want_logits else True
