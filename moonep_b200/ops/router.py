"""Python front end of csrc/device/router.cu: top-k routing of a block's gate logits and its gradient, and the dense
SwiGLU of a shared expert."""

from __future__ import annotations

import torch

from .. import _native


def supported(E: int, K: int) -> bool:
    return K <= 32 and K <= E <= _native.load().mep_route_max_experts()


def route(logits, bias, K: int):
    """``(w [S, K] fp32, topk [S, K] int32, tokens_per_expert [E] int32)`` of bf16 ``logits [S, E]`` plus the fp32
    ``bias [E]``: the K largest per token, descending, softmax over them."""
    S, E = logits.shape
    assert logits.dtype == torch.bfloat16 and logits.is_contiguous() and bias.dtype == torch.float32 and bias.numel() == E
    dev = logits.device
    w = torch.empty((S, K), dtype=torch.float32, device=dev)
    ints = torch.empty(S * K + E, dtype=torch.int32, device=dev)
    topk, tpe = ints[:S * K].view(S, K), ints[S * K:]
    rc = _native.load().mep_route(logits.data_ptr(), bias.data_ptr(), w.data_ptr(), topk.data_ptr(), tpe.data_ptr(), S, E, K, _native.raw_stream())
    if rc:
        _native.check(rc, "route")
    return w, topk, tpe


def route_bwd(w, dw, topk, E: int):
    """Gradient of the logits (bf16 ``[S, E]``) from the gradient ``dw`` of the route weights."""
    S, K = w.shape
    assert dw.dtype == torch.float32 and dw.is_contiguous() and w.is_contiguous() and topk.is_contiguous()
    out = torch.empty((S, E), dtype=torch.bfloat16, device=w.device)
    rc = _native.load().mep_route_bwd(w.data_ptr(), dw.data_ptr(), topk.data_ptr(), out.data_ptr(), S, E, K, _native.raw_stream())
    if rc:
        _native.check(rc, "route_bwd")
    return out


def swiglu(gu):
    """``silu(gu[:, :n]) * gu[:, n:]`` for a contiguous bf16 ``[rows, 2n]``."""
    rows, n = gu.shape[0], gu.shape[1] // 2
    act = torch.empty((rows, n), dtype=torch.bfloat16, device=gu.device)
    rc = _native.load().mep_swiglu(gu.data_ptr(), act.data_ptr(), rows, n, _native.raw_stream())
    if rc:
        _native.check(rc, "swiglu")
    return act
