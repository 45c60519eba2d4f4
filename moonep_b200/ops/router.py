"""Python front end of csrc/device/router.cu: top-k routing of a block's gate logits and its gradient, and the dense
SwiGLU of a shared expert."""

from __future__ import annotations

import torch

from .. import _native


def supported(E: int, K: int) -> bool:
    return K <= 32 and K <= E <= _native.load().mep_route_max_experts()


def route(logits, bias, K: int, with_probs: bool = False):
    """``(w [S, K] fp32, topk [S, K] int32, tokens_per_expert [E] int32, probs)`` of bf16 ``logits [S, E]`` plus the fp32
    ``bias [E]``: the K most probable experts per token, descending, their probabilities renormalised.  ``probs``
    (fp32 ``[S, E]``, for ``route_bwd``) only with ``with_probs``.  Bit for bit what the torch operators give."""
    S, E = logits.shape
    assert logits.dtype == torch.bfloat16 and logits.is_contiguous() and bias.dtype == torch.float32 and bias.numel() == E
    dev = logits.device
    w = torch.empty((S, K), dtype=torch.float32, device=dev)
    ints = torch.empty(S * K + E, dtype=torch.int32, device=dev)
    topk, tpe = ints[:S * K].view(S, K), ints[S * K:]
    probs = torch.empty((S, E), dtype=torch.float32, device=dev) if with_probs else None
    rc = _native.load().mep_route(logits.data_ptr(), bias.data_ptr(), w.data_ptr(), topk.data_ptr(), tpe.data_ptr(), _native.ptr(probs),
                                  S, E, K, _native.raw_stream())
    if rc:
        _native.check(rc, "route")
    return w, topk, tpe, probs


def route_bwd(probs, dw, topk):
    """Gradient of the logits (bf16 ``[S, E]``) from the gradient ``dw`` of the route weights."""
    (S, K), E = topk.shape, probs.shape[1]
    assert dw.dtype == torch.float32 and dw.is_contiguous() and probs.is_contiguous() and topk.is_contiguous()
    out = torch.empty((S, E), dtype=torch.bfloat16, device=probs.device)
    rc = _native.load().mep_route_bwd(probs.data_ptr(), dw.data_ptr(), topk.data_ptr(), out.data_ptr(), S, E, K, _native.raw_stream())
    if rc:
        _native.check(rc, "route_bwd")
    return out


def swiglu(gu):
    """``silu(gu[:, :n]) * gu[:, n:]`` for a contiguous bf16 ``[rows, 2n]``, rounded like the two operators."""
    rows, n = gu.shape[0], gu.shape[1] // 2
    act = torch.empty((rows, n), dtype=torch.bfloat16, device=gu.device)
    rc = _native.load().mep_swiglu(gu.data_ptr(), act.data_ptr(), rows, n, _native.raw_stream())
    if rc:
        _native.check(rc, "swiglu")
    return act


def swiglu_bwd(dact, gu):
    """Gradient of ``swiglu`` with respect to ``gu``."""
    rows, n = dact.shape
    assert dact.is_contiguous() and gu.is_contiguous()
    dgu = torch.empty_like(gu)
    rc = _native.load().mep_swiglu_dense_bwd(dact.data_ptr(), gu.data_ptr(), dgu.data_ptr(), rows, n, _native.raw_stream())
    if rc:
        _native.check(rc, "swiglu_bwd")
    return dgu
