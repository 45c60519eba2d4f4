"""MoE transformer FFN blocks of the model families the benchmarks name.

``MoEBlock`` = router (softmax top-k over a dense gate projection) + expert-parallel routed
experts (SwiGLU) + optional dense shared expert, with a fused SGD step for benchmarks.  Shapes:

    deepseek_v3   H=7168, H'=2048, K=8, epn=32 (E=256 at EP=8)
    kimi_k2       H=7168, H'=2048, K=8, epn=48 (E=384 at EP=8), one shared expert
    qwen3_30b_a3b H=2048, H'=768,  K=8, epn=16 (E=128 at EP=8)

The reference library contains no model code; these blocks exist so that its headline
benchmark ("MoE-layer step vs maxvio") can be run end to end through this package.
"""

from __future__ import annotations

import os
from dataclasses import dataclass

import torch
import torch.distributed as dist

from ..api import Buffer
from ..moe_layer import ExpertParallelMoE, moe_apply, no_update
from ..ops import grouped_gemm as gg
from ..ops import router as rt
from ..pools import ExpertPools


@dataclass(frozen=True)
class MoEConfig:
    name: str
    H: int
    Hp: int
    K: int
    epn: int
    shared_experts: int = 0
    S: int = 4096
    token_padding: int = 128


CONFIGS = {
    "deepseek_v3": MoEConfig("deepseek_v3", 7168, 2048, 8, 32),
    "kimi_k2": MoEConfig("kimi_k2", 7168, 2048, 8, 48, shared_experts=1),
    "qwen3_30b_a3b": MoEConfig("qwen3_30b_a3b", 2048, 768, 8, 16, S=8192),
    "tiny": MoEConfig("tiny", 256, 256, 2, 2, shared_experts=1, S=128),
}


def _block_forward(blk, hidden, router, s0, s1, keep: bool):
    """Output, and with ``keep`` what the backward pass needs: (MoE context, probabilities, table, shared gate/up, activation)."""
    w, topk, tpe, probs = rt.route(hidden @ router, blk.router_bias, blk.cfg.K, with_probs=keep)
    out, mctx = blk.moe.forward(hidden, w, topk, tpe, need_backward=keep)
    gu = act = None
    if s0 is not None:
        gu = hidden @ s0
        act = rt.swiglu(gu)
        out.addmm_(act, s1)
    return out, mctx, probs, topk, gu, act


class _BlockFn(torch.autograd.Function):
    """A whole block as one autograd node: the three contributions to the input gradient (experts, router, shared
    expert, added in this order) are accumulated by the GEMMs that produce them instead of by additions over ``[S, H]``."""

    @staticmethod
    def forward(ctx, hidden, router, s0, s1, blk):
        out, ctx.mctx, probs, topk, gu, act = _block_forward(blk, hidden, router, s0, s1, True)
        ctx.blk = blk
        ctx.save_for_backward(hidden, router, s0, s1, probs, topk, gu, act)
        return out

    @staticmethod
    def backward(ctx, dy):
        hidden, router, s0, s1, probs, topk, gu, act = ctx.saved_tensors
        need = ctx.needs_input_grad
        if torch.is_grad_enabled():      # create_graph: what comes back has to have derivatives of its own
            return _block_backward_graph(ctx, dy)
        dy = dy.contiguous()
        dx = drouter = ds0 = ds1 = None
        if need[0] or need[1]:           # else nothing in front of the experts wants a gradient, and they are frozen with it
            dx, dw = ctx.blk.moe.backward(ctx.mctx, dy)
            dl = rt.route_bwd(probs, dw, topk)
            drouter = hidden.t() @ dl if need[1] else None
            if need[0]:
                dx.addmm_(dl, router.t())
        if s0 is not None:
            dgu = rt.swiglu_bwd(dy @ s1.t(), gu)
            ds1 = act.t() @ dy if need[3] else None
            ds0 = hidden.t() @ dgu if need[2] else None
            if need[0]:
                dx.addmm_(dgu, s0.t())
        return dx if need[0] else None, drouter, ds0, ds1, None


def _block_backward_graph(ctx, dy):
    """``_BlockFn.backward`` in torch operators around the experts, whose gradients are constants as they are behind
    ``moe_apply``."""
    hidden, router, s0, s1, probs, topk, _, _ = ctx.saved_tensors
    need = ctx.needs_input_grad
    outs, douts, dx = [], [], None
    if need[0] or need[1]:
        with torch.no_grad():
            dx, dw = ctx.blk.moe.backward(ctx.mctx, dy.contiguous())
        logits = (hidden @ router).float()
        v = torch.softmax(probs.log() + (logits - logits.detach()), dim=-1).gather(1, topk.long())      # the saved ones, as functions of the logits
        outs, douts = [v / v.sum(dim=-1, keepdim=True)], [dw]
    if s0 is not None:
        gu = hidden @ s0
        hs = gu.shape[1] // 2
        outs.append((torch.nn.functional.silu(gu[:, :hs]) * gu[:, hs:]) @ s1)
        douts.append(dy)
    ins = [t for t, n in zip((hidden, router, s0, s1), need) if n]
    got = iter(torch.autograd.grad(outs, ins, douts, create_graph=True, allow_unused=True))
    g = [next(got) if n else None for n in need[:4]]
    if need[0]:
        g[0] = dx if g[0] is None else dx + g[0]
    return *g, None


class MoEBlock:
    """One MoE FFN block on this rank of the EP group (weights random-init N(0, 0.02))."""

    def __init__(self, cfg: MoEConfig, world: int = 1, rank: int = 0, group=None, num_sms: int = 32, seed: int = 0,
                 router_skew: float = 0.0, buffer: Buffer | None = None, shared_slots=None):
        """``buffer`` / ``shared_slots``: a ``Buffer`` and a ``pools.SharedSlots`` that several blocks of
        one model use in turn (the communication buffers and the prefetch / reduce slots are scratch
        between a layer's dispatch and its combine, so a model needs them once); without them the
        block creates its own."""
        self.cfg, self.world, self.rank = cfg, world, rank
        dev = torch.device("cuda", torch.cuda.current_device())
        self.E = cfg.epn * world
        # the down GEMM's epilogue sends its rows to their source ranks itself; costs a [S*K, H]
        # receive area per rank (MOONEP_PUSH_COMBINE=0: plain stores, then the combine pulls)
        push = os.environ.get("MOONEP_PUSH_COMBINE", "1") != "0"
        self._own_buffer = buffer is None
        self.buf = buffer if buffer is not None else Buffer(cfg.S, cfg.H, cfg.K, self.E, world, num_sms=num_sms,
                                                            token_padding=cfg.token_padding, group=group, push_combine=push)
        self.pools = ExpertPools(cfg.epn, (cfg.H, cfg.Hp), (cfg.H, cfg.Hp), (cfg.Hp, cfg.H), group=group, with_grads=True,
                                 shared=shared_slots if world > 1 else None)
        g = torch.Generator(device=dev).manual_seed(seed * 7919 + rank)
        for n in ("gate", "up", "down"):
            w = self.pools.local_weight(n)
            w.copy_((torch.randn(w.shape, device=dev, generator=g) * 0.02).to(torch.bfloat16))
            self.pools.compute_grad(n).zero_()
        gs = torch.Generator(device=dev).manual_seed(seed)       # router is replicated: same on all ranks
        self.router = (torch.randn(cfg.H, self.E, device=dev, generator=gs) * 0.02).to(torch.bfloat16).requires_grad_(True)
        # a per-expert bias added to the logits skews the routing (maxvio sweeps)
        self.router_bias = (torch.randn(self.E, device=dev, generator=gs) * router_skew).float()
        # router, experts and shared expert as one autograd node with fused element-wise kernels; sizes those do not
        # cover take the plain torch operators
        self._fused_route = rt.supported(self.E, cfg.K)
        self.shared = None
        if cfg.shared_experts:
            hs = cfg.Hp * cfg.shared_experts
            self.shared = [(torch.randn(cfg.H, 2 * hs, device=dev, generator=g) * 0.02).to(torch.bfloat16).requires_grad_(True),
                           (torch.randn(hs, cfg.H, device=dev, generator=g) * 0.02).to(torch.bfloat16).requires_grad_(True)]
        self.moe = ExpertParallelMoE(self.buf, self.pools)
        # sgd_step() joins the last gradient reduction before it updates ``up``
        self.moe.defer_last_reduction = os.environ.get("MOONEP_DEFER_LAST_REDUCTION", "1") != "0"
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier(group=group)

    def route(self, hidden):
        """Weights (differentiable as often and by whatever transform the caller likes), table and counts, as torch operators;
        a whole block's ``forward`` has them in one launch."""
        cfg = self.cfg
        logits = (hidden @ self.router).float() + self.router_bias
        probs = torch.softmax(logits, dim=-1)
        w, topk = torch.topk(probs, cfg.K, dim=-1)
        w = (w / w.sum(dim=-1, keepdim=True)).contiguous()
        topk = topk.to(torch.int32).contiguous()
        tpe = torch.zeros(self.E, dtype=torch.int32, device=hidden.device)
        tpe.scatter_add_(0, topk.reshape(-1).long(), torch.ones(topk.numel(), dtype=torch.int32, device=hidden.device))
        return w, topk, tpe

    def _fused(self, hidden) -> bool:
        """Whether the fused kernels compute what the torch operators would: bf16 operands in rows, a plain fp32 bias that
        wants no gradient, no autocast to another type."""
        b, bf = self.router_bias, torch.bfloat16
        return (self._fused_route and hidden.dtype == bf and hidden.ndim == 2 and hidden.is_contiguous() and self.router.dtype == bf
                and b.dtype == torch.float32 and b.shape == (self.E,) and b.is_contiguous() and not b.requires_grad
                and (self.shared is None or self.shared[0].dtype == self.shared[1].dtype == bf and self.shared[0].shape[1] % 16 == 0)
                and (not torch.is_autocast_enabled("cuda") or torch.get_autocast_dtype("cuda") == bf))

    def forward(self, hidden):
        if self._fused(hidden):
            shared = self.shared or (None, None)
            if not torch.is_grad_enabled():
                return _block_forward(self, hidden, self.router, *shared, False)[0]
            return _BlockFn.apply(hidden, self.router, *shared, self)
        w, topk, tpe = self.route(hidden)
        out = moe_apply(self.moe, hidden, w, topk, tpe)
        if self.shared is not None:
            gu = hidden @ self.shared[0]
            hs = gu.shape[1] // 2
            out = out + (torch.nn.functional.silu(gu[:, :hs]) * gu[:, hs:]) @ self.shared[1]
        return out

    def parameters(self):
        ps = [self.router]
        if self.shared is not None:
            ps += self.shared
        return ps

    def fuse_optimizer(self, lr: float | None, in_epilogue: bool = False):
        """Apply the experts' SGD update inside the backward pass: each projection is updated on a
        side stream as soon as its gradient is final (``ExpertParallelMoE.on_grad_ready``), beside
        the GEMMs that are still running.  ``None`` switches back to updating in ``sgd_step``.

        ``in_epilogue``: the experts are updated by their weight-gradient GEMMs themselves
        (``wgrad(update=...)``: no fp32 gradient is written or read back for an expert whose gradient is
        complete on this rank); the side-stream kernel then only covers the experts that have replicas on
        other ranks, whose gradients are reduced first.  Same arithmetic, same result."""
        self._fused_lr = lr
        moe = self.moe
        # shapes the CTA-pair weight-gradient kernel does not cover fall back to the stand-alone kernels
        in_epilogue = in_epilogue and all(gg.wgrad_update_supported(*self.pools.shape(n)) for n in ("gate", "up", "down"))
        moe.epilogue_lr = lr if (in_epilogue and lr is not None) else None
        if lr is None:
            moe.on_grad_ready = None
        elif moe.epilogue_lr is None:
            beside = 8 * moe._total_sms             # blocks that find room next to the GEMMs on the other streams
            moe.on_grad_ready = lambda n: gg.sgd_step(self.pools.local_weight(n), self.pools.local_grad(n), lr, num_blocks=beside)
        elif self.world == 1:
            moe.on_grad_ready = no_update           # no replicas: the epilogues have updated every expert
        else:
            moe.on_grad_ready = lambda n: gg.sgd_step_groups(self.pools.local_weight(n), self.pools.local_grad(n), lr,
                                                             moe._upd_mask, want=False, num_blocks=2 * moe._total_sms)

    def sgd_step(self, lr: float):
        if self.moe.on_grad_ready is None:
            names = ("down", "gate", "up")
            if self.moe.grads_pending is None:
                ps = self.pools
                ps.kept("sgd", lambda: gg.SgdMany([ps.local_weight(n) for n in names], [ps.local_grad(n) for n in names])).step(lr)
            else:
                for n in names:                  # ``up`` last: its cross-rank reduction may still be running, and these beside it
                    self.moe.wait_grads(n)
                    gg.sgd_step(self.pools.local_weight(n), self.pools.local_grad(n), lr, num_blocks=8 * self.moe._total_sms)
        else:
            assert lr == self._fused_lr, "the experts were already updated with another learning rate"
            self.moe.wait_grads()       # the last reduction and the update behind it may still be running
        with torch.no_grad():
            ps = [p for p in self.parameters() if p.grad is not None]
            if ps:
                torch._foreach_add_(ps, [p.grad.to(p.dtype) for p in ps], alpha=-lr)
                for p in ps:
                    p.grad = None

    def destroy(self):
        self.moe.wait_grads()        # nothing of this layer may still be queued on the comm stream
        self.pools.destroy()
        if self._own_buffer:
            self.buf.destroy()


def smoke_step() -> float:
    """One tiny forward + backward + SGD step on the current device (single rank)."""
    torch.manual_seed(0)
    blk = MoEBlock(CONFIGS["tiny"], num_sms=4)
    x = torch.randn(blk.cfg.S, blk.cfg.H, device="cuda").to(torch.bfloat16).requires_grad_(True)
    y = blk.forward(x)
    loss = (y.float() ** 2).mean()
    loss.backward()
    blk.sgd_step(1e-3)
    torch.cuda.synchronize()
    blk.buf.check()
    gg.check_status()
    assert x.grad is not None and torch.isfinite(x.grad.float()).all() and torch.isfinite(loss)
    v = float(loss)
    blk.destroy()
    return v
