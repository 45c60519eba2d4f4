"""The work this framework is used for on one GPU, as measurable cases.

Four kinds of use, each through the public entry points:

* ``exchange``: ``Buffer.dispatch`` and ``Buffer.combine`` around somebody else's expert computation -- the way an
  integrating training or serving framework calls the library.  Forward (a fresh plan, route weights travel along)
  or backward (the saved plan; the gradients of the route weights are gathered), on the communication shard itself
  (``zero_copy``) or with private copies.
* ``experts``: ``ExpertParallelMoE.forward(need_backward=False)``: an inference server that has its own router.
* ``block``: ``MoEBlock.forward`` under ``torch.no_grad``: inference with the block's router.
* ``step``: one training step of a ``MoEBlock``: forward, backward, SGD; launched from Python or replayed as a
  captured step (``GraphedSteps``), the experts' update in the weight-gradient GEMMs or behind the backward pass.

Shapes are those of ``moonep_b200.models.CONFIGS`` (deepseek_v3, kimi_k2, qwen3_30b_a3b, tiny), the benchmark's, and
odd ones between them.  Everything is bf16 with fp32 gradients and route weights, which is all the framework computes in.
"""

import math

import torch

from moonep_b200 import Buffer, routing
from moonep_b200.models.moe_block import MoEBlock, MoEConfig
from moonep_b200.moe_layer import ExpertParallelMoE
from moonep_b200.pools import ExpertPools
from moonep_b200.utils import GraphedSteps

LR = 0.02


def listed():
    return [
        # a decode batch of 64 sequences, the integrator's own experts: launches and host work
        dict(name="exchange_decode_64", kind="exchange", S=64, H=2048, K=8, E=16, pad=128, skew=0.4, backward=False, zero_copy=True),
        # the benchmark's layer (DeepSeek-V3 shape), forward: plan, scatter, gather
        dict(name="exchange_train_4096", kind="exchange", S=4096, H=7168, K=8, E=32, pad=128, skew=0.4, backward=False, zero_copy=True),
        # the same layer's backward pass: saved plan, gradients of the route weights
        dict(name="exchange_back_4096", kind="exchange", S=4096, H=7168, K=8, E=32, pad=128, skew=0.4, backward=True, zero_copy=True),
        # a ragged batch with many experts, small padding and the default private copies
        dict(name="exchange_odd_3001", kind="exchange", S=3001, H=4096, K=6, E=60, pad=16, skew=0.8, backward=False, zero_copy=False),
        # decode step of a small MoE (Qwen3-30B-A3B layer): few tokens for each expert
        dict(name="decode_64_small", kind="experts", S=64, H=2048, Hp=768, K=8, E=16, skew=0.4),
        # decode step of a large MoE: every expert's weights are streamed for a handful of tokens
        dict(name="decode_256_large", kind="experts", S=256, H=7168, Hp=2048, K=8, E=32, skew=0.4),
        # prefill chunk of odd length, own router
        dict(name="prefill_odd_1531", kind="experts", S=1531, H=2048, Hp=768, K=8, E=16, skew=0.8),
        # prefill of a full chunk through the block
        dict(name="prefill_4096_large", kind="block", S=4096, H=7168, Hp=2048, K=8, E=32, skew=0.5, shared=0),
        # training of a tiny model: one step is mostly launches
        dict(name="step_tiny_128", kind="step", S=128, H=256, Hp=256, K=2, E=2, skew=0.5, shared=1, graph=False, epilogue=False),
        # training of a Qwen3-30B-A3B layer, captured step
        dict(name="step_small_8192", kind="step", S=8192, H=2048, Hp=768, K=8, E=16, skew=0.5, shared=0, graph=True, epilogue=True),
        # the benchmark's training step (DeepSeek-V3 layer), captured step
        dict(name="step_large_4096", kind="step", S=4096, H=7168, Hp=2048, K=8, E=32, skew=0.5, shared=0, graph=True, epilogue=True),
        # an odd microbatch of a Kimi-K2 layer with its shared expert; gradients are kept, the optimizer follows
        dict(name="step_odd_1531", kind="step", S=1531, H=7168, Hp=2048, K=8, E=48, skew=0.8, shared=1, graph=False, epilogue=False),
    ]


def _spread(rng, lo, hi):
    """An integer in [lo, hi], even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _taken(H, E):
    """Whether ``Buffer.dispatch`` takes the size: a few row lengths fill its ring of rows in shared memory so evenly
    that the tables behind it find no room, and the call is refused."""
    return 12 * H * min(8, 180 * 1024 // (12 * H)) + 48 * 1024 + 16 * E + 8 <= 226 * 1024


def draw(rng):
    kind = rng.choice(["exchange", "exchange", "experts", "block", "step", "step"])
    while True:
        if kind == "exchange":
            K = rng.randint(1, 8)
            c = dict(kind=kind, S=_spread(rng, 16, 8192), H=8 * _spread(rng, 64, 896), K=K, E=max(K, _spread(rng, 8, 256)),
                     pad=rng.choice([1, 16, 128]), skew=round(rng.uniform(0.1, 1.5), 3), backward=rng.random() < 0.5, zero_copy=rng.random() < 0.5)
            if c["S"] * c["K"] * c["H"] <= 4096 * 8 * 7168 and _taken(c["H"], c["E"]):
                return c
            continue
        K = rng.randint(2, 8)
        c = dict(kind=kind, S=_spread(rng, 64 if kind == "step" else 1, 8192), H=256 * _spread(rng, 2, 28), Hp=256 * _spread(rng, 1, 8), K=K,
                 E=max(K, _spread(rng, 4, 48)), skew=round(rng.uniform(0.2, 1.2), 3))
        if kind != "experts":
            c["shared"] = rng.randint(0, 1)
        if kind == "step":
            c.update(graph=rng.random() < 0.5, epilogue=rng.random() < 0.5)
        small = c["E"] * c["H"] * c["Hp"] <= 32 * 7168 * 2048
        if small and c["S"] * (c["K"] + c.get("shared", 0)) * c["H"] * c["Hp"] <= 4096 * 8 * 7168 * 2048:
            return c


class _State:
    """What one prepared program holds; gives the communication buffers and pools back when it goes."""

    def __init__(self, case):
        self.case, self.owned = case, []

    def __del__(self):
        for o in self.owned:
            o.destroy()


def _routing(case, seed):
    c = case
    topk, w, tpe = routing.softmax_topk(c["S"], c["K"], c["E"], c["skew"], seed, 0, device="cuda")
    return topk, w, tpe


def _normal(gen, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=gen) * scale).to(torch.bfloat16)


def _block(case, seed):
    c = case
    cfg = MoEConfig("case", c["H"], c["Hp"], c["K"], c["E"], shared_experts=c["shared"], S=c["S"])
    return MoEBlock(cfg, seed=seed, router_skew=c["skew"])


def prepare(case, seed):
    c, s = case, _State(case)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if c["kind"] == "exchange":
        s.buf = Buffer(c["S"], c["H"], c["K"], c["E"], 1, token_padding=c["pad"])
        s.owned = [s.buf]
        s.topk, s.w, s.tpe = _routing(c, seed)
        s.x = _normal(gen, c["S"], c["H"])
        _, _, _, s.plan = s.buf.dispatch(s.x, s.w, s.topk, s.tpe, zero_copy=True, router_weights_zero_copy=True)   # the forward pass's
        if c["backward"]:      # what the expert computation of the backward pass leaves: d(route weight) for each row
            s.dw = s.buf.router_weight_buffer_view
            s.dw.copy_(torch.randn(s.dw.shape, device="cuda", generator=gen))
            if not c["zero_copy"]:
                s.dw = s.dw.clone()
        return s
    if c["kind"] == "experts":
        s.buf = Buffer(c["S"], c["H"], c["K"], c["E"], 1)
        s.pools = ExpertPools(c["E"], (c["H"], c["Hp"]), (c["H"], c["Hp"]), (c["Hp"], c["H"]))
        s.owned = [s.pools, s.buf]
        for n in ("gate", "up", "down"):
            w = s.pools.local_weight(n)
            for e in range(c["E"]):
                w[e].copy_(torch.randn(w[e].shape, device="cuda", generator=gen) * 0.02)
        s.layer = ExpertParallelMoE(s.buf, s.pools)
        s.topk, s.w, s.tpe = _routing(c, seed)
        s.x = _normal(gen, c["S"], c["H"])
        return s
    s.blk = _block(c, seed)
    s.owned = [s.blk]
    s.x = _normal(gen, c["S"], c["H"])
    if c["kind"] == "block":
        return s
    if c["epilogue"]:
        s.blk.fuse_optimizer(LR, in_epilogue=True)
    s.graphed = None
    if c["graph"]:             # as a training loop does: some steps from Python, then the captured one
        for _ in range(3):
            _step(s, s.x.detach())
        torch.cuda.synchronize()
        s.graphed = GraphedSteps(lambda x: _step(s, x), [s.x])
    return s


def _step(s, x):
    """Forward, backward, SGD on the loss sum(y^2) / 2S, whose gradient is y / S; returns the loss."""
    x.requires_grad_(True)
    y = s.blk.forward(x)
    d = y.detach() * (1.0 / s.case["S"])
    loss = 0.5 * s.case["S"] * torch.linalg.vector_norm(d.reshape(-1), dtype=torch.float32).square()
    y.backward(d)
    s.blk.sgd_step(LR)
    s.y, s.dx = y.detach(), x.grad
    x.grad = None
    return loss


def _updated(s):
    out = dict(y=s.y, dx=s.dx)
    out.update({n: s.blk.pools.local_weight(n) for n in ("gate", "up", "down")})
    out.update({"param%d" % i: p.detach() for i, p in enumerate(s.blk.parameters())})
    if not s.case["epilogue"]:
        out.update({"d" + n: s.blk.pools.local_grad(n) for n in ("gate", "up", "down")})
    return out


def run(s):
    c = s.case
    if c["kind"] == "exchange":
        z = c["zero_copy"]
        n = c["S"] * c["K"]    # that many rows are in use at least; those behind the last expert's are no result
        if c["backward"]:
            h, _, _, _ = s.buf.dispatch(s.x, plan=s.plan, zero_copy=z)
            out, w, _ = s.buf.combine(plan=s.plan, hidden_nvsh=h, route_weights_nvs=s.dw, zero_copy=z, router_weights_zero_copy=z)
            got = dict(out=out, w=w)
        else:
            h, w, cu, plan = s.buf.dispatch(s.x, s.w, s.topk, s.tpe, zero_copy=z, router_weights_zero_copy=z)
            out, _, _ = s.buf.combine(plan=plan, hidden_nvsh=h, zero_copy=z)
            got = dict(out=out, w=w[:n], cu=cu, dst=plan.dst, fill=plan.zero_fill_ranges)
        if not z:              # on the shard itself the combine has used the rows up
            got["rows"] = h[:n]
        return got
    if c["kind"] == "experts":
        out, _ = s.layer.forward(s.x, s.w, s.topk, s.tpe, need_backward=False)
        return out
    if c["kind"] == "block":
        with torch.no_grad():
            return s.blk.forward(s.x)
    if s.graphed is not None:
        s.graphed.replay(0)
        loss = s.graphed.losses[0]
    else:
        loss = _step(s, s.x.detach())
    return dict(_updated(s), loss=loss)


def work(case):
    c = case
    n = c["S"] * c["K"]
    if c["kind"] == "exchange":     # dispatch: tokens read, rows written; combine: rows read, sums written; index tables
        return dict(bytes=2.0 * 2 * c["H"] * (c["S"] + n) + 16.0 * n, flops=1.0 * n * c["H"])
    used = c["E"] * (1.0 - (1.0 - min(1.0, c["K"] / c["E"])) ** c["S"])     # experts that get a token
    expert, shared, router = 3.0 * c["H"] * c["Hp"], 3.0 * c["H"] * c["Hp"] * c.get("shared", 0), 0.0
    if c["kind"] != "experts":
        router = 1.0 * c["H"] * c["E"]
    params = used * expert + shared + router
    flops = 2.0 * (n * expert + c["S"] * (shared + router))
    if c["kind"] != "step":
        return dict(bytes=2.0 * params + 2.0 * 2 * c["S"] * c["H"], flops=flops)
    grads = 0.0 if c["epilogue"] else 4.0 * c["E"] * expert
    return dict(bytes=4.0 * params + grads + 3.0 * 2 * c["S"] * c["H"], flops=3.0 * flops)


def tolerance(case):
    # bf16 results of sums in fp32; whole numbers (plan, cu_seqlens) have one right value
    return {"rel": 1e-2, "max": 0.2}
