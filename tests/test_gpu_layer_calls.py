"""Calls of a single-rank layer and block besides the plain training step: optional arguments, inputs of other forms,
contexts and pools that the caller has changed."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def make_block(shared=0, H=256, Hp=256, **kw):
    from moonep_b200.models.moe_block import MoEBlock, MoEConfig
    cfg = MoEConfig("t", H=H, Hp=Hp, K=2, epn=4, shared_experts=shared, S=130)
    return MoEBlock(cfg, num_sms=4, seed=3, router_skew=0.5, **kw)


def normal(shape, seed, scale=0.5):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


def test_layer_without_route_weights_is_unscaled(cuda_device):
    """Without route weights the rows are not scaled, whatever an earlier call has left in the buffers of the weights."""
    blk = make_block()
    x = normal((130, 256), 1)
    with torch.no_grad():
        w, topk, tpe = blk.route(x)
    ones = torch.ones_like(w)
    ref, _ = blk.moe.forward(x, ones, topk, tpe, need_backward=False)
    for keep in (False, True):
        blk.moe.forward(x, w * 3, topk, tpe, need_backward=keep)
        out, ctx = blk.moe.forward(x, None, topk, tpe, need_backward=False)
        torch.cuda.synchronize()
        assert ctx is None and torch.equal(out, ref)
    with pytest.raises(AssertionError, match="route weights"):
        blk.moe.forward(x, None, topk, tpe, need_backward=True)
    blk.destroy()


def test_backward_with_a_hook_refuses_a_bad_gradient(cuda_device):
    """With a hook between the launches the backward pass runs from Python; its gradient is checked there too."""
    blk = make_block()
    blk.moe.on_grad_ready = lambda n: None
    x, dy = normal((130, 256), 1), normal((130, 256), 2)
    with torch.no_grad():
        w, topk, tpe = blk.route(x)
    _, ctx = blk.moe.forward(x, w, topk, tpe)
    for bad in (dy[:1].expand(130, 256), dy.float(), dy[:129]):
        with pytest.raises(AssertionError, match="hidden_sh"):
            blk.moe.backward(ctx, bad)
    dx, _ = blk.moe.backward(ctx, dy)
    torch.cuda.synchronize()
    blk.buf.check()
    assert bool(torch.isfinite(dx.float()).all())
    blk.destroy()


def test_layer_uses_the_pools_it_has(cuda_device):
    """Weights and gradients are those of the layer's pools at the time of the call; pools without gradients have no
    backward pass, destroyed ones no pass at all."""
    from moonep_b200.pools import ExpertPools
    a, b = make_block(), make_block()
    for n in ("gate", "up", "down"):
        b.pools.local_weight(n).mul_(-0.5)
    x, dy = normal((130, 256), 1), normal((130, 256), 2)
    with torch.no_grad():
        w, topk, tpe = a.route(x)
    want, ctx = b.moe.forward(x, w, topk, tpe)
    b.moe.backward(ctx, dy)
    grads = [b.pools.local_grad(n).clone() for n in ("gate", "up", "down")]
    a.moe.forward(x, w, topk, tpe)
    own, a.moe.pools = a.moe.pools, b.pools
    out, ctx = a.moe.forward(x, w, topk, tpe)
    for n in ("gate", "up", "down"):
        b.pools.local_grad(n).zero_()
    a.moe.backward(ctx, dy)
    torch.cuda.synchronize()
    assert torch.equal(out, want)
    assert all(torch.equal(b.pools.local_grad(n), g) for n, g in zip(("gate", "up", "down"), grads))
    a.moe.pools = ExpertPools(4, (256, 256), (256, 256), (256, 256))
    _, ctx = a.moe.forward(x, w, topk, tpe)
    with pytest.raises(KeyError):
        a.moe.backward(ctx, dy)
    a.moe.pools = own
    own.destroy()
    for call in (lambda: a.moe.forward(x, w, topk, tpe), lambda: a.moe.backward(ctx, dy), lambda: a.sgd_step(0.1)):
        with pytest.raises(AttributeError):
            call()
    a.destroy()
    b.destroy()


@pytest.mark.parametrize("how", ["assign", "replace"])
def test_context_with_private_copies_outlives_the_next_forward_pass(how, cuda_device):
    """A caller with two batches in flight gives the first context copies of what the second pass overwrites."""
    import dataclasses
    from moonep_b200.moe_layer import MoEContext
    blk = make_block()
    xs, dy = [normal((130, 256), s) for s in (1, 2)], normal((130, 256), 3)
    with torch.no_grad():
        routes = [blk.route(x) for x in xs]
    names = ("gate", "up", "down")
    _, ctx = blk.moe.forward(xs[0], *routes[0])
    dx, dw = blk.moe.backward(ctx, dy)
    grads = [blk.pools.local_grad(n).clone() for n in names]
    for n in names:
        blk.pools.local_grad(n).zero_()
    _, ctx = blk.moe.forward(xs[0], *routes[0])
    assert isinstance(ctx, MoEContext)
    kept = {f: getattr(ctx, f).clone() for f in ("x", "w_nvs", "act", "gu")}
    if how == "replace":
        ctx = dataclasses.replace(ctx, **kept)
    else:
        for f, t in kept.items():
            setattr(ctx, f, t)
    blk.moe.forward(xs[1], *routes[1])
    dx2, dw2 = blk.moe.backward(ctx, dy)
    torch.cuda.synchronize()
    blk.buf.check()
    assert torch.equal(dx, dx2) and torch.equal(dw, dw2)
    assert all(torch.equal(blk.pools.local_grad(n), g) for n, g in zip(names, grads))
    blk.destroy()


def test_route_goes_through_transforms(cuda_device):
    """``MoEBlock.route`` alone is made of torch operators: leading dimensions, second derivatives, forward mode, autocast."""
    blk = make_block()
    x = normal((130, 256), 1)
    w, topk, tpe = blk.route(x)
    w3, topk3, tpe3 = blk.route(x.view(13, 10, 256))
    assert torch.equal(w3.flatten(0, 1), w) and torch.equal(topk3.flatten(0, 1), topk) and torch.equal(tpe3, tpe)
    xr = x.clone().requires_grad_(True)
    c = torch.linspace(-1, 1, 260, device="cuda").view(130, 2)
    (g,) = torch.autograd.grad((blk.route(xr)[0] * c).sum(), xr, create_graph=True)
    (g2,) = torch.autograd.grad(g.float().square().sum(), blk.router)
    assert bool(g2.abs().sum() > 0) and bool(torch.isfinite(g2.float()).all())
    with torch.autograd.forward_ad.dual_level():
        d = blk.route(torch.autograd.forward_ad.make_dual(x, x * 0.5))[0]
        assert torch.autograd.forward_ad.unpack_dual(d).tangent.shape == w.shape
    with torch.autocast("cuda", torch.float16):
        assert float((blk.route(x)[0] - w).detach().abs().max()) < 0.05
    blk.destroy()


@pytest.mark.parametrize("form", ["strided", "bf16", "per_token", "scalar", "parameter"])
def test_router_bias_of_any_form(form, cuda_device):
    """The bias is the caller's to replace: every form that torch adds to the logits counts, and one with a gradient gets it."""
    blk = make_block(shared=1)
    x, dy = normal((130, 256), 1), normal((130, 256), 2)
    g = torch.Generator(device="cuda").manual_seed(9)
    r = torch.randn(130, 8, device="cuda", generator=g)
    blk.router_bias = {"strided": r[0, ::2], "bf16": r[0, :4].bfloat16(), "per_token": r[:, :4],
                       "scalar": r[0, 0], "parameter": r[0, :4].clone().requires_grad_(True)}[form]
    got = []
    for fused in (True, False):
        blk._fused_route = fused
        xr = x.clone().requires_grad_(True)
        y = blk.forward(xr)
        y.backward(dy)
        got.append([y.detach(), xr.grad] + [p.grad for p in blk.parameters()] + [blk.router_bias.grad])
        for p in blk.parameters():
            p.grad = None
        blk.router_bias.grad = None
    assert (got[0][-1] is not None) == (form == "parameter")
    assert all((a is None and b is None) or torch.equal(a, b) for a, b in zip(*got))
    blk.destroy()


def test_block_under_autocast(cuda_device):
    """Autocast to bf16 changes nothing; to fp16 the router's logits are fp16, as the operators make them."""
    blk = make_block()
    x, dy = normal((130, 256), 1), normal((130, 256), 2)
    y0 = blk.forward(x)
    with torch.autocast("cuda", torch.bfloat16):
        assert torch.equal(blk.forward(x), y0)
    for grad in (True, False):
        with torch.autocast("cuda", torch.float16), torch.set_grad_enabled(grad):
            y = blk.forward(x)
    assert float((y.float() - y0.detach().float()).norm() / y0.detach().float().norm()) < 2e-2
    blk.destroy()


def test_frozen_router_and_input_freeze_the_experts(cuda_device):
    """Without a gradient for the input or the router the experts have no backward pass; the shared expert still has its own."""
    blk = make_block(shared=1)
    blk.router.requires_grad_(False)
    x, dy = normal((130, 256), 1), normal((130, 256), 2)
    got = []
    for fused in (True, False):
        blk._fused_route = fused
        for n in ("gate", "up", "down"):
            blk.pools.local_grad(n).fill_(7.0)
        blk.forward(x).backward(dy)
        torch.cuda.synchronize()
        assert all(bool((blk.pools.local_grad(n) == 7.0).all()) for n in ("gate", "up", "down"))
        assert blk.router.grad is None
        got.append([p.grad for p in blk.shared])
        for p in blk.shared:
            p.grad = None
    assert all(torch.equal(a, b) for a, b in zip(*got))
    blk.destroy()


@pytest.mark.parametrize("shared", [0, 1])
def test_second_derivatives_of_a_block(shared, cuda_device):
    """With ``create_graph`` the gradients can be differentiated as those of the operators can: the experts' part is a
    constant, router and shared expert are not."""
    blk = make_block(shared=shared)
    x, dy = normal((130, 256), 1), normal((130, 256), 2)
    got = []
    for fused in (True, False):
        blk._fused_route = fused
        xr, d = x.clone().requires_grad_(True), dy.clone().requires_grad_(True)
        ps = blk.parameters()
        first = torch.autograd.grad(blk.forward(xr), [xr] + ps, d, create_graph=True)
        second = torch.autograd.grad(sum(f.float().square().sum() for f in first), [xr] + ps + ([d] if shared else []))
        got.append([t.detach().float() for t in (*first, *second)])
    for i, (a, b) in enumerate(zip(*got)):      # bf16 operators on both sides: a few roundings of 2^-9
        assert float(b.norm()) > 0 and float((a - b).norm() / b.norm()) < 1.5e-2, i
    blk.destroy()


def test_native_calls_follow_the_launch_switch(cuda_device):
    """``Buffer.enable_pdl`` decides at every call how the layer's kernels are launched; the results are the same bits."""
    blk = make_block()
    x, dy = normal((130, 256), 1), normal((130, 256), 2)
    with torch.no_grad():
        route = blk.route(x)
    got = []
    for pdl in (True, False):
        blk.buf.enable_pdl = pdl
        y, ctx = blk.moe.forward(x, *route)
        assert blk.moe._native._args.pdl == pdl
        blk.moe._native._args.pdl = blk.moe._native._pdl = 2
        dx, dw = blk.moe.backward(ctx, dy)
        assert blk.moe._native._args.pdl == pdl
        got.append([y, dx, dw] + [blk.pools.local_grad(n).clone() for n in ("gate", "up", "down")])
    torch.cuda.synchronize()
    blk.buf.check()
    assert all(torch.equal(a, b) for a, b in zip(*got))
    blk.destroy()


@pytest.mark.parametrize("lr", [None, 0.05], ids=["gradients", "update"])
@pytest.mark.parametrize("ctas", [None, 6])
def test_native_passes_give_the_bits_of_single_launches(ctas, lr, cuda_device):
    """16 to 40 blocks of depth (more than a ring holds), 26 experts of which six are empty, more tiles than pairs: the native passes, whose GEMMs start
    early and share launches, against the same operators issued one by one from Python."""
    from moonep_b200.models.moe_block import MoEBlock, MoEConfig
    blk = MoEBlock(MoEConfig("t", H=1024, Hp=1280, K=4, epn=26, shared_experts=0, S=700), num_sms=4, seed=3)
    if lr is not None:
        blk.fuse_optimizer(lr, in_epilogue=True)
    g = torch.Generator(device="cuda").manual_seed(4)
    p = torch.rand(700, 26, device="cuda", generator=g) * torch.linspace(0.2, 2, 26, device="cuda")
    p[:, [0, 5, 6, 13, 20, 25]] = -1
    w, topk = torch.topk(p, 4, dim=1)
    topk = topk.to(torch.int32).contiguous()
    tpe = torch.bincount(topk.flatten().long(), minlength=26).to(torch.int32)
    x, dy = normal((700, 1024), 1), normal((700, 1024), 2)
    names, got = ("gate", "up", "down"), []
    before = [blk.pools.local_weight(n).clone() for n in names]
    native = blk.moe._native
    assert native is not None
    for use in (native, None):
        blk.moe._native = use
        if use is not None and ctas is not None:
            use._args.num_ctas = ctas
        for n, b in zip(names, before):
            blk.pools.local_weight(n).copy_(b)
            blk.pools.local_grad(n).fill_(7.0)
        infer, _ = blk.moe.forward(x, w, topk, tpe, need_backward=False)
        y, ctx = blk.moe.forward(x, w, topk, tpe)
        dx, dw = blk.moe.backward(ctx, dy)
        torch.cuda.synchronize()
        blk.buf.check()
        got.append([infer, y, dx, dw] + [blk.pools.local_grad(n).clone() for n in names] + [blk.pools.local_weight(n).clone() for n in names])
    assert all(torch.equal(a, b) for a, b in zip(*got))
    assert (lr is None) == all(torch.equal(a, b) for a, b in zip(got[0][7:], before))
    blk.destroy()


@pytest.mark.parametrize("flags", [False, True], ids=["local", "ranks"])
def test_a_layers_launches_say_which_groups_hold_rows(flags, cuda_device, monkeypatch):
    """With a hook the GEMMs are issued one by one; they name the experts and rows that the native passes name, forwards (without route weights) and
    backwards, and so does the code for several ranks."""
    from moonep_b200.ops import grouped_gemm as gg
    blk, seen, launch = make_block(), [], gg._launch

    def spy(mode, *a, **kw):
        seen.append((mode, kw.get("held")))
        return launch(mode, *a, **kw)
    monkeypatch.setattr(gg, "_launch", spy)
    if flags:
        blk.moe._local, blk.moe._native = False, None
    blk.moe.on_grad_ready = lambda n: None
    x, dy = normal((130, 256), 1), normal((130, 256), 2)
    with torch.no_grad():
        w, topk, tpe = blk.route(x)
    if not flags:
        blk.moe.forward(x, None, topk, tpe, need_backward=False)
    _, ctx = blk.moe.forward(x, w, topk, tpe)
    blk.moe.backward(ctx, dy)
    torch.cuda.synchronize()
    blk.buf.check()
    assert {m for m, _ in seen} >= {gg.GATE_UP, gg.DOWN, gg.DGRAD, gg.DGRAD_GU}
    assert {h for m, h in seen if m != gg.WGRAD} == {(4, 260)}
    native = blk.moe._native_layer()._args
    assert (native.E, native.S * native.K) == (4, 260)
    blk.destroy()


@pytest.mark.parametrize("last", ["weights", "counts"])
def test_queued_passes_see_what_the_kernel_before_wrote(last, cuda_device):
    """The GEMMs of a pass load weights and token counts while its dispatch still runs, and the dispatch sets itself up beside the kernel before: weights or
    counts written by the kernel right in front of a pass, passes queued without a pause, give what ordinary launches give with a pause behind everything."""
    from moonep_b200.models.moe_block import MoEBlock, MoEConfig
    names = ("gate", "up", "down")
    blk = MoEBlock(MoEConfig("t", H=512, Hp=512, K=4, epn=8, shared_experts=0, S=600), num_sms=4, seed=3, router_skew=0.5)
    assert blk.moe._native is not None
    xs, dys = [normal((600, 512), i) for i in (1, 2)], [normal((600, 512), i) for i in (3, 4)]
    with torch.no_grad():
        routes = [tuple(t.clone() for t in blk.route(x)) for x in xs]
    assert not torch.equal(routes[0][2], routes[1][2])
    base = {n: blk.pools.local_weight(n).clone() for n in names}
    zero = torch.zeros_like(routes[0][2])
    w, topk, tpe = (t.clone() for t in routes[0])
    x, dy = xs[0].clone(), dys[0].clone()

    def write(i, order):
        todo = {"inputs": lambda: [torch.add(a, 0, out=b) for a, b in zip((xs[i % 2], dys[i % 2], *routes[i % 2][:2]), (x, dy, w, topk))],
                "counts": lambda: torch.add(routes[i % 2][2], zero, out=tpe),
                "weights": lambda: [torch.mul(base[n], 1.0 + 0.125 * (i % 3), out=blk.pools.local_weight(n)) for n in order]}
        for k in sorted(todo, key=lambda k: k == last):
            todo[k]()

    def one(i, pause):
        write(i, ("up", "down", "gate"))               # gate/up is the first GEMM of a forward pass
        pause()
        out, _ = blk.moe.forward(x, w, topk, tpe, need_backward=False)
        pause()
        write(i + 1, ("down", "gate", "up"))
        pause()
        y, ctx = blk.moe.forward(x, w, topk, tpe)
        pause()
        for n in ("gate", "up", "down"):                # dgrad(down) the first of a backward pass
            torch.mul(base[n], 1.0 + 0.125 * ((i + 2) % 3), out=blk.pools.local_weight(n))
        pause()
        dx, dw = blk.moe.backward(ctx, dy)
        pause()
        return [out, y, dx, dw] + [blk.pools.local_grad(n).clone() for n in names]

    blk.buf.enable_pdl = False
    want = [one(i, torch.cuda.synchronize) for i in range(6)]
    blk.buf.enable_pdl = True
    got = [one(i % 6, lambda: None) for i in range(12)]
    torch.cuda.synchronize()
    blk.buf.check()
    for i, g in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(g, want[i % 6])), f"pass {i}"
    blk.destroy()
