"""Fused routing, its gradient and the block's single autograd node against torch operators, at the expert counts where
the kernel's lanes hold one more expert each."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,E,K", [(1, 1, 1), (7, 31, 8), (130, 32, 32), (64, 33, 2), (300, 65, 8), (96, 200, 5), (50, 512, 32)])
def test_route_matches_torch(S, E, K, cuda_device):
    from moonep_b200.ops import router as rt
    g = torch.Generator(device="cuda").manual_seed(S + E)
    # the bias makes the sums distinct: the order of equal ones is anybody's
    logits = torch.randn(S, E, device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(E, device="cuda", generator=g)
    w, topk, tpe, probs = rt.route(logits, bias, K, with_probs=True)
    lf = logits.clone().requires_grad_(True)
    pr = torch.softmax(lf.float() + bias, -1)
    wr, tr = torch.topk(pr, K, -1)
    wr = wr / wr.sum(-1, keepdim=True)
    dw = torch.randn(S, K, device="cuda", generator=g)
    wr.backward(dw)
    torch.cuda.synchronize()
    assert torch.equal(probs, pr) and torch.equal(topk.long(), tr) and torch.equal(w, wr)
    assert torch.equal(tpe.long(), torch.bincount(topk.flatten().long(), minlength=E))
    assert torch.equal(rt.route_bwd(probs, dw, topk), lf.grad)


@pytest.mark.parametrize("rows,n", [(1, 8), (130, 256), (33, 2056)])
def test_dense_swiglu_matches_torch(rows, n, cuda_device):
    from moonep_b200.ops import router as rt
    g = torch.Generator(device="cuda").manual_seed(n)
    gu = (torch.randn(rows, 2 * n, device="cuda", generator=g) * 3).to(torch.bfloat16).requires_grad_(True)
    d = torch.randn(rows, n, device="cuda", generator=g).to(torch.bfloat16)
    act = torch.nn.functional.silu(gu[:, :n]) * gu[:, n:]
    act.backward(d)
    assert torch.equal(rt.swiglu(gu.detach()), act) and torch.equal(rt.swiglu_bwd(d, gu.detach()), gu.grad)


def test_route_of_nans_names_existing_experts(cuda_device):
    from moonep_b200.ops import router as rt
    logits = torch.full((5, 48), float("nan"), device="cuda").to(torch.bfloat16)
    logits[1, :40] = 1.0          # one NaN makes every probability of its row NaN
    w, topk, tpe, _ = rt.route(logits, torch.zeros(48, device="cuda"), 8)
    t = topk.cpu()
    assert int(t.min()) >= 0 and int(t.max()) < 48 and all(len(set(r)) == 8 for r in t.tolist()) and int(tpe.sum()) == 40
    assert bool(torch.isnan(w).all())


@pytest.mark.parametrize("shared", [0, 1])
def test_block_node_matches_torch_operators(shared, cuda_device):
    from moonep_b200.models.moe_block import MoEBlock, MoEConfig
    cfg = MoEConfig("t", H=256, Hp=256, K=2, epn=4, shared_experts=shared, S=130)
    g = torch.Generator(device="cuda").manual_seed(2)
    x0 = (torch.randn(cfg.S, cfg.H, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
    dy = (torch.randn(cfg.S, cfg.H, device="cuda", generator=g) * 0.1).to(torch.bfloat16)
    got = []
    for fused in (True, False):
        blk = MoEBlock(cfg, num_sms=4, seed=3, router_skew=0.5)
        assert blk._fused_route
        blk._fused_route = fused
        x = x0.clone().requires_grad_(True)
        y = blk.forward(x)
        y.backward(dy)
        with torch.no_grad():
            yn = blk.forward(x0)
        torch.cuda.synchronize()
        blk.buf.check()
        assert torch.equal(yn, y)
        got.append([y.detach(), x.grad] + [p.grad for p in blk.parameters()] + [blk.pools.local_grad(n).clone() for n in ("gate", "up", "down")])
        blk.destroy()
    for i, (a, b) in enumerate(zip(*got)):
        if i == 1:      # the input gradient: its bf16 parts are added in another order, some with one rounding less (2^-9 for each)
            assert float((a.float() - b.float()).norm() / b.float().norm()) < 8e-3
        else:
            assert torch.equal(a, b), i
