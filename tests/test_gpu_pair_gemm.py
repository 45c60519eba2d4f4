"""CTA-pair grouped GEMMs with a table of padding rows: groups whose real sizes lie around the kernels' steps (32-token
units, 128-row halves, 256-row tiles, evenly shared tiles above that), against an fp32 reference."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = {"units": [1, 31, 32, 33, 64, 65, 0, 127], "tiles": [128, 129, 255, 256, 257, 0, 300, 511], "large": [513, 1000, 0, 1281]}


def _rel(a, b):
    return float((a.float() - b.float()).norm() / (b.float().norm() + 1e-12))


@pytest.mark.parametrize("dynamic", [False, True], ids=["static", "dynamic"])
@pytest.mark.parametrize("kn", [(256, 256), (320, 512)], ids=["256x256", "320x512"])
@pytest.mark.parametrize("sizes", list(SIZES))
def test_padding_rows_are_skipped(sizes, kn, dynamic, cuda_device):
    from moonep_b200.ops import grouped_gemm as gg
    n = SIZES[sizes]
    (K, N), G = kn, len(n)
    padded = [(r + 127) // 128 * 128 for r in n]
    ends = torch.tensor(padded).cumsum(0)
    cu = ends.to(torch.int32).cuda()
    pad = torch.tensor([[int(e) - p + r, p - r] if p > r else [0, 0] for r, p, e in zip(n, padded, ends)], dtype=torch.int32).cuda()
    g = torch.Generator(device="cuda").manual_seed(1)
    rows = int(ends[-1]) + 128
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    x, wg, wu, wd, scale = bf(rows, K, sc=0.5), bf(G, K, N, sc=0.05), bf(G, K, N, sc=0.05), bf(G, N, 256, sc=0.05), torch.rand(rows, device="cuda", generator=g) + 0.5
    full = lambda c, dt=torch.bfloat16: torch.full((rows, c), float("nan"), dtype=dt, device="cuda")    # noqa: E731
    act, gu, y, dA = full(N), full(2 * N), full(256), full(N)
    kw = dict(pad=pad, dynamic=dynamic)
    gg.gate_up(x, wg, wu, cu, act, gu, row_scale=scale, **kw)
    gg.down(act, wd, cu, y, row_scale=scale, **kw)
    if N % 256 == 0:
        gg.dgrad(y, wd, cu, dA, **kw)
    dW = torch.full((G, 256, N), 7.0, device="cuda")
    torch.cuda.synchronize()
    gg.check_status()
    written = torch.zeros(rows, dtype=torch.bool)
    for i, (r, p, e) in enumerate(zip(n, padded, ends.tolist())):
        a = e - p
        written[a:a + (r + 31) // 32 * 32] = True
        if r == 0:
            continue
        s = slice(a, a + r)
        gr, ur = x[s].float() @ wg[i].float(), x[s].float() @ wu[i].float()
        # bf16 results of fp32 sums: half a bf16 ulp is 2^-9
        assert _rel(gu[s, :N], gr) < 4e-3 and _rel(gu[s, N:], ur) < 4e-3, f"group {i} ({r} rows): pre-activations"
        assert _rel(act[s], torch.nn.functional.silu(gr) * ur * scale[s, None]) < 4e-3, f"group {i} ({r} rows): swiglu"
        assert _rel(y[s], (act[s].float() @ wd[i].float()) * scale[s, None]) < 4e-3, f"group {i} ({r} rows): down"
        assert _rel(dA[s], y[s].float() @ wd[i].float().T) < 4e-3, f"group {i} ({r} rows): dgrad"
    for t in (act, gu, y, dA):
        nan = torch.isnan(t.float()).any(dim=1).cpu()
        assert not bool(nan[written].any()) and bool(nan[~written].all()), "rows behind the 32-row step were written"
    # weight gradients read no row behind the step (NaN there); the rows up to it must be zero on one side, as a
    # dispatch leaves them
    for i, (r, p, e) in enumerate(zip(n, padded, ends.tolist())):
        y[e - p + r:e - p + (r + 31) // 32 * 32] = 0
    gg.wgrad(y, act, cu, dW, zero_empty_below=G, **kw)
    torch.cuda.synchronize()
    gg.check_status()
    for i, (r, p, e) in enumerate(zip(n, padded, ends.tolist())):
        ref = y[e - p:e - p + r].float().T @ act[e - p:e - p + r].float()
        assert torch.equal(dW[i], torch.zeros_like(dW[i])) if r == 0 else _rel(dW[i], ref) < 1e-4, f"group {i} ({r} rows): wgrad"


@pytest.mark.parametrize("dynamic", [False, True], ids=["static", "dynamic"])
def test_large_groups_are_walked_in_bands(dynamic, cuda_device):
    """4096 deep, a group of more than 18 token tiles (36 MB) is taken in bands of at most 8: the last size below the line,
    the first above it, bands of unequal size, between small groups."""
    from moonep_b200.ops import grouped_gemm as gg
    K, N, n = 4096, 512, [128, 4608, 4736, 0, 6272, 256]
    cu = torch.tensor(n).cumsum(0).to(torch.int32).cuda()
    g = torch.Generator(device="cuda").manual_seed(2)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    x, w, wu, wt = bf(sum(n), K), bf(len(n), K, N, sc=0.02), bf(len(n), K, N, sc=0.02), bf(len(n), N, K, sc=0.02)
    full = lambda c: torch.full((sum(n), c), float("nan"), dtype=torch.bfloat16, device="cuda")    # noqa: E731
    act, gu, y, dA = full(N), full(2 * N), full(N), full(N)
    gg.gate_up(x, w, wu, cu, act, gu, dynamic=dynamic)
    gg.down(x, w, cu, y, dynamic=dynamic)
    gg.dgrad(x, wt, cu, dA, dynamic=dynamic)
    torch.cuda.synchronize()
    gg.check_status()
    a = 0
    for i, r in enumerate(n):
        if r:
            s = slice(a, a + r)
            for got, ref in ((gu[s, :N], w[i]), (gu[s, N:], wu[i]), (y[s], w[i]), (dA[s], wt[i].T)):
                # bf16 results of fp32 sums: half a bf16 ulp is 2^-9; rows one by one, so that a misplaced tile shows
                d, f = x[s].float() @ ref.float(), got.float()
                assert bool(((f - d).norm(dim=1) < 4e-3 * d.norm(dim=1)).all()), f"group {i} ({r} rows)"
        a += r


@pytest.mark.parametrize("M", [2048, 2816, 4352])
def test_weight_gradient_of_large_groups(M, cuda_device):
    """Above 9 M elements of x in a group on average the row blocks go in bands of at most 8: 8 in one, 6 + 5, 6 + 6 + 5."""
    from moonep_b200.ops import grouped_gemm as gg
    n, N = [6400, 128, 0, 14976], 512
    cu = torch.tensor(n).cumsum(0).to(torch.int32).cuda()
    g = torch.Generator(device="cuda").manual_seed(3)
    x, dy = ((torch.randn(sum(n), c, device="cuda", generator=g)).to(torch.bfloat16) for c in (M, N))
    dW = torch.full((len(n), M, N), 7.0, device="cuda")
    gg.wgrad(x, dy, cu, dW, zero_empty_below=len(n))
    torch.cuda.synchronize()
    gg.check_status()
    a = 0
    for i, r in enumerate(n):
        ref = x[a:a + r].float().T @ dy[a:a + r].float()
        # fp32 sums of the same products in another order; 256 x 256 blocks one by one, so that a misplaced tile shows
        for got, want in zip(dW[i].unfold(0, 256, 256).unfold(1, 256, 256).flatten(0, 1), ref.unfold(0, 256, 256).unfold(1, 256, 256).flatten(0, 1)):
            assert bool((got == 0).all()) if r == 0 else _rel(got, want) < 1e-4, f"group {i} ({r} rows)"
        a += r


def test_swiglu_epilogue_of_extreme_pre_activations(cuda_device):
    """Gate values outside the epilogue's branch-free range (|g| >= 60, tiny) and zeros beside ordinary ones: with
    a unit gate weight and an up weight of one the activation is g / (1 + exp(-g)) * 1, rounded to bf16 once."""
    from moonep_b200.ops import grouped_gemm as gg
    vals = [0.0, -0.0, 1.0, -1.0, 59.9, -59.9, 60.0, -60.0, 87.0, -87.0, 88.5, -88.5, 104.0, -104.0, 1e30, -1e30, 3e38, -3e38,
            1e-30, -1e-30, 1e-37, -1e-37, 2.5, -2.5, float("inf"), float("-inf"), float("nan"), 17.0, -17.0, 30.0, -30.0, 0.5]
    rows, K, N = 128, 64, 128
    x = torch.zeros(rows, K, device="cuda")
    v = torch.tensor(vals, device="cuda").repeat(4)
    x[:, 1] = 1.0
    finite = torch.isfinite(v)
    wg, wu = torch.zeros(1, K, N, device="cuda"), torch.zeros(1, K, N, device="cuda")
    wg[0, 0] = 1.0                       # gate = x[:, 0] in every column
    wu[0, 1] = 1.0                       # up = 1
    x[:, 0] = torch.where(finite, v, torch.zeros_like(v))
    cu = torch.tensor([rows], dtype=torch.int32, device="cuda")
    x, wg, wu = x.to(torch.bfloat16), wg.to(torch.bfloat16), wu.to(torch.bfloat16)
    act, gu = torch.empty(rows, N, dtype=torch.bfloat16, device="cuda"), torch.empty(rows, 2 * N, dtype=torch.bfloat16, device="cuda")
    gg.gate_up(x, wg, wu, cu, act, gu)
    torch.cuda.synchronize()
    gg.check_status()
    g = x[:, 0].double()
    ref = (g / (1.0 + torch.exp(-g)))[:, None].expand(rows, N)
    assert torch.equal(gu[:, :N], x[:, :1].expand(rows, N)) and bool((gu[:, N:] == 1).all())
    # exp's two ulp and one bf16 rounding: within one bf16 ulp (2^-7); below the smallest normal number fp32 exp ends in zero
    assert bool(((act.double() - ref).abs() <= 2.0 ** -7 * ref.abs() + 2e-36).all())


@pytest.mark.parametrize("split", [(33, 115), (1, 147), (31, 33, 84)], ids=str)
def test_launches_of_odd_size_share_a_ticket(split, cuda_device, monkeypatch):
    """The launches on one ticket divide the tiles among them whatever their sizes, and leave the counter clean."""
    from moonep_b200.ops import grouped_gemm as gg
    monkeypatch.setenv("MOONEP_GEMM_2CTA", "1")
    K, N, n = 256, 512, [256, 0, 640, 128]
    cu = torch.tensor(n).cumsum(0).to(torch.int32).cuda()
    g = torch.Generator(device="cuda").manual_seed(4)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    x, w, wu, wt = bf(sum(n), K), bf(4, K, N, sc=0.05), bf(4, K, N, sc=0.05), bf(4, N, K, sc=0.05)
    dy = bf(sum(n), N)
    calls = {"gate_up": (lambda o, **kw: gg.gate_up(x, w, wu, cu, o, **kw), (sum(n), N), torch.bfloat16),
             "down": (lambda o, **kw: gg.down(x, w, cu, o, **kw), (sum(n), N), torch.bfloat16),
             "dgrad": (lambda o, **kw: gg.dgrad(x, wt, cu, o, **kw), (sum(n), N), torch.bfloat16),
             "wgrad": (lambda o, **kw: gg.wgrad(x, dy, cu, o, zero_empty_below=4, **kw), (4, K, N), torch.float32)}
    for name, (call, shape, dt) in calls.items():
        want, got = torch.full(shape, 7.0, dtype=dt, device="cuda"), torch.full(shape, 9.0, dtype=dt, device="cuda")
        call(want)
        tk = gg.Ticket(x.device, sum(split))
        for c in split:
            call(got, num_ctas=c, ticket=tk)
        torch.cuda.synchronize()
        gg.check_status()
        assert torch.equal(got, want), name
        assert not bool(gg._sched_cache[gg._dev_index(x.device)][0].any()), f"{name}: the counter was left behind"


@pytest.mark.parametrize("G,r,K,N", [(1, 128, 64, 256), (16, 384, 2048, 768), (4, 128, 2048, 768), (3, 1152, 256, 512)])
def test_both_kernels_give_the_same_bits(G, r, K, N, cuda_device, monkeypatch):
    """Left alone, a GEMM runs on single CTAs or on pairs: the sizes lie on both sides of the rule."""
    from moonep_b200.ops import grouped_gemm as gg
    cu = (torch.arange(1, G + 1, device="cuda") * r).to(torch.int32)
    g = torch.Generator(device="cuda").manual_seed(8)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    x, x2, w, wu, scale = bf(G * r, K), bf(G * r, 2 * K), bf(G, K, N, sc=0.05), bf(G, K, N, sc=0.05), torch.rand(G * r, device="cuda", generator=g)
    got = []
    for env in (None, "0", "1"):
        monkeypatch.delenv("MOONEP_GEMM_2CTA", raising=False) if env is None else monkeypatch.setenv("MOONEP_GEMM_2CTA", env)
        act, gu, y, dA, dx = (torch.full((G * r, c), float("nan"), dtype=torch.bfloat16, device="cuda") for c in (N, 2 * N, N, N, N))
        gg.gate_up(x, w, wu, cu, act, gu, row_scale=scale)
        gg.down(x, w, cu, y, row_scale=scale)
        gg.dgrad(x, w.view(G, N, K), cu, dA)
        gg.dgrad_gate_up(x2, w.view(G, N, K), wu.view(G, N, K), cu, dx)
        torch.cuda.synchronize()
        gg.check_status()
        got.append((act, gu, y, dA, dx))
    assert all(torch.equal(a, b) and torch.equal(a, c) for a, b, c in zip(*got))


@pytest.mark.parametrize("pairs", ["0", "1"], ids=["single", "pairs"])
def test_pushed_rows_and_flagged_tiles_on_both_kernels(pairs, cuda_device, monkeypatch):
    """The push epilogues and the tile flags, at sizes that the rule gives to one kernel only, on either of them."""
    from test_gpu_comm import test_push_combine_matches_sum_of_rows
    from test_gpu_flags import test_gemm_consumes_tiles_while_dispatch_runs
    monkeypatch.setenv("MOONEP_GEMM_2CTA", pairs)
    test_push_combine_matches_sum_of_rows(4, cuda_device)
    test_gemm_consumes_tiles_while_dispatch_runs(2, "dgrad", cuda_device)
    test_gemm_consumes_tiles_while_dispatch_runs(4, "gate_up", cuda_device)


@pytest.mark.parametrize("H,E", [(256, 4), (768, 16)], ids=["small", "streamed"])
@pytest.mark.parametrize("pairs", ["0", "1"], ids=["single", "pairs"])
def test_dgrad_pushes_rows_and_their_scalars(pairs, H, E, cuda_device, monkeypatch):
    """dgrad(gate/up) with identity weights: every dispatched row and its scalar go back to the token that it came from."""
    from moonep_b200 import Buffer, routing
    from moonep_b200.ops import grouped_gemm as gg
    monkeypatch.setenv("MOONEP_GEMM_2CTA", pairs)
    S, K = 96, 4
    topk, w, tpe = routing.softmax_topk(S, K, E, 1.0, 5, 0, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(7)
    x = torch.randn(S, H, device="cuda", generator=g).to(torch.bfloat16)
    buf = Buffer(S, H, K, E, 1, push_combine=True)
    h, wn, cu, _ = buf.dispatch(x, w, topk, tpe, zero_copy=True, router_weights_zero_copy=True)
    eye, zero = torch.eye(H, dtype=torch.bfloat16, device="cuda").repeat(2 * E, 1, 1).contiguous(), torch.zeros(2 * E, H, H, dtype=torch.bfloat16, device="cuda")
    dgu = torch.cat([h, torch.zeros_like(h)], 1).contiguous()
    dgu[int(cu[-1]):] = 0
    gg.dgrad_gate_up(dgu, eye, zero, cu, torch.empty_like(h), push=buf.push_target(), push_w=wn)
    out, ow, _ = buf.combine_pushed(want_weights=True)
    torch.cuda.synchronize()
    buf.check()
    gg.check_status()
    assert torch.equal(out, (x.float() * K).to(torch.bfloat16)) and torch.equal(ow, w)
    buf.destroy()


@pytest.mark.parametrize("accumulate", [False, True])
def test_two_weight_gradients_in_one_launch(accumulate, cuda_device):
    """The halves of dy's columns give two matrices: the same bits as two launches, with an update in the epilogue for some groups,
    groups without tokens and a group whose k-blocks do not fill the last one."""
    from moonep_b200.ops import grouped_gemm as gg
    n, M, N = [128, 0, 384, 256, 0], 512, 256
    cu = torch.tensor(n).cumsum(0).to(torch.int32).cuda()
    g = torch.Generator(device="cuda").manual_seed(5)
    x, dy = ((torch.randn(sum(n), c, device="cuda", generator=g)).to(torch.bfloat16) for c in (M, 2 * N))
    mask = None if accumulate else torch.tensor([1, 1, 0, 1, 0], dtype=torch.int32, device="cuda")
    w0 = [(torch.randn(len(n), M, N, device="cuda", generator=g)).to(torch.bfloat16) for _ in range(2)]
    runs = []
    for together in (False, True):
        out, w = [torch.full((len(n), M, N), 7.0, device="cuda") for _ in range(2)], [t.clone() for t in w0]
        up = lambda i: None if accumulate else (w[i], 0.1, mask)     # noqa: E731
        kw = dict(accumulate=accumulate, zero_empty_below=4)
        if together:
            gg.wgrad(x, dy, cu, out[0], update=up(0), out_b=out[1], update_b=None if accumulate else w[1], **kw)
        else:
            gg.wgrad(x, dy[:, :N], cu, out[0], update=up(0), **kw)
            gg.wgrad(x, dy[:, N:], cu, out[1], update=up(1), **kw)
        torch.cuda.synchronize()
        gg.check_status()
        runs.append(out + w)
    for a, b in zip(*runs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("blocks", [None, 1, 5])
def test_sgd_at_the_edges_of_its_chunks(blocks, cuda_device):
    """Chunks are 8192 parameters. One rounding to fp32 and one to bf16: what double precision gives for a rate with few bits."""
    from moonep_b200.ops import grouped_gemm as gg
    sizes = [8, 2040, 2048, 8184, 8192, 8200, 3 * 8192 + 2056, 40 * 8192]
    g = torch.Generator(device="cuda").manual_seed(6)
    ps = [(torch.randn(n, device="cuda", generator=g)).to(torch.bfloat16) for n in sizes]
    gs = [torch.randn(n, device="cuda", generator=g) for n in sizes]
    want = [(p.double() - 0.125 * d.double()).float().to(torch.bfloat16) for p, d in zip(ps, gs)]
    for p, d, w in zip(ps, gs, want):
        a = p.clone()
        gg.sgd_step(a, d, 0.125, num_blocks=blocks)
        assert torch.equal(a, w), f"{p.numel()} parameters"
    many = [p.clone() for p in ps]
    for i in (0, 4):
        gg.SgdMany(many[i:i + 4], gs[i:i + 4], num_blocks=blocks).step(0.125)
    assert all(torch.equal(a, w) for a, w in zip(many, want))
    p, d = (torch.cat([t[5][:8200]] * 3).view(3, -1) for t in (ps, gs))
    mask = torch.tensor([1, 0, 1], dtype=torch.int32, device="cuda")
    got = p.clone()
    gg.sgd_step_groups(got, d, 0.125, mask, True, num_blocks=blocks)
    assert torch.equal(got[0], want[5]) and torch.equal(got[1], p[1]) and torch.equal(got[2], want[5])


@pytest.mark.parametrize("ctas", [2, 12, 148])
def test_weight_gradients_of_many_uneven_groups(ctas, cuda_device):
    """189 groups of 0 to 512 rows, larger ones first in the tile list, every other round backwards: the bits of each group alone. What a
    CTA orders its list with must not reach the operands of its first tile."""
    from moonep_b200.ops import grouped_gemm as gg
    n, M, N = [128 * (7 * i * i % 6) for i in range(189)], 256, 256
    cu = torch.tensor(n).cumsum(0).to(torch.int32).cuda()
    g = torch.Generator(device="cuda").manual_seed(9)
    x, dy = ((torch.randn(sum(n), c, device="cuda", generator=g)).to(torch.bfloat16) for c in (M, N))
    full = lambda: torch.full((len(n), M, N), 7.0, device="cuda")     # noqa: E731
    want = full()
    for i in range(len(n)):
        gg.wgrad(x, dy, cu, want, zero_empty_below=100, groups=(i, i + 1))
    for dynamic in (False, True):
        got = full()
        gg.wgrad(x, dy, cu, got, zero_empty_below=100, num_ctas=ctas, dynamic=dynamic)
        torch.cuda.synchronize()
        gg.check_status()
        assert torch.equal(got, want)
    a = sum(n[:5])
    assert n[5] and _rel(want[5], x[a:a + n[5]].float().T @ dy[a:a + n[5]].float()) < 1e-5       # fp32 sums of the same products


class _Early:
    """Launches made inside set themselves up while the kernel before them runs, as those of a layer's native pass do, with the given limit of
    their waits."""

    def __init__(self, monkeypatch, budget_ns=None, **fields):
        self.mp, self.fields = monkeypatch, dict(early=1, pdl=1, **fields)
        if budget_ns is not None:
            self.fields["budget_ns"] = budget_ns

    def __enter__(self):
        from moonep_b200.ops import grouped_gemm as gg
        new = gg._new_args

        def early(device, cu, pad):
            args = new(device, cu, pad)
            for k, v in self.fields.items():
                setattr(args, k, v)
            return args
        self.ctx = self.mp.context()
        self.ctx.__enter__().setattr(gg, "_new_args", early)

    def __exit__(self, *exc):
        self.ctx.__exit__(*exc)


@pytest.mark.parametrize("kind", ["down", "gate_up", "wgrad"])
def test_early_launch_waits_for_the_kernel_before_without_limit(kind, cuda_device, monkeypatch):
    """The kernel before holds one pair of SMs for about 25 ms; the next launch starts beside it, on all others, with waits of 1 ms.
    Those count from the end of the kernel before, whose output it reads."""
    from moonep_b200.ops import grouped_gemm as gg
    monkeypatch.setenv("MOONEP_GEMM_2CTA", "1")
    S, K, N = 8192, 7168, 2048
    cu = torch.tensor([S], dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(10)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    x, wg, wu, w, w2, dy = bf(S, K), bf(1, K, N, sc=0.02), bf(1, K, N, sc=0.02), bf(1, N, 512, sc=0.05), bf(1, N, 512, sc=0.05), bf(S, 256)
    act = torch.zeros(S, N, dtype=torch.bfloat16, device="cuda")
    out = {"wgrad": lambda: torch.full((1, N, 256), 7.0, device="cuda")}.get(kind, lambda: torch.full((S, 512), 7.0, dtype=torch.bfloat16, device="cuda"))
    call = {"down": lambda o: gg.down(act, w, cu, o), "gate_up": lambda o: gg.gate_up(act, w, w2, cu, o), "wgrad": lambda o: gg.wgrad(act, dy, cu, o)}[kind]
    got, want = out(), out()
    torch.cuda.synchronize()
    t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    t[0].record()
    gg.gate_up(x, wg, wu, cu, act, num_ctas=2)
    with _Early(monkeypatch, budget_ns=1_000_000):
        call(got)
    t[1].record()
    call(want)
    torch.cuda.synchronize()
    gg.check_status()
    assert t[0].elapsed_time(t[1]) > 8, "the kernel before is meant to outlast the limit several times over"
    assert torch.equal(got, want)


@pytest.mark.parametrize("call", ["dispatch", "again", "combine"])
def test_early_launch_behind_an_exchange_call_finds_what_came_before_it(call, cuda_device, monkeypatch):
    """A dispatch or combine that set itself up beside the kernel before lets the next launch begin only when that kernel is done: weights which a kernel
    in front of the exchange call writes, on one pair of SMs for about half a millisecond, are there when an early launch behind the call loads them."""
    from moonep_b200 import Buffer, routing
    from moonep_b200.ops import grouped_gemm as gg
    monkeypatch.setenv("MOONEP_GEMM_2CTA", "1")
    S, H, K, E = 40, 256, 2, 4                          # fewer CTAs than SMs: all of them run beside the kernel before
    buf = Buffer(S, H, K, E, 1)
    topk, _, tpe = routing.softmax_topk(S, K, E, 0.5, 3, 0, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(14)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    hid, src, w_src, x = bf(S, H), bf(2048, 7168), bf(1, 7168, 512, sc=0.02), bf(384, 2048)
    cu_src, cu = (torch.tensor([n], dtype=torch.int32, device="cuda") for n in (2048, 384))
    w, out = torch.zeros(1, 2048, 512, dtype=torch.bfloat16, device="cuda"), torch.empty(384, 512, dtype=torch.bfloat16, device="cuda")
    rows, _, _, plan = buf.dispatch(hid, None, topk, tpe)
    calls = dict(dispatch=lambda: buf.dispatch(hid, None, topk, tpe, zero_copy=True), again=lambda: buf.dispatch(hid, plan=plan, zero_copy=True),
                 combine=lambda: buf.combine(plan=plan, hidden_nvsh=rows))
    gg.down(src, w_src, cu_src, w[0])
    gg.down(x, w, cu, out)
    want = out.clone()
    for _ in range(5):
        w.zero_()
        out.zero_()
        torch.cuda.synchronize()
        gg.down(src, w_src, cu_src, w[0], num_ctas=2)
        calls[call]()
        with _Early(monkeypatch):
            gg.down(x, w, cu, out)
        torch.cuda.synchronize()
        gg.check_status()
        buf.check()
        assert torch.equal(out, want)
    buf.destroy()


@pytest.mark.parametrize("split", [(2,), (28,), (30,), (148,), (10, 138)], ids=str)
def test_token_major_tiles_of_uneven_groups(split, cuda_device, monkeypatch):
    """Groups of 0 to 1000 rows, ordered by the size of their tiles up to twelve rounds (gate/up from 15 pairs on, the others from 8) and by number above: the
    bits of each group alone, with tickets too. Launches on one ticket order their list alike, although alone they would not."""
    from moonep_b200.ops import grouped_gemm as gg
    monkeypatch.setenv("MOONEP_GEMM_2CTA", "1")
    K, N, n = 256, 512, [[40, 0, 1000, 257, 33, 512, 128, 700, 1][i % 9] for i in range(27)]
    p = [(r + 127) // 128 * 128 for r in n]
    ends = torch.tensor(p).cumsum(0)
    cu = ends.to(torch.int32).cuda()
    pad = torch.tensor([[int(e) - q + r, q - r] if q > r else [0, 0] for r, q, e in zip(n, p, ends)], dtype=torch.int32).cuda()
    g = torch.Generator(device="cuda").manual_seed(11)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    x, x2, w, wu, scale = bf(sum(p), K), bf(sum(p), 2 * K), bf(27, K, N, sc=0.05), bf(27, K, N, sc=0.05), torch.rand(sum(p), device="cuda", generator=g)
    calls = [lambda o, **kw: gg.gate_up(x, w, wu, cu, o, row_scale=scale, pad=pad, **kw), lambda o, **kw: gg.down(x, w, cu, o, pad=pad, **kw),
             lambda o, **kw: gg.dgrad(x, w.view(27, N, K), cu, o, pad=pad, **kw), lambda o, **kw: gg.dgrad_gate_up(x2, w.view(27, N, K), wu.view(27, N, K), cu, o, pad=pad, **kw)]
    for call in calls:
        want, *got = (torch.full((sum(p), N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(3))
        for i in range(27):
            call(want, groups=(i, i + 1))
        if len(split) == 1:
            call(got[0], num_ctas=split[0])
            call(got[1], num_ctas=split[0], dynamic=True)
        else:
            for o in got:
                tk = gg.Ticket(x.device, sum(split))
                for c in split:
                    call(o, num_ctas=c, ticket=tk)
        torch.cuda.synchronize()
        gg.check_status()
        assert all(torch.equal(o.view(torch.int16), want.view(torch.int16)) for o in got)


def _around_the_depth_of_the_ring(most, depths, block, columns, tokens, check, monkeypatch):
    """A launch that fills its ring with weights while the kernel before still writes its rows: fewer blocks of depth than stages, as many, more;
    27 groups, some empty, on two pairs (many tiles each) and on all (some without one); tiles from token counts or from cu_seqlens.
    The bits of an ordinary launch behind the kernel before; with `check` of single CTAs, too, and of launches that stream their weights."""
    import ctypes as C

    from moonep_b200 import _native
    from moonep_b200.ops import grouped_gemm as gg
    monkeypatch.setenv("MOONEP_GEMM_2CTA", "1")
    E = 27
    wide = (2 * block * max(depths) + 256 + 255) // 256 * 256
    n = [(most, 0, 1, most // 2, 32, 0, most - 1)[i % 7] for i in range(E)]
    p = [(r + 127) // 128 * 128 for r in n]
    ends = torch.tensor(p).cumsum(0)
    rows, cu = sum(p), ends.to(torch.int32).cuda()
    pad = torch.tensor([[int(e) - q + r, q - r] if q > r else [0, 0] for r, q, e in zip(n, p, ends)], dtype=torch.int32).cuda()
    real = torch.cat([torch.arange(e - q, e - q + r) for r, q, e in zip(n, p, ends.tolist())]).cuda()
    tpe = torch.tensor(n, dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(12)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    src, w_src = bf(rows, 512), bf(E, 512, wide, sc=0.05)
    whole = torch.tensor([rows] + [rows] * (E - 1), dtype=torch.int32, device="cuda")
    x = torch.zeros(rows, wide, dtype=torch.bfloat16, device="cuda")
    before = lambda: gg.down(src, w_src, whole, x, num_ctas=2)     # noqa: E731
    fields = dict(tokens=tpe.data_ptr(), tokens_n=E, token_padding=128) if tokens else {}
    for d in depths:
        K = block * d
        N = columns(E * K)
        w, wu, dy = bf(E, K, N, sc=0.05), bf(E, K, N, sc=0.05), bf(rows, N)
        for r, q, e in zip(n, p, ends.tolist()):
            dy[e - q + r:e] = 0
        calls = {"gate_up": lambda o, **kw: gg.gate_up(x[:, :K], w, wu, cu, o, pad=pad, **kw), "down": lambda o, **kw: gg.down(x[:, :K], w, cu, o, pad=pad, **kw),
                 "dgrad": lambda o, **kw: gg.dgrad(x[:, :K], w.view(E, N, K), cu, o, pad=pad, **kw),
                 "dgrad_gu": lambda o, **kw: gg.dgrad_gate_up(x[:, :2 * K], w.view(E, N, K), wu.view(E, N, K), cu, o, pad=pad, **kw)}
        if d == depths[0] and block == 64:
            calls["wgrad"] = lambda o, **kw: gg.wgrad(x[:, :512], dy, cu, o, pad=pad, zero_empty_below=E, **kw)
        for name, call in calls.items():
            shape, dt = ((E, 512, N), torch.float32) if name == "wgrad" else ((rows, N), torch.bfloat16)
            want, *got = (torch.full(shape, 7.0, dtype=dt, device="cuda") for _ in range(3))
            before()
            call(want)
            for o, ctas in zip(got, (4, 148)):
                x.zero_()
                before()
                with _Early(monkeypatch, **fields):
                    call(o, num_ctas=ctas)
            torch.cuda.synchronize()
            gg.check_status()
            assert all(torch.equal(o, want) for o in got), f"{name}, {d} blocks"
            if check and name != "wgrad":
                mode, k = dict(gate_up=(gg.GATE_UP, K), down=(gg.DOWN, K), dgrad=(gg.DGRAD, K), dgrad_gu=(gg.DGRAD_GU, 2 * K))[name]
                assert _native.load().mep_pair_kind(mode, C.c_int64(rows), E, N, k, 0, 0, 1) == 2, "not the kernel that streams"
                single = torch.empty_like(want)
                with monkeypatch.context() as m:
                    m.setenv("MOONEP_GEMM_2CTA", "0")
                    call(single)
                assert torch.equal(single[real], want[real]), f"{name}, {d} blocks: single CTAs"


@pytest.mark.parametrize("tokens", [False, True], ids=["cu", "tokens"])
@pytest.mark.parametrize("most,depths", [(32, (9, 10, 11, 20)), (128, (7, 8, 9)), (300, (1, 5, 6, 7, 13))], ids=["ring10", "ring8", "ring6"])
def test_early_launches_around_the_depth_of_the_ring(most, depths, tokens, cuda_device, monkeypatch):
    """64-deep blocks."""
    _around_the_depth_of_the_ring(most, depths, 64, lambda k: 256, tokens, False, monkeypatch)


@pytest.mark.parametrize("tokens", [False, True], ids=["cu", "tokens"])
@pytest.mark.parametrize("most,depths", [(32, (1, 2, 4, 5, 6, 11)), (96, (3, 4, 5)), (128, (3, 4, 5, 9)), (255, (1, 2, 3, 4, 7))], ids=["ring5", "ring4_16", "ring4", "ring3"])
def test_early_launches_of_streamed_weights_around_the_depth_of_the_ring(most, depths, tokens, cuda_device, monkeypatch):
    """128-deep blocks: 27 matrices of 32 MiB, the narrowest that are so large."""
    _around_the_depth_of_the_ring(most, depths, 128, lambda k: -(-(32 << 20) // (2 * k * 256)) * 256, tokens, True, monkeypatch)


def test_counts_that_fall_give_no_tiles(cuda_device):
    """Ends of groups that fall, as a corrupt table may have them: such a group has no tiles, the others have theirs, and every access stays inside
    the tensors (all ends do)."""
    from moonep_b200.ops import grouped_gemm as gg
    cu = torch.tensor([256, 128, 384], dtype=torch.int32, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(13)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    x, w, wt, dy = bf(384, 256), bf(3, 256, 512, sc=0.05), bf(3, 512, 256, sc=0.05), bf(384, 256)
    y, dA, dW = (torch.full(s, 7.0, dtype=t, device="cuda") for s, t in (((384, 512), torch.bfloat16), ((384, 512), torch.bfloat16), ((3, 256, 256), torch.float32)))
    pad = torch.zeros(3, 2, dtype=torch.int32, device="cuda")
    gg.down(x, w, cu, y, pad=pad)
    gg.dgrad(x, wt, cu, dA, pad=pad)
    gg.wgrad(x, dy, cu, dW, pad=pad)
    torch.cuda.synchronize()
    gg.check_status()
    for out, ref in ((y, w), (dA, wt.transpose(1, 2))):      # rows 128 to 255 belong to two groups
        assert _rel(out[:128], x[:128].float() @ ref[0].float()) < 4e-3 and _rel(out[256:], x[256:].float() @ ref[2].float()) < 4e-3
    assert _rel(dW[0], x[:256].float().T @ dy[:256].float()) < 1e-4 and _rel(dW[2], x[128:].float().T @ dy[128:].float()) < 1e-4
    assert bool((dW[1] == 7.0).all())


@pytest.mark.parametrize("n", [[1, 32, 256, 257, 0, 600, 255, 512], [1, 32, 96, 64, 0, 33, 16, 95], [1, 128, 97, 64, 0, 127, 128, 33]], ids=["rows128", "rows16", "rows64"])
@pytest.mark.parametrize("K", [1984, 2048], ids=["kept", "streamed"])
def test_weights_that_are_read_once(K, n, cuda_device):
    """From 32 MiB of matrices on (8 of 2048 x 1024) the weights of groups with one token tile leave L2 first, in stages of 128: the same bits as group by
    group, where they never do, with tiles that share their weights in between; with rows in boxes of 128, 64 and 16, in both tile orders, and behind flags
    of tiles and groups (which are all up)."""
    import ctypes as C

    from moonep_b200 import _native
    from moonep_b200.api import SlotReady, TileReady
    from moonep_b200.ops import grouped_gemm as gg
    N = 1024
    p = [(r + 127) // 128 * 128 for r in n]
    ends = torch.tensor(p).cumsum(0)
    pad = torch.tensor([[int(e) - q + r, q - r] if q > r else [0, 0] for r, q, e in zip(n, p, ends)], dtype=torch.int32)
    g = torch.Generator(device="cuda").manual_seed(5)
    bf = lambda *s, sc=1.0: (torch.randn(*s, device="cuda", generator=g) * sc).to(torch.bfloat16)     # noqa: E731
    x, h, w, wu = bf(sum(p), K), bf(sum(p), 2 * N), bf(8, K, N, sc=0.02), bf(8, K, N, sc=0.02)
    wt = w.transpose(1, 2).contiguous()

    up = torch.full((64,), 5, dtype=torch.int32, device="cuda")          # flags and their epoch
    flags = dict(ready=TileReady(up.data_ptr(), up.data_ptr(), 148), slots=SlotReady(up.data_ptr(), up.data_ptr(), 3))

    def run(x, h, w, wu, wt, cu, pad, dynamic=False, gated={}):
        out = [torch.zeros(len(x), c, dtype=torch.bfloat16, device="cuda") for c in (N, 2 * N, N, N)]
        kw = dict(pad=pad.cuda(), dynamic=dynamic)
        gg.gate_up(x, w, wu, cu.cuda(), out[0], out[1], **kw, **gated)
        gg.down(x, w, cu.cuda(), out[2], **kw)
        gg.dgrad(x, wt, cu.cuda(), out[3], **kw, **gated)
        if K % 256 == 0:
            out.append(torch.zeros(len(x), K, dtype=torch.bfloat16, device="cuda"))
            gg.dgrad_gate_up(h, w, wu, cu.cuda(), out[4], **kw)
        return out

    args = x, h, w, wu, wt, ends.to(torch.int32), pad
    assert _native.load().mep_pair_kind(gg.DOWN, C.c_int64(sum(p)), 8, N, K, 0, 0, 0) == (2 if K == 2048 else 0)
    got = run(*args)
    for kw in (dict(dynamic=True), dict(gated=flags), dict(dynamic=True, gated=flags)):
        assert all(torch.equal(a, b) for a, b in zip(got, run(*args, **kw)))
    for i, (q, e) in enumerate(zip(p, ends.tolist())):
        if q:
            s, one = slice(e - q, e), torch.tensor([q], dtype=torch.int32)
            table = torch.tensor([[n[i], q - n[i]] if q > n[i] else [0, 0]], dtype=torch.int32)
            for a, b in zip(got, run(x[s].contiguous(), h[s].contiguous(), w[i:i + 1], wu[i:i + 1], wt[i:i + 1], one, table)):
                assert torch.equal(a[s], b), f"group {i} ({n[i]} rows)"
    torch.cuda.synchronize()
    gg.check_status()
