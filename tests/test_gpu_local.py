"""Single-rank dispatch / combine (one kernel each) against the CPU oracle, at the sizes where the kernels' splits
end: fewer tokens than CTAs, chunks of 1024 entries, one to many experts per thread, rows from 16 bytes to several
zero-fill stores, one to 32 entries per token."""
import numpy as np
import pytest
import torch

from moonep_b200 import Buffer
from moonep_b200.sim import plan_cluster, ops as simops
from gpu_helpers import make_topk, traceable_hidden, check_plans, defined_rows

pytestmark = pytest.mark.gpu

CASES = [
    # S      K   E     H      pad  routing
    (1,      1,  1,    8,     1,   "random"),
    (3,      32, 32,   16,    16,  "random"),
    (147,    8,  16,   2048,  128, "biased"),
    (149,    7,  24,   2056,  16,  "random"),
    (700,    4,  257,  256,   1,   "random"),
    (512,    2,  2048, 64,    8,   "random"),
    (333,    5,  5,    7168,  128, "single_expert"),
    (64,     8,  8,    15360, 128, "biased"),
    (20000,  8,  32,   64,    128, "biased"),
    (3072,   8,  64,   128,   16,  "random"),     # 24576 entries: counted in six whole rounds of 4096
    (3511,   7,  64,   128,   16,  "random"),     # 24577
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "S%d_K%d_E%d_H%d" % c[:4])
def test_local_exchange(case, cuda_device):
    S, K, E, H, pad, kind = case
    topk, tpe = make_topk(kind, S, K, E, 1, seed=7)
    cp = plan_cluster(np.stack([t.numpy() for t in topk]), E, pad)
    buf = Buffer(S, H, K, E, 1, token_padding=pad)
    hidden = traceable_hidden(S, H, 0)
    w = (torch.arange(S * K, dtype=torch.int32) + 1).view(torch.float32).reshape(S, K)
    eh, ew = simops.dispatch(cp, [hidden.view(torch.int16).float()], [w.view(torch.int32).float()], fill=-1.0)
    m = defined_rows(cp, 0)
    g = torch.Generator().manual_seed(3)
    y = torch.randn(cp.NvS, H, generator=g).to(torch.bfloat16)
    args = hidden.cuda(), w.cuda(), topk[0].cuda(), tpe[0].cuda()
    for zero_copy in (True, False, True):           # the launch's counters reset themselves
        buf.hidden_nvsh_buffer_view.view(torch.int16).fill_(0x5555)
        buf.router_weight_buffer_view.view(torch.int32).fill_(0x55555555)
        h, wn, cu, plan = buf.dispatch(*args, zero_copy=zero_copy, router_weights_zero_copy=zero_copy)
        torch.cuda.synchronize()
        buf.check()
        check_plans([plan], [cu], cp, 1)
        assert torch.equal(h.cpu().view(torch.int16).float()[m], eh[0][m])
        assert torch.equal(wn.cpu().view(torch.int32).float()[m], ew[0][m])
    assert bool((buf.hidden_nvsh_buffer_view.cpu().view(torch.int16)[~m] == 0x5555).all()), "rows of no group were written"
    ydw = wn.clone()
    # the saved plan brings the same rows, and nothing else
    buf.hidden_nvsh_buffer_view.view(torch.int16).fill_(0x3333)
    buf.router_weight_buffer_view.view(torch.int32).fill_(0x33333333)
    h2, w2, cu2, plan2 = buf.dispatch(args[0], plan=plan, zero_copy=True)
    torch.cuda.synchronize()
    assert plan2 is plan and w2 is None and cu2 is None
    assert torch.equal(h2.cpu().view(torch.int16).float()[m], eh[0][m])
    assert bool((buf.router_weight_buffer_view.view(torch.int32) == 0x33333333).all())
    # combine: fp32 sum in ascending k, rounded once
    yd = y.cuda()
    out, gw, _ = buf.combine(plan=plan, hidden_nvsh=yd, route_weights_nvs=ydw)
    torch.cuda.synchronize()
    buf.check()
    eo, _ = simops.combine(cp, [y])
    assert torch.equal(out.cpu(), eo[0])
    assert torch.equal(gw.cpu().view(torch.int32), w.view(torch.int32)) and torch.equal(yd.cpu(), y)
    buf.destroy()


def test_local_exchange_reports_bad_tables(cuda_device):
    """A foreign table must end in a status, not in an access outside the buffers: an expert id that does not exist,
    counts that are not those of the table, rows of the saved plan outside the shard."""
    from moonep_b200.engine import MoonEPTimeout
    S, H, K, E = 40, 64, 4, 8
    topk, tpe = (t[0].cuda() for t in make_topk("random", S, K, E, 1, seed=5))
    x = torch.zeros(S, H, dtype=torch.bfloat16, device="cuda")
    for what in ("expert", "counts", "plan", "combine"):
        buf = Buffer(S, H, K, E, 1, token_padding=8)
        h, _, _, plan = buf.dispatch(x, None, topk, tpe, zero_copy=True)
        if what == "expert":
            bad = topk.clone(); bad[3, 1] = E + 5
            buf.dispatch(x, None, bad, tpe)
        elif what == "counts":
            bad = tpe.clone(); bad[int(bad.argmax())] -= 3
            buf.dispatch(x, None, topk, bad)
        else:
            plan.dst[7] = buf.NvS + 11
            if what == "plan":
                buf.dispatch(x, plan=plan)
            else:
                buf.combine(plan=plan, hidden_nvsh=h, zero_copy=True)
        with pytest.raises(MoonEPTimeout) as ei:
            buf.check()
        assert ei.value.status["code"] == 3
        buf.reset()
        buf.destroy()


def test_combine_of_rows_that_start_off_a_16_byte_boundary(cuda_device):
    S, H, K, E = 40, 64, 4, 8
    topk, tpe = (t[0].cuda() for t in make_topk("random", S, K, E, 1, seed=5))
    x = torch.randn(S, H, device="cuda").to(torch.bfloat16)
    buf = Buffer(S, H, K, E, 1, token_padding=8)
    h, _, _, plan = buf.dispatch(x, None, topk, tpe)
    rows = torch.empty(h.numel() + 1, dtype=h.dtype, device="cuda")[1:].view(h.shape)
    rows.copy_(h)
    a, _, _ = buf.combine(plan=plan, hidden_nvsh=h)
    b, _, _ = buf.combine(plan=plan, hidden_nvsh=rows)
    torch.cuda.synchronize()
    buf.check()
    assert rows.data_ptr() % 16 == 2 and torch.equal(a, b)
    buf.destroy()


def test_padding_rows_are_counted(cuda_device):
    """A Buffer's dispatch clears every padding row, fresh or saved; a layer's those that its GEMMs read."""
    from moonep_b200.models.moe_block import MoEBlock, MoEConfig
    S, H, K, E = 700, 64, 4, 8
    topk, tpe = (t[0].cuda() for t in make_topk("biased", S, K, E, 1, seed=5))
    x = torch.zeros(S, H, dtype=torch.bfloat16, device="cuda")
    buf = Buffer(S, H, K, E, 1)
    _, _, _, plan = buf.dispatch(x, None, topk, tpe, zero_copy=True)
    pads = buf.stats(plan)["padded_rows"]
    assert pads > 0 and buf.counters()["padding_rows_cleared"] == pads
    buf.dispatch(x, plan=plan, zero_copy=True)
    assert buf.counters(reset=True)["padding_rows_cleared"] == 2 * pads
    buf.destroy()
    blk = MoEBlock(MoEConfig("t", H=256, Hp=256, K=2, epn=4, S=130), num_sms=4, seed=3)
    y = torch.randn(130, 256, device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        _, _, tpe = blk.route(y)
        blk.forward(y)
    assert blk.buf.counters()["padding_rows_cleared"] == int((-tpe % 32).sum())
    blk.destroy()


# Every CTA counts the entries before its own up to 65536 of them, in rounds of 4096; above that the CTAs hand over their histograms (COUNT_CASES), and
# from 24576 * 7168 elements of rows on (ROW_CASES: the last batch below and the first above, with two slots a warp).
COUNT_CASES = [
    (4097,   1,  8,    64,    16,  "random"),
    (4213,   2,  300,  16,    1,   "biased"),
    (8192,   8,  64,   128,   16,  "random"),
    (9363,   7,  64,   64,    16,  "biased"),
    (9400,   7,  700,  16,    1,   "random"),     # the hand-over with more experts than a CTA has threads
]


ROW_CASES = [
    (2194,   11, 24,   7296,  16,  "random"),
    (2195,   11, 24,   7296,  16,  "random"),
]


@pytest.mark.parametrize("case", COUNT_CASES + ROW_CASES, ids=lambda c: "S%d_K%d_E%d_H%d" % c[:4])
def test_local_exchange_at_the_ends_of_counting(case, cuda_device):
    test_local_exchange(case, cuda_device)


# Large batches (200 MiB moved): the saved plan's rows come from many short CTAs and the combine begins with the last tokens. Just above
# the line, one entry per token, a token for each CTA with rows of which three fit. Their fresh plans are counted; ROW_CASES has large ones with the hand-over.
LARGE_CASES = [
    (2048, 8,  48,   5696,  16,  "random"),
    (5003, 5,  40,   3496,  128, "biased"),
    (9600, 1,  7,    5464,  1,   "random"),
    (200,  32, 64,   15904, 16,  "random"),
]


@pytest.mark.parametrize("case", LARGE_CASES, ids=lambda c: "S%d_K%d_E%d_H%d" % c[:4])
def test_local_exchange_of_large_batches(case, cuda_device):
    test_local_exchange(case, cuda_device)


@pytest.mark.parametrize("limit", [None, 12])
def test_saved_plan_of_a_large_batch_keeps_to_the_sm_limit(limit, cuda_device, monkeypatch):
    """``MOONEP_NUM_SMS_DEDUP`` bounds the CTAs of every dispatch, also of one that would be copied by many short ones."""
    from moonep_b200 import engine
    monkeypatch.setenv("MOONEP_TRACE", "1")
    if limit is not None:
        monkeypatch.setenv("MOONEP_NUM_SMS_DEDUP", str(limit))
    S, K, E, H = 2048, 8, 48, 5696
    topk, tpe = (t[0].cuda() for t in make_topk("random", S, K, E, 1, seed=7))
    buf = Buffer(S, H, K, E, 1)
    x = traceable_hidden(S, H, 0).cuda()
    h, _, _, plan = buf.dispatch(x, None, topk, tpe)
    engine.read_trace(buf._states[0])
    again, _, _, _ = buf.dispatch(x, plan=plan)
    ctas = {r[3] for r in engine.read_trace(buf._states[0])}
    buf.check()
    assert len(ctas) <= limit if limit else len(ctas) > torch.cuda.get_device_properties(0).multi_processor_count
    rows = torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long()
    assert torch.equal(again.view(torch.int16)[rows], h.view(torch.int16)[rows])
    buf.destroy()


@pytest.mark.parametrize("pdl", [(True,), (False,), (True, False)], ids=["pdl", "plain", "in_turn"])
@pytest.mark.parametrize("shape", [(64, 8, 16, 256), (4000, 4, 32, 1024), (9000, 8, 16, 64), (2048, 8, 48, 5696)], ids=str)
def test_queued_calls_see_what_the_kernel_before_wrote(shape, pdl, cuda_device):
    """Launches may begin while the one before still runs: batches queued without a pause, each routed and filled by kernels right in front of its
    calls, give what ordinary launches give with a pause behind every one. ``enable_pdl`` may be changed from one batch to the next."""
    S, K, E, H = shape
    buf = Buffer(S, H, K, E, 1, token_padding=16)
    base, scale = torch.randn(S, H, device="cuda").to(torch.bfloat16), torch.rand(S, K, device="cuda")
    tables = [tuple(t[0].cuda() for t in make_topk("random", S, K, E, 1, seed=s)) for s in (1, 2, 3)]
    x, w, topk, tpe = torch.empty_like(base), torch.empty_like(scale), torch.empty_like(tables[0][0]), torch.empty_like(tables[0][1])

    def batch(i, pause):
        """The producer in front of the first call is another one in every third batch."""
        fill = [lambda: torch.mul(base, 1.0 + 0.25 * (i % 5), out=x), lambda: torch.add(tables[i % 3][1], 0, out=tpe),
                lambda: torch.add(tables[i % 3][0], 0, out=topk), lambda: torch.mul(scale, 1.0 + i, out=w)]
        for f in fill[i % 4:] + fill[:i % 4]:
            f()
            pause()
        h, wn, cu, plan = buf.dispatch(x, w, topk, tpe, zero_copy=True, router_weights_zero_copy=True)
        pause()
        y, wb, _ = buf.combine(plan=plan, hidden_nvsh=h, route_weights_nvs=wn, zero_copy=True, router_weights_zero_copy=True)
        pause()
        h, _, _, _ = buf.dispatch(y, plan=plan, zero_copy=True)
        pause()
        z = buf.combine(plan=plan, hidden_nvsh=h, zero_copy=True)[0]
        pause()
        return y, wb, z, cu, plan.dst, plan.zero_fill_ranges

    buf.enable_pdl = False
    want = [batch(i, torch.cuda.synchronize) for i in range(12)]
    got = []
    for i in range(24):
        buf.enable_pdl = pdl[i % len(pdl)]
        got.append(batch(i % 12, lambda: None))
    torch.cuda.synchronize()
    buf.check()
    for i, g in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(g, want[i % 12])), f"batch {i}"
    buf.destroy()


def test_calls_on_the_communication_stream_are_ordinary_launches(cuda_device):
    """They follow an event and no kernel, and share the SMs with what runs on other streams; calls on the caller's stream follow the switch again."""
    S, K, E, H = 300, 4, 16, 256
    buf = Buffer(S, H, K, E, 1, token_padding=16)
    topk, tpe = (t[0].cuda() for t in make_topk("random", S, K, E, 1, seed=5))
    x = torch.randn(S, H, device="cuda").to(torch.bfloat16)
    seen = []
    for enabled in (True, False):
        for asynchronous in (False, True, False):
            buf.enable_pdl = enabled
            h, _, _, plan, *ev = buf.dispatch(x, None, topk, tpe, async_finish=asynchronous)
            seen.append(buf._local_ex._args.pdl)
            for e in ev:
                torch.cuda.current_stream().wait_event(e)
            y, _, e = buf.combine(plan=plan, hidden_nvsh=h, async_finish=asynchronous)
            seen.append(buf._local_ex._args.pdl)
            if e is not None:
                torch.cuda.current_stream().wait_event(e)
            torch.cuda.synchronize()
            assert torch.equal(y, x * 4)               # four equal numbers: exact
    buf.check()
    assert seen == [1, 1, 0, 0, 1, 1] + [0] * 6
    buf.destroy()


@pytest.mark.parametrize("pdl", [False, True], ids=["plain", "pdl"])
@pytest.mark.parametrize("before", ["copy", "memset", "kernel", "join"])
def test_captured_calls_behind_nodes_of_every_kind(before, pdl, cuda_device):
    """The first exchange call of a captured graph right behind a copy, a memset, a kernel, and a join of two streams whose last nodes are a kernel and a
    copy; replayed back to back with new inputs."""
    S, K, E, H = 300, 4, 16, 512
    buf = Buffer(S, H, K, E, 1, token_padding=16, enable_pdl=pdl)
    tables = [tuple(t[0].cuda() for t in make_topk("random", S, K, E, 1, seed=s)) for s in (1, 2, 3)]
    xs = [torch.randn(S, H, device="cuda").to(torch.bfloat16) for _ in range(3)]
    src_x, src_k, src_t = xs[0].clone(), tables[0][0].clone(), tables[0][1].clone()
    x, topk, tpe, junk = torch.empty_like(src_x), src_k.clone(), src_t.clone(), torch.empty(1 << 22, dtype=torch.uint8, device="cuda")
    side = torch.cuda.Stream()

    def body():
        if before == "join":
            cur = torch.cuda.current_stream()
            side.wait_stream(cur)
            with torch.cuda.stream(side):
                x.copy_(src_x)
            torch.add(src_k, 0, out=topk)
            torch.add(src_t, 0, out=tpe)
            cur.wait_stream(side)
        else:
            torch.add(src_k, 0, out=topk)
            torch.add(src_t, 0, out=tpe)
            torch.add(src_x, 0, out=x) if before == "kernel" else x.copy_(src_x)
            if before == "memset":
                junk.zero_()
        h, _, _, plan = buf.dispatch(x, None, topk, tpe, zero_copy=True)
        return buf.combine(plan=plan, hidden_nvsh=h, zero_copy=True)[0]

    body()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = body()
    for i in range(9):
        src_x.copy_(xs[i % 3])
        src_k.copy_(tables[i // 3][0])
        src_t.copy_(tables[i // 3][1])
        graph.replay()
        graph.replay()
        got = y.clone()
        torch.cuda.synchronize()
        # every token's row comes back K = 4 times: the sum of four equal numbers is exact
        assert torch.equal(got, xs[i % 3] * 4)
    buf.check()
    del graph
    buf.destroy()


@pytest.mark.parametrize("limit,shapes", [(None, {(8192, 8, 64): 0, (8193, 8, 64): 1, (2194, 11, 7296): 0, (2195, 11, 7296): 1}), (99, {(8192, 8, 64): 0}), (98, {(5120, 8, 64): 0, (5121, 8, 64): 1}),
                                          (16, {(5120, 8, 64): 0, (8192, 8, 64): 1})], ids=str)
def test_which_dispatches_hand_over(limit, shapes, cuda_device, monkeypatch):
    """Up to 65536 entries and 24576 * 7168 elements every CTA counts for itself, up to 40960 where it may use less than two thirds of the (148) SMs; only the hand-over numbers its launches."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the limits are those of 148 SMs")
    if limit is not None:
        monkeypatch.setenv("MOONEP_NUM_SMS_DEDUP", str(limit))
    for (S, K, H), launches in shapes.items():
        topk, tpe = make_topk("biased", S, K, 24, 1, seed=5)
        cp = plan_cluster(np.stack([t.numpy() for t in topk]), 24, 16)
        buf = Buffer(S, H, K, 24, 1, token_padding=16)
        x = traceable_hidden(S, H, 0).cuda()
        h, _, cu, plan = buf.dispatch(x, None, topk[0].cuda(), tpe[0].cuda(), zero_copy=True)
        torch.cuda.synchronize()
        buf.check()
        check_plans([plan], [cu], cp, 1)
        rows = torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long()
        assert torch.equal(h.view(torch.int16)[rows], x.view(torch.int16).repeat_interleave(K, 0))
        assert int(buf._states[0].scratch["loc_sync"][0]) == launches
        buf.destroy()
