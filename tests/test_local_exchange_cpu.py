"""What the single-rank exchange hands to its native calls, without a GPU."""
from types import SimpleNamespace

import torch


def test_the_hint_for_the_order_of_a_combine_belongs_to_its_plan(monkeypatch):
    """Two batches in flight: whichever was dispatched last, a combine is told how the rows of its own plan were dispatched."""
    from moonep_b200 import engine
    from moonep_b200.geometry import Geometry
    g = Geometry.make(16, 64, 2, 4, 1, 8, 4)
    st = SimpleNamespace(geo=g, ctx_ptr=0, local=True, local_blocks=148, srcinfo_local=None, device=torch.device("cpu"),
                         hidden_local=torch.empty(g.NvS, g.H, dtype=torch.bfloat16), weights_local=torch.empty(g.NvS),
                         scratch={k: torch.empty(4, dtype=torch.int32) for k in ("loc_sync", "loc_hist")})
    monkeypatch.setattr(engine._native, "raw_stream", lambda: 0)
    ex, hints = engine.LocalExchange(st, 148), []
    ex._lib = SimpleNamespace(mep_local_dispatch_call=lambda *a: 0, mep_local_combine_call=lambda *a: hints.append(engine._native.MoeLocal.from_address(a[0]).in_order) or 0)
    x, rows, topk, tpe = torch.empty(g.S, g.H, dtype=torch.bfloat16), st.hidden_local, torch.empty(g.N, dtype=torch.int32), torch.empty(g.E, dtype=torch.int32)
    (a, _), (b, _) = (ex.dispatch(x, None, topk, tpe, rows, None) for _ in range(2))
    ex.combine(a, rows, None)
    ex.dispatch_again(x, None, b, rows, None)
    ex.combine(a, rows, None)
    ex.combine(b, rows, None)
    ex.dispatch(x, None, topk, tpe, rows, None)
    ex.combine(b, rows, None)
    ex.combine(b.clone(), rows, None)
    assert hints == [0, 0, 1, 1, 0]
