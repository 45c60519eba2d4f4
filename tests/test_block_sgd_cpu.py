"""How a block launches its experts' update, without a GPU."""
from types import SimpleNamespace

import torch


def test_update_beside_a_reduction_names_its_blocks(monkeypatch):
    """While the reduction of ``up`` still runs on the communication stream, ``down`` and ``gate`` are updated beside it, by small
    blocks, each behind its own gradient."""
    from moonep_b200.models import moe_block
    calls = []
    monkeypatch.setattr(moe_block.gg, "sgd_step", lambda p, g, lr, num_blocks=None: calls.append(("sgd", p, g, lr, num_blocks)))
    blk = object.__new__(moe_block.MoEBlock)
    blk.moe = SimpleNamespace(on_grad_ready=None, grads_pending=("up", None), _total_sms=148, wait_grads=lambda n: calls.append(("wait", n)))
    blk.pools = SimpleNamespace(local_weight=lambda n: "w_" + n, local_grad=lambda n: "d_" + n)
    blk.router, blk.shared = torch.zeros(1), None
    blk.sgd_step(0.5)
    assert calls == [c for n in ("down", "gate", "up") for c in (("wait", n), ("sgd", "w_" + n, "d_" + n, 0.5, 8 * 148))]


def test_a_negative_number_of_blocks_is_refused():
    import ctypes as C

    from moonep_b200 import _native
    lib, p, n, lr = _native.load(), C.c_void_p(4096), C.c_int64(64), C.c_float(0.5)
    many = (C.c_void_p * 1)(4096), (C.c_void_p * 1)(4096), (C.c_int64 * 1)(64)
    for call in (lambda b: lib.mep_sgd_step(p, p, lr, n, b, None), lambda b: lib.mep_sgd_step_many(1, *many, lr, b, None),
                 lambda b: lib.mep_sgd_step_groups(p, p, lr, n, 1, p, 1, b, None)):
        assert call(-1) != 0 and lib.mep_last_error().endswith(b"-1 blocks")
