"""Which kernel a token-major grouped GEMM runs on: the rule's fixed points, without a GPU."""
import pytest

from moonep_b200.ops.grouped_gemm import DGRAD, DGRAD_GU, DOWN, GATE_UP, _on_pairs

MODES = [GATE_UP, DOWN, DGRAD, DGRAD_GU]


@pytest.mark.parametrize("mode", MODES)
def test_the_switch_decides_for_all(mode, monkeypatch):
    for env in ("0", "1"):
        monkeypatch.setenv("MOONEP_GEMM_2CTA", env)
        for pad in (False, True):
            for rows in (128, 100000):
                assert _on_pairs(mode, rows, 4, 4, 512, 512, pad, 148, False) == (env == "1")
                assert not _on_pairs(mode, rows, 4, 4, 512, 512, pad, 1, False), "a single CTA is no pair"


@pytest.mark.parametrize("mode", MODES)
def test_padding_is_skipped_by_pairs_only(mode, monkeypatch):
    monkeypatch.delenv("MOONEP_GEMM_2CTA", raising=False)
    for rows in (1, 128, 5000, 100000):
        for K in (64, 512, 7168):
            assert _on_pairs(mode, rows, 16, 16, 512, K, True, 148, False)


def test_measured_sides_of_the_line(monkeypatch):
    """(mode, groups, rows of each, K, N) with the kernel that was measured to be faster by 5 % or more."""
    monkeypatch.delenv("MOONEP_GEMM_2CTA", raising=False)
    single = [(DOWN, 16, 384, 2048, 768), (DGRAD, 16, 384, 2048, 768), (DGRAD_GU, 16, 384, 4096, 768), (DOWN, 32, 128, 2048, 768),
              (DOWN, 4, 2048, 1024, 256), (DGRAD, 4, 2048, 1024, 256), (DOWN, 96, 128, 512, 512), (DGRAD, 96, 256, 512, 512),
              (DOWN, 60, 512, 256, 2816), (DGRAD, 68, 640, 512, 1792)]
    pairs = [(DOWN, 32, 384, 7168, 2048), (DGRAD, 32, 384, 7168, 2048), (DGRAD_GU, 32, 384, 14336, 2048), (DOWN, 4, 128, 7168, 2048),
             (DGRAD_GU, 16, 128, 4096, 768), (DOWN, 8, 4096, 7168, 2048), (GATE_UP, 32, 1024, 7168, 2048), (GATE_UP, 16, 128, 2048, 768)]
    for want, cases in ((False, single), (True, pairs)):
        for mode, G, r, K, N in cases:
            assert _on_pairs(mode, G * r, G, G, N, K, False, 148, False) == want, (mode, G, r, K, N)


@pytest.mark.parametrize("total", [1, 2, 3, 148])
def test_a_ticket_of_any_size_has_a_kernel(total, monkeypatch):
    """The rule is asked with the ticket's CTAs and not the launch's, so that all its launches run on one kernel."""
    monkeypatch.delenv("MOONEP_GEMM_2CTA", raising=False)
    for mode in MODES:
        for rows, K in ((0, 64), (128, 64), (6144, 2048), (40000, 7168)):
            assert _on_pairs(mode, rows, 16, 16, 768, K, False, total, True) in (True, False)


@pytest.mark.parametrize("upd_w,upd_w_b,n_each", [(0, 0, 0), (4096, 0, 256), (0, 4096, 256)])
def test_an_update_needs_the_weights_of_every_matrix(upd_w, upd_w_b, n_each):
    """The launcher refuses a mask without weights, of one matrix or of two, before it looks at anything else of the call."""
    import ctypes as C

    from moonep_b200 import _native
    from moonep_b200.ops.grouped_gemm import GemmArgs
    a = GemmArgs()
    a.G, a.M_w, a.N, a.g_end, a.out, a.n_each = 1, 256, 2 * n_each or 256, 1, 4096, n_each
    a.out_b, a.upd_mask, a.upd_w, a.upd_w_b = 4096 if n_each else 0, 4096, upd_w, upd_w_b
    with pytest.raises(_native.MoonEPNativeError, match="without the weights of every matrix"):
        p = C.c_void_p(4096)
        _native.check(_native.load().mep_grouped_wgrad_2cta(p, C.c_int64(128), C.c_int64(256), p, C.c_int64(512), C.byref(a), 148, None))


def test_a_second_update_comes_with_the_first_and_a_second_matrix():
    import torch

    from moonep_b200.ops import grouped_gemm as gg
    w, out, cu, x = torch.zeros(1, 256, 256, dtype=torch.bfloat16), torch.zeros(1, 256, 256), torch.tensor([128], dtype=torch.int32), torch.zeros(128, 256)
    up = (w, 0.1, torch.ones(1, dtype=torch.int32))
    for kw in (dict(update_b=w), dict(update_b=w, out_b=out), dict(update_b=w, update=up), dict(update=up, out_b=out)):
        with pytest.raises(AssertionError, match="update_b comes with"):
            gg.wgrad(x, x, cu, out, **kw)


PLAIN, BANDED, STREAM = range(3)


@pytest.mark.parametrize("H,Hp,E,K,S,early,late", [
    (2048, 768, 16, 8, 64, STREAM, STREAM), (2048, 768, 16, 8, 256, STREAM, STREAM), (2048, 768, 16, 8, 257, PLAIN, PLAIN),      # 128 rows an expert, one more
    (2048, 768, 11, 1, 64, STREAM, STREAM), (2048, 768, 10, 1, 64, PLAIN, STREAM), (2048, 768, 8, 8, 64, PLAIN, STREAM),          # 33, 30 and 24 MiB of matrices
    (2048, 768, 5, 1, 64, PLAIN, PLAIN), (1024, 1024, 16, 4, 200, STREAM, STREAM), (960, 1024, 16, 4, 200, PLAIN, STREAM),
    (1024, 1024, 8, 4, 200, PLAIN, STREAM), (960, 1024, 8, 4, 200, PLAIN, PLAIN), (7168, 2048, 32, 8, 256, STREAM, STREAM), (2048, 768, 16, 8, 1531, PLAIN, PLAIN)])
def test_which_gemms_stream_their_weights(H, Hp, E, K, S, early, late):
    """What decides is the experts at home and the batch's rows, on one rank in a table of 2E groups with room for all their padding, in a native pass
    (early) as in one issued from Python (late)."""
    from moonep_b200 import _native
    kind, room = _native.load().mep_pair_kind, S * K + 127 * 2 * E
    for mode, N, k in ((GATE_UP, Hp, H), (DOWN, H, Hp), (DGRAD, Hp, H), (DGRAD_GU, H, 2 * Hp)):
        deep = k % 128 == 0
        assert kind(mode, _i64(room), 2 * E, N, k, E, S * K, 1) == (early if deep else PLAIN)
        assert kind(mode, _i64(room), 2 * E, N, k, E, S * K, 0) == (late if deep else PLAIN)


def test_a_direct_call_counts_its_groups_and_the_room_for_their_rows():
    from moonep_b200 import _native
    kind = _native.load().mep_pair_kind
    for early in (0, 1):
        for G, rows, want in ((11, 11 * 320, STREAM), (11, 11 * 320 + 1, PLAIN), (10, 10, PLAIN)):
            for mode, N, k in ((GATE_UP, 768, 2048), (DOWN, 2048, 768), (DGRAD, 768, 2048), (DGRAD_GU, 2048, 1536)):
                assert kind(mode, _i64(rows), G, N, k, 0, 0, early) == want


def test_large_groups_are_banded_whoever_holds_them():
    from moonep_b200 import _native
    kind = _native.load().mep_pair_kind
    for held in ((0, 0), (1, 1000), (32, 100000)):           # 18 MiB of rows for each of 64 groups, whether they hold any or not
        assert kind(GATE_UP, _i64(32 * 4096), 64, 2048, 4608, *held, 0) == PLAIN
        assert kind(GATE_UP, _i64(32 * 4096 + 1), 64, 2048, 4608, *held, 0) == BANDED


def _i64(n):
    import ctypes as C
    return C.c_int64(n)
