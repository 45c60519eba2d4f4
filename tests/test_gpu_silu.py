"""The branch-free sigmoid and SiLU of the SwiGLU kernels against the division that they stand for."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LAST = 0x42700000           # bits of 60.0: the first float that the callers keep away from the branch-free forms
TINY = 0x0DA24260           # bits of 1e-30: below it, except for zero, the SiLU is left to the division


@pytest.mark.parametrize("sign", [0, 0x80000000], ids=["positive", "negative"])
def test_every_float_rounds_like_the_division(sign, cuda_device):
    from moonep_b200 import _native
    bad, seen = (torch.zeros(2, dtype=torch.int64, device="cuda") for _ in range(2))
    rc = _native.load().mep_silu_sweep(sign, LAST + 1000, bad.data_ptr(), seen.data_ptr(), _native.raw_stream())
    _native.check(rc, "silu_sweep")
    torch.cuda.synchronize()
    assert seen.tolist() == [LAST, LAST - TINY + 1]
    assert bad.tolist() == [0, 0]


def test_epilogue_of_infinite_and_nan_gates(cuda_device, monkeypatch):
    """Gates that overflow in the accumulator, with an up projection of one, and NaN tokens, beside finite ones: inf, -inf * 0 = NaN,
    NaN."""
    from moonep_b200.ops import grouped_gemm as gg
    monkeypatch.setenv("MOONEP_GEMM_2CTA", "1")
    rows, K, N, big = 128, 64, 128, 3e38
    x, wg, wu = (torch.zeros(s, dtype=torch.bfloat16, device="cuda") for s in ((rows, K), (1, K, N), (1, K, N)))
    x[:, 0], wu[0, 0] = 1.0, 1.0
    wg[0, 1], wg[0, 3] = big, 1.0
    x[0::4, 1] = big                        # +inf
    x[1::4, 1] = -big                       # -inf
    x[2::4, 1] = float("nan")               # in the up projection as well
    x[3::4, 3] = 1.5
    cu = torch.tensor([rows], dtype=torch.int32, device="cuda")
    act, gu = torch.empty(rows, N, dtype=torch.bfloat16, device="cuda"), torch.empty(rows, 2 * N, dtype=torch.bfloat16, device="cuda")
    gg.gate_up(x, wg, wu, cu, act, gu)
    torch.cuda.synchronize()
    gg.check_status()
    inf, nan = float("inf"), float("nan")
    gate = torch.tensor([inf, -inf, nan, 1.5], device="cuda").repeat(rows // 4)[:, None].expand(rows, N)
    assert torch.allclose(gu[:, :N].float(), gate, rtol=0, atol=0, equal_nan=True)
    assert bool(((gu[:, N:] == 1) | torch.isnan(gate)).all())
    want = (gate / (1 + torch.exp(-gate))).to(torch.bfloat16)
    assert torch.allclose(act.float(), want.float(), rtol=2.0 ** -7, atol=0, equal_nan=True)


def test_backward_of_extreme_gates(cuda_device):
    """Gates on both sides of the branch-free range, one kind or mixed in a vector of eight, against the same formula in fp32."""
    from moonep_b200.ops import grouped_gemm as gg
    inf, nan = float("inf"), float("nan")
    vals = [0.0, -0.0, 1.0, -1.0, 59.75, -59.75, 60.0, -60.0, 64.0, -64.0, 87.0, -87.0, 88.5, -88.5, 104.0, -104.0, 1e30, -1e30,
            3e38, -3e38, 1e-30, -1e-30, 1e-38, -1e-38, inf, -inf, nan, 17.0, -17.0, 30.0, -30.0, 0.5]
    rows, Hp = 64, 256
    v = torch.tensor(vals, device="cuda")
    gate = torch.empty(rows, Hp, device="cuda")
    gate[:32] = v[:, None]                                                  # a kind for each row
    gate[32:] = v[(torch.arange(Hp, device="cuda") + torch.arange(32, device="cuda")[:, None]) % 32]     # all kinds in a row
    g = torch.Generator(device="cuda").manual_seed(6)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(torch.bfloat16)     # noqa: E731
    dA, up, w = rnd(rows, Hp), rnd(rows, Hp), torch.rand(rows, device="cuda", generator=g) + 0.5
    gu = torch.cat([gate.to(torch.bfloat16), up], 1).contiguous()
    dgu, dw = torch.empty_like(gu), torch.empty(rows, device="cuda")
    gg.swiglu_bwd(dA, gu, w, dgu, dw, torch.tensor([rows], dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    gf, uf, a = gu[:, :Hp].float(), up.float(), dA.float()
    sig = 1 / (1 + torch.exp(-gf))
    silu, d = gf * sig, a * w[:, None]
    want = torch.cat([d * uf * sig * (1 + gf * (1 - sig)), d * silu], 1)
    # one bf16 rounding; the fast exponential is good to 2 + 1.2 |g| ulp, at most 2^-16; behind its range it ends in zero
    # where the exact one leaves a sigmoid below 2e-38, which g, up to 104, and two factors of a few multiply
    ok = (dgu.float() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-34
    both = torch.isnan(dgu.float()) & torch.isnan(want) | (dgu.float() == want)
    assert bool((ok | both).all())
    row = (a * silu * uf).sum(1)
    fin = torch.isfinite(row) & (row.abs() < 1e30)
    mag = (a * silu * uf).abs().sum(1)
    assert bool(((dw - row).abs()[fin] <= 1e-4 * mag[fin]).all()) and bool((torch.isnan(dw) | ~torch.isnan(row)).all())
