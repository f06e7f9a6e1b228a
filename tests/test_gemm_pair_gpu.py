"""Products of many rows (pairs of CTAs) against fp32 references of the same op."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _data(rows, n, k, seed, pad=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(rows, k + pad, device="cuda", generator=g).bfloat16()[:, :k]
    w = (torch.randn(n, k + pad, device="cuda", generator=g) * k ** -0.5).bfloat16()[:, :k]
    return x, w, g


def _close(got, want, roundings=1):
    # a bf16 result is off by at most 2^-9 of its value per rounding, the fp32 sums by far less (k 2^-24 of their terms)
    torch.testing.assert_close(got.float(), want.float(), rtol=roundings * 2.0 ** -8, atol=2e-3)


# whole and partial tiles of 256 features (the second CTA of a pair without any), partial row tiles, K below and past the stages
@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("rows,n,k", [(257, 24576, 64), (400, 11400, 72), (512, 11264, 1000), (1000, 2944, 256), (1023, 4001, 520), (4096, 1024, 1024)])
def test_plain(rows, n, k, static):
    from crosspool_b200.ops import gemm

    x, w, g = _data(rows, n, k, rows + n + k, pad=8)
    b = torch.randn(n, device="cuda", generator=g)
    torch.cuda.synchronize()
    want = x.float() @ w.float().t()
    _close(gemm.linear(x, w, w_static=static), want)
    _close(gemm.linear(x, w, bias=b, out_scale=0.5, w_static=static), 0.5 * want + b)
    gemm.check_status(x.device)


def test_epilogues():
    from crosspool_b200.ops import gemm

    rows, n, k = 700, 5000, 264
    x, w, g = _data(rows, n, k, 3)
    r = torch.randn(rows, n, device="cuda", generator=g).bfloat16()
    y = x.float() @ w.float().t()
    # the product is rounded before the sum: where its order of sums flips that rounding, the sum is off by a unit of the product
    got, want = gemm.linear(x, w, resid=r).float(), y.bfloat16().float() + r.float()
    assert ((got - want).abs() <= 2.0 ** -7 * y.abs() + 2.0 ** -8 * want.abs() + 1e-5).all()
    _close(gemm.linear(x, w, out_fp32=True), y)
    _close(gemm.linear(x, w, silu_cols=50), torch.cat([torch.nn.functional.silu(y[:, :50]), y[:, 50:]], 1))
    out, tail = torch.empty(rows, n, device="cuda", dtype=torch.bfloat16), torch.empty(rows, 7, device="cuda")
    gemm.linear(x, w, out=out, tail=tail)
    _close(out[:, :n - 7], y[:, :n - 7])
    _close(tail, y[:, n - 7:])
    _close(gemm.linear_relu2(x, w, torch.empty_like(r)), y.clamp_min(0).square())
    v = y.bfloat16().float()
    _close(gemm.linear_gate_mul(x, w, r, torch.empty_like(r), 1.5, 0.04), v * torch.sigmoid(1.5 * v * (1 + 0.04 * v * v)) * r.float(), 3)
    odd = torch.zeros(rows, n + 3, device="cuda", dtype=torch.bfloat16)[:, :n]      # rows that 16-byte stores cannot address
    _close(gemm.linear(x, w, out=odd), y)
    gemm.check_status(x.device)


@pytest.mark.parametrize("rows,inter,k", [(300, 12288, 64), (513, 3000, 896), (700, 6144, 2048), (1100, 2304, 4096), (2049, 1000, 2056)])
def test_gated(rows, inter, k):
    from crosspool_b200.ops import gemm

    x, w, g = _data(rows, 2 * inter, k, rows + inter)
    b = torch.randn(2 * inter, device="cuda", generator=g)
    gate, up = (x.float() @ w.float().t() + b).bfloat16().float().chunk(2, -1)
    # the gate and up values are rounded in their own order of sums: one more unit in the last place of each
    _close(gemm.gateup_swiglu(x, w, bias=b), torch.nn.functional.silu(gate) * up, 4)
    gemm.check_status(x.device)


def test_repeated_calls_are_bitwise_stable():
    from crosspool_b200.ops import gemm

    x, w, _ = _data(1500, 6144, 1024, 9)
    first = gemm.linear(x, w)
    for _ in range(5):
        assert torch.equal(gemm.linear(x, w), first)
