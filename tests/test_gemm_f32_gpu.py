"""The fp32 product against 64 bits at the edges of its forms: one to eight rows (streamed), row tiles of 16, 32 and 64 rows,
partial feature tiles and K slices, pitches and bases that are not multiples of 16 bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(out, x, w, extra=0.0):
    ref = x.double() @ w.double().t() + extra
    # every term is rounded once and the sum at most k times: k eps |x| |w| bounds it, far from reached
    bound = (x.double().abs() @ w.double().abs().t()) * (x.shape[1] ** 0.5 + 8) * 2.0 ** -24 + 1e-6
    assert ((out.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 64, 65, 300])
@pytest.mark.parametrize("n,k", [(1, 4), (70, 36), (129, 130), (1000, 1024), (64, 2052), (4096, 260)])
def test_fp32_product_against_64_bits(rows, n, k):
    from crosspool_b200.ops import gemm

    g = torch.Generator(device="cuda").manual_seed(rows * 131 + n + k)
    x, w = (torch.randn(*s, device="cuda", generator=g) for s in ((rows, k), (n, k)))
    bias = torch.randn(n, device="cuda", generator=g)
    _check(gemm.linear(x, w, bias=bias), x, w, bias.double())


@pytest.mark.parametrize("rows", [3, 20])
@pytest.mark.parametrize("pad,shift", [(1, 0), (4, 1), (4, 4)])
def test_fp32_product_takes_any_pitch_and_base(rows, pad, shift):
    from crosspool_b200.ops import gemm

    n, k = 96, 200
    x = torch.randn(rows, k + pad + shift, device="cuda")[:, shift:shift + k]
    w = torch.randn(n, k + pad + shift, device="cuda")[:, shift:shift + k]
    out = torch.full((rows, n + 3), 7.0, device="cuda")
    gemm.linear(x, w, out=out[:, :n], silu_cols=0)
    _check(out[:, :n], x, w)
    assert (out[:, n:] == 7.0).all()


@pytest.mark.parametrize("rows", [2, 40])
def test_fp32_batched_product_and_silu(rows):
    from crosspool_b200.ops import gemm

    groups, n, k = 5, 72, 64
    x, w = torch.randn(groups, rows, k, device="cuda"), torch.randn(groups * n, k, device="cuda")
    out = torch.empty(rows, groups * n, device="cuda")
    gemm.linear_batched(x, w, out, n)
    for i in range(groups):
        _check(out[:, i * n:(i + 1) * n], x[i], w[i * n:(i + 1) * n])
    y = gemm.linear(x[0], w, silu_cols=100)
    ref = x[0].double() @ w.double().t()
    ref[:, :100] = torch.nn.functional.silu(ref[:, :100])
    torch.testing.assert_close(y.double(), ref, rtol=1e-5, atol=1e-5)
