"""Products of at most 16 rows (the kernel that streams weights through registers) against fp32 references of the same op."""
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


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("rows", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(1, 8), (15, 40), (16, 32), (17, 64), (40, 72), (130, 896), (1024, 3072), (300, 4104), (6144, 512), (20000, 128)])
def test_plain(rows, n, k, static):
    from crosspool_b200.ops import gemm

    x, w, _ = _data(rows, n, k, rows + n + k, pad=8)
    torch.cuda.synchronize()
    want = x.float() @ w.float().t()
    _close(gemm.linear(x, w, w_static=static), want)
    assert torch.equal(gemm.linear(x, w, out_fp32=True).bfloat16(), gemm.linear(x, w))


@pytest.mark.parametrize("rows", [1, 8, 13])
def test_epilogues(rows):
    from crosspool_b200.ops import gemm

    n, k = 200, 1032
    x, w, g = _data(rows, n, k, rows)
    b = torch.randn(n, device="cuda", generator=g)
    r = torch.randn(rows, n, device="cuda", generator=g).bfloat16()
    y = x.float() @ w.float().t()
    _close(gemm.linear(x, w, bias=b, out_scale=0.5), y * 0.5 + b)
    # the product is rounded before the sum: where its order of sums flips that rounding, the sum is off by a unit of the product
    got, want = gemm.linear(x, w, resid=r).float(), y.bfloat16().float() + r.float()
    assert ((got - want).abs() <= 2.0 ** -7 * y.abs() + 2.0 ** -8 * want.abs() + 1e-5).all()
    got = gemm.linear(x, w, silu_cols=50)
    _close(got, torch.cat([torch.nn.functional.silu(y[:, :50]), y[:, 50:]], 1))
    out, tail = torch.empty(rows, n, device="cuda", dtype=torch.bfloat16), torch.empty(rows, 7, device="cuda")
    gemm.linear(x, w, out=out, tail=tail)
    _close(out[:, :n - 7], y[:, :n - 7])
    _close(tail, y[:, n - 7:])
    _close(gemm.linear_relu2(x, w, torch.empty_like(r)), y.clamp_min(0).square())
    e = gemm.linear_gate_mul(x, w, r, torch.empty_like(r), 1.5, 0.04)
    v = y.bfloat16().float()
    _close(e, v * torch.sigmoid(1.5 * v * (1 + 0.04 * v * v)) * r.float(), 3)


@pytest.mark.parametrize("rows", [1, 8, 16])
@pytest.mark.parametrize("inter,k", [(8, 64), (24, 896), (3072, 1024), (640, 4096)])
def test_gated(rows, inter, k):
    from crosspool_b200.ops import gemm

    x, w, g = _data(rows, 2 * inter, k, rows + inter)
    b = torch.randn(2 * inter, device="cuda", generator=g)
    gate, up = (x.float() @ w.float().t() + b).bfloat16().float().chunk(2, -1)
    _close(gemm.gateup_swiglu(x, w, bias=b), torch.nn.functional.silu(gate) * up, 3)
    gate, up = gate.clamp(max=1.0), up.clamp(-1.0, 1.0)
    _close(gemm.gateup_swiglu(x, w, bias=b, gate_limit=1.0, up_add=1.0, act_alpha=1.7), gate * torch.sigmoid(1.7 * gate) * (up + 1), 3)


@pytest.mark.parametrize("rows", [2, 11])
@pytest.mark.parametrize("heads,n,k", [(3, 24, 40), (16, 128, 512), (16, 512, 128)])
def test_batched_and_tiled(rows, heads, n, k):
    from crosspool_b200.ops import gemm

    g = torch.Generator(device="cuda").manual_seed(rows + heads)
    x = torch.randn(heads, rows, k, device="cuda", generator=g).bfloat16()
    w = (torch.randn(heads * n, k, device="cuda", generator=g) * k ** -0.5).bfloat16()
    gate = torch.randn(rows, heads * n, device="cuda", generator=g).bfloat16()
    want = torch.einsum("hrk,hnk->rhn", x.float(), w.view(heads, n, k).float()).reshape(rows, heads * n)
    out = torch.empty(rows, heads * n, device="cuda", dtype=torch.bfloat16)
    _close(gemm.linear_batched(x, w, out, n), want)
    _close(gemm.linear_batched(x, w, out, n, gate=gate), want * torch.sigmoid(gate.float()))
    if heads * n % 128 == 0 and k % 64 == 0:
        assert torch.equal(gemm.linear(x[0], gemm.tile_weight(w)), gemm.linear(x[0], w))


def test_refuses_what_it_refused():
    from crosspool_b200 import native
    from crosspool_b200.ops import gemm

    x, w, _ = _data(4, 64, 64, 0)
    flat = torch.zeros(4 * 64 + 1, device="cuda", dtype=torch.bfloat16)
    with pytest.raises(native.NativeLibraryError):      # rows that do not start on 16 bytes
        gemm.linear(flat[1:].view(4, 64), w)
    with pytest.raises(native.NativeLibraryError):
        gemm.linear(torch.zeros(4, 68, device="cuda", dtype=torch.bfloat16)[:, :64], w)


def _raw(x, w, n_out, w_rows_total, **kw):
    import ctypes as C

    from crosspool_b200 import native
    from crosspool_b200.ops import gemm

    out = torch.full((x.shape[0], n_out), 7.0, device="cuda", dtype=torch.bfloat16)
    a = gemm._args(x, w, out, n_out=n_out, rows=x.shape[0], epilogue=kw.pop("epilogue", gemm.EPI_STORE), **kw)
    a.w_rows_total = w_rows_total
    native.check(native.kernels().xp_gemm(C.byref(a)), "xp_gemm")
    return out


@pytest.mark.parametrize("rows", [1, 16, 17])     # 17: the tiled kernel
def test_features_without_weight_rows_are_zero(rows):
    """A caller that names fewer weight rows than features gets zeros there, whichever kernel runs; nothing is read behind them."""
    from crosspool_b200 import native
    from crosspool_b200.ops import gemm

    x, w, _ = _data(rows, 200, 256, rows)
    want = x.float() @ w.float().t()
    want[:, 130:] = 0
    _close(_raw(x, w, 200, 130), want)
    gate, up = want[:, :100].bfloat16().float(), want[:, 100:].bfloat16().float()
    _close(_raw(x, w, 100, 130, epilogue=gemm.EPI_SWIGLU, dual=1, up_offset=100), torch.nn.functional.silu(gate) * up, 3)
    tiled = gemm.tile_weight(torch.randn(256, 256, device="cuda").bfloat16())
    with pytest.raises(native.NativeLibraryError):
        _raw(x, tiled, 128, 130)
