"""The product's kernels against one another: operands are small multiples of 1/8, so that every order of sums gives the same fp32 sum, and the
streamed form and the pairs of CTAs must store the bits of the tiled form whatever the epilogue."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(rows, n, k, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)

    def ints(lo, hi, *shape):
        return torch.randint(lo, hi + 1, shape, device="cuda", generator=g)

    x, w = ints(-3, 3, rows, k).bfloat16(), (ints(-2, 2, n, k) / 8).bfloat16()      # |sums| <= k, multiples of 1/8: exact for k <= 4096
    return x, w, (ints(-9, 9, n) / 4).float(), (ints(-40, 40, rows, n) / 16).bfloat16()


def _run(x, w, n, rows, bn, *, f32=False, tail=0, batch=0, pitch=0, **kw):
    """One xp_gemm call; ``bn`` > 0 names a tile width, which means the tiled kernel."""
    from crosspool_b200 import native
    from crosspool_b200.ops import gemm

    relu2 = kw.pop("relu2", 0)
    out = torch.zeros(rows, n * max(1, batch) + pitch, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    kept = torch.zeros(rows, max(tail, 1), device="cuda")
    a = gemm._args(x, w, out, n_out=n, rows=rows, bn=bn, splits=1 if bn else 0, **kw)
    a.relu2 = relu2
    if tail:
        a.tail, a.tail_from, a.ld_tail = kept.data_ptr(), n - tail, tail
    if batch:
        a.batch, a.x_group_rows, a.w_rows_per_group, a.out_group_stride = batch, rows, n, n
    native.check(native.kernels().xp_gemm(C.byref(a)), "xp_gemm")
    return out, kept


def _same(x, w, n, rows, **kw):
    got, want = _run(x, w, n, rows, 0, **kw), _run(x, w, n, rows, 256 if rows > 16 and not kw.get("dual") else 128 if rows > 16 else 16, **kw)
    assert want[0].float().abs().sum() > 0
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


STREAMED, PAIRS = [(1, 200, 1032), (8, 330, 1032), (16, 1024, 1024)], [(700, 5000, 264), (1000, 6144, 1024)]


@pytest.mark.parametrize("rows,n,k", STREAMED + PAIRS)
def test_single_products(rows, n, k):
    from crosspool_b200.ops import gemm

    x, w, b, r = _operands(rows, n, k, rows + n)
    _same(x, w, n, rows, epilogue=gemm.EPI_STORE)
    _same(x, w, n, rows, epilogue=gemm.EPI_STORE, bias=b, out_scale=0.5, pitch=3)
    _same(x, w, n, rows, epilogue=gemm.EPI_STORE, bias=b, silu_cols=50)
    _same(x, w, n, rows, epilogue=gemm.EPI_STORE, relu2=1)
    _same(x, w, n, rows, epilogue=gemm.EPI_STORE, tail=7)
    _same(x, w, n, rows, epilogue=gemm.EPI_STORE_F32, f32=True, bias=b, silu_cols=33)
    _same(x, w, n, rows, epilogue=gemm.EPI_RESIDUAL, resid=r, bias=b)
    _same(x, w, n, rows, epilogue=gemm.EPI_GATE_MUL, resid=r, act_alpha=1.5, act_cubic=0.04)
    _same(x, w, n, rows, epilogue=gemm.EPI_SIGMOID, resid=r, bias=b)


# pairs of CTAs with gated tiles 128 and 256 wide
@pytest.mark.parametrize("rows,inter,k", [(1, 100, 1032), (8, 328, 512), (16, 512, 1024), (513, 3000, 896), (700, 6144, 2048)])
def test_gated_products(rows, inter, k):
    from crosspool_b200.ops import gemm

    x, w, b, _ = _operands(rows, 2 * inter, k, rows + inter)
    kw = dict(epilogue=gemm.EPI_SWIGLU, dual=1, up_offset=inter)
    _same(x, w, inter, rows, **kw)
    _same(x, w, inter, rows, bias=b, gate_limit=3.0, up_add=1.0, act_alpha=1.7, **kw)
    _same(x, w, inter, rows, bias=b, act_alpha=1.5957691216, act_cubic=0.044715, **kw)


@pytest.mark.parametrize("rows", [1, 11, 16])
def test_batched_products(rows):
    from crosspool_b200.ops import gemm

    heads, n, k = 5, 72, 136
    x, w, _, r = _operands(heads * rows, heads * n, k, rows)
    gate = r.view(rows, -1)[:, :heads * n].contiguous()
    _same(x, w, n, rows, batch=heads, epilogue=gemm.EPI_STORE)
    _same(x, w, n, rows, batch=heads, epilogue=gemm.EPI_SIGMOID, resid=gate)


@pytest.mark.parametrize("rows,n,k,dual", [(4, 19204, 4096, 0), (5, 19204, 4096, 0), (4, 19200, 4096, 0), (16, 19200, 4096, 0), (1, 9601, 4096, 1), (1, 9600, 4096, 1)])
def test_large_matrices_at_the_limits_of_the_streamed_form(rows, n, k, dual):
    """150 MB of weights, four rows, gated or not: either side of each line gives the tiled form's bits."""
    from crosspool_b200.ops import gemm

    x, w, _, _ = _operands(rows, n * (2 if dual else 1), k, rows + n)
    _same(x, w, n, rows, **(dict(epilogue=gemm.EPI_SWIGLU, dual=1, up_offset=n) if dual else dict(epilogue=gemm.EPI_STORE)))
