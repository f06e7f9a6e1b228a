"""Order of memory operations between kernels that may start before their predecessor ends: a kernel of this library writes an
operand, the next one reads it, the one after that overwrites it, all queued without the host between them."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TIMES = 12
# products of a few rows (streamed weights), of some (tiles), of many (pairs of CTAs), and of few features (K cut over a cluster)
FORMS = [(1, 6144, 1024), (16, 4096, 1024), (3, 96, 4096), (64, 4096, 1024), (700, 6144, 1024)]


def _chain(write, compute, contents, shape):
    """Results of ``compute`` behind each write, queued in one go behind a delay, and the same with a wait in front of every launch."""
    def run(step):
        out = [torch.empty(shape, device="cuda", dtype=torch.bfloat16) for _ in range(TIMES)]
        for i in range(TIMES):
            step()
            write(contents[i % 2])
            step()
            compute(out[i])
        torch.cuda.synchronize()
        return out

    torch.cuda.synchronize()
    want = run(torch.cuda.synchronize)
    a = torch.randn(8192, 8192, device="cuda")
    for _ in range(8):      # the queue fills while these run
        a @ a
    return run(lambda: None), want


def _operands(rows, n, k):
    g = torch.Generator(device="cuda").manual_seed(rows + n + k)
    table = (torch.randn(max(rows, n) + 1, k, device="cuda", generator=g) * k ** -0.25).bfloat16()
    ids = [torch.randint(0, len(table), (max(rows, n),), device="cuda", generator=g, dtype=torch.int32) for _ in range(2)]
    return table, ids


def _same(got, want):
    assert not torch.equal(want[0], want[1])
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and all(torch.equal(want[i], want[i % 2]) for i in range(TIMES))


@pytest.mark.parametrize("rows,n,k", FORMS)
def test_weights_written_by_the_kernel_before(rows, n, k):
    from crosspool_b200.ops import attention as A
    from crosspool_b200.ops import gemm

    table, ids = _operands(rows, n, k)
    x, w = table[:rows].clone(), torch.empty(n, k, device="cuda", dtype=torch.bfloat16)
    _same(*_chain(lambda i: A.embedding(i[:n], table, out=w), lambda y: gemm.linear(x, w, out=y), ids, (rows, n)))
    gemm.check_status(x.device)


@pytest.mark.parametrize("rows,n,k", FORMS)
def test_activations_written_by_the_kernel_before(rows, n, k):
    from crosspool_b200.ops import attention as A
    from crosspool_b200.ops import gemm

    table, ids = _operands(rows, n, k)
    w, x = table[:n].clone(), torch.empty(rows, k, device="cuda", dtype=torch.bfloat16)
    _same(*_chain(lambda i: A.embedding(i[:rows], table, out=x), lambda y: gemm.linear(x, w, out=y, w_static=True), ids, (rows, n)))
    # the summand of the epilogue
    r, wide = torch.empty(rows, n, device="cuda", dtype=torch.bfloat16), torch.randn(len(table), n, device="cuda").bfloat16()
    x = table[:rows].clone()
    _same(*_chain(lambda i: A.embedding(i[:rows], wide, out=r), lambda y: gemm.linear(x, w, out=y, resid=r, w_static=True), ids, (rows, n)))
    gemm.check_status(x.device)


@pytest.mark.parametrize("hidden", [1024, 4096])       # a row per warp, a row per CTA
def test_norm_weights_written_by_the_kernel_before(hidden):
    from crosspool_b200.ops import attention as A
    from crosspool_b200.ops import norm

    table, ids = _operands(64, 64, hidden)
    p, w = table[:33].clone(), torch.empty(1, hidden, device="cuda", dtype=torch.bfloat16)
    _same(*_chain(lambda i: A.embedding(i[:1], table, out=w), lambda y: norm.add_rmsnorm([p], w[0], out=y), ids, (33, hidden)))


def test_sampled_tokens_feed_the_next_pass():
    """Logits -> token -> embedding -> logits, as a decode step chains them."""
    from crosspool_b200.ops import attention as A
    from crosspool_b200.ops import gemm

    table, _ = _operands(8, 500, 512)
    head = table.roll(1, 0).contiguous()               # the next token is the id one on
    x = torch.empty(8, 512, device="cuda", dtype=torch.bfloat16)
    ids = torch.arange(8, device="cuda", dtype=torch.int32) * 11
    start, seen = ids.clone(), []
    a = torch.randn(8192, 8192, device="cuda")
    for _ in range(4):
        a @ a
    for _ in range(40):
        A.embedding(ids, table, out=x)
        ids = A.argmax(gemm.linear(x, head, w_static=True))
        seen.append(ids)
    assert torch.equal(torch.stack(seen), (start + 1 + torch.arange(40, device="cuda", dtype=torch.int32)[:, None]) % len(table))
