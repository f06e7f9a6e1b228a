"""Edges of the row kernels: rows of a warp and of a CTA, rows in several CTAs' heads, rows off 4- and 16-byte boundaries, whole clusters."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("static", [False, True])
@pytest.mark.parametrize("rows,hidden", [(1, 8), (9, 1016), (7, 1024), (8, 1032), (3, 8192)])
def test_norm_rows(rows, hidden, static):
    from crosspool_b200.ops import norm

    g = torch.Generator(device="cuda").manual_seed(rows + hidden)
    p, r = (torch.randn(rows, hidden, device="cuda", generator=g).bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).bfloat16()
    torch.cuda.synchronize()
    s = (p.float() + r.float()).bfloat16()
    want = (s.float() * torch.rsqrt(s.float().square().mean(-1, keepdim=True) + 1e-6)).bfloat16().float() * w.float()
    y = norm.add_rmsnorm([p], w, 1e-6, resid=r, w_static=static)
    assert torch.equal(r, s)
    torch.testing.assert_close(y.float(), want, rtol=2.0 ** -7, atol=1e-6)      # two roundings to bf16


@pytest.mark.parametrize("rows", [591, 592])          # a warp per head; a CTA per row
@pytest.mark.parametrize("pad", [0, 1])               # odd pitches: no 4-byte loads
def test_rope_rows(rows, pad):
    from crosspool_b200.ops import attention as A

    hq, hk, d = 5, 3, 128
    g = torch.Generator(device="cuda").manual_seed(rows)
    qkv = torch.randn(rows, (hq + 2 * hk) * d + pad, device="cuda", generator=g).bfloat16()[:, :(hq + 2 * hk) * d]
    q = torch.empty(rows, hq, d, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.zeros(rows // 16 + 1, 16, hk, d, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    pos = torch.arange(rows, device="cuda", dtype=torch.int32)
    slots = pos.clone()
    slots[5] = -1
    A.rope_kv_write(qkv, q, k, v, pos, slots, q_heads=hq, kv_heads=hk, head_dim=d, theta=1e4)
    x = qkv.float().view(rows, hq + 2 * hk, d) if not pad else qkv.float().reshape(rows, hq + 2 * hk, d)
    f = 1e4 ** (-torch.arange(0, d, 2, device="cuda").double() / d)
    c, s = (t[:, None] for t in ((pos[:, None] * f).cos().float(), (pos[:, None] * f).sin().float()))
    a, b = x[..., :d // 2], x[..., d // 2:]
    rot = torch.cat([a * c - b * s, b * c + a * s], -1)
    keep = slots >= 0
    # angles are fp32: at position p they are off by p 2^-23 or so, which turns a pair by as much
    torch.testing.assert_close(q.float(), rot[:, :hq], rtol=2.0 ** -8, atol=2e-3)
    torch.testing.assert_close(k.view(-1, hk, d)[:rows][keep].float(), rot[keep][:, hq:hq + hk], rtol=2.0 ** -8, atol=2e-3)
    assert torch.equal(v.view(-1, hk, d)[:rows][keep].float(), x[keep][:, hq + hk:]) and not k.view(-1, hk, d)[5].any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("vocab", [1, 7, 8, 2049, 151936])
def test_argmax_rows(vocab, dtype):
    from crosspool_b200.ops import attention as A

    x = torch.randn(9, vocab, device="cuda", generator=torch.Generator(device="cuda").manual_seed(vocab)).to(dtype)
    x[1] = -float("inf")
    x[2, vocab // 2] = x[2, vocab - 1] = float("inf")      # ties go to the lower id
    want = torch.stack([(r == r.max()).nonzero()[0, 0] for r in x]).int()
    assert torch.equal(A.argmax(x), want)


@pytest.mark.parametrize("vocab", [1, 64, 1000])
def test_argmax_of_short_rows_back_to_back(vocab):
    """Rows that a cluster scans in no time, more clusters than the GPU holds, launches one behind the other: a CTA's winners go to
    the first CTA of its cluster only once that has started."""
    from crosspool_b200.ops import attention as A

    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = torch.randn(3000, vocab, device="cuda", generator=g)
    want = x.argmax(-1).int()          # no ties: 3000 x 1000 draws of 24-bit normals, checked below
    assert ((x == x.max(-1, keepdim=True).values).sum(-1) == 1).all()
    torch.cuda.synchronize()
    got = [A.argmax(x) for _ in range(50)]
    assert all(torch.equal(t, want) for t in got)


@pytest.mark.parametrize("hidden", [248, 256, 264, 512, 520, 1024, 2040, 2048, 2056, 4096, 4104, 8184])      # pieces a thread holds: 1, 2, 4
@pytest.mark.parametrize("parts", [1, 2, 4])
def test_norm_forms_store_the_same_bits(hidden, parts):
    """Rows of one part, rows of several and rows that a flag guards go through different kernels; sums are in the same order."""
    from crosspool_b200.ops import norm

    g = torch.Generator(device="cuda").manual_seed(hidden + parts)
    p = [torch.randn(21, hidden, device="cuda", generator=g).bfloat16() for _ in range(parts)]
    w = (1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).bfloat16()
    r = torch.randn(21, hidden, device="cuda", generator=g).bfloat16()
    ready = torch.ones(8, device="cuda", dtype=torch.int32)
    torch.cuda.synchronize()
    got_r, want_r = r.clone(), r.clone()
    got = norm.add_rmsnorm(p, w, 1e-6, resid=got_r)
    want = norm.add_rmsnorm(p, w, 1e-6, resid=want_r, wait_flag_ptrs=[ready.data_ptr()] * parts, wait_seq=1)
    assert torch.equal(got, want) and torch.equal(got_r, want_r)
    s = (sum(t.float() for t in p).bfloat16().float() if parts > 1 else p[0].float()) + r.float()
    assert torch.equal(got_r, s.bfloat16())


# a cluster of 8, 4 or 2 CTAs a row, a CTA of 256, 512 or 1024 threads; the winner in any of their parts, ties between parts
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows", [1, 32, 33, 64, 65, 300])
@pytest.mark.parametrize("vocab", [1000, 4096, 8200, 20000, 32768, 33001])
def test_argmax_forms(vocab, rows, dtype):
    from crosspool_b200.ops import attention as A

    g = torch.Generator(device="cuda").manual_seed(vocab + rows)
    x = torch.rand(rows, vocab, device="cuda", generator=g).to(dtype)
    at = torch.randint(0, vocab, (rows,), device="cuda", generator=g)
    x[torch.arange(rows, device="cuda"), at] = 2
    x[torch.arange(rows, device="cuda"), (at + vocab // 3) % vocab] = 2
    assert torch.equal(A.argmax(x), torch.minimum(at, (at + vocab // 3) % vocab).int())
