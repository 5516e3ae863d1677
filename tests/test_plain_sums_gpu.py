"""The 32-bit path's product and attention at the sizes where their kernels change over: edges of tiles, of k segments and of key
chunks, and that the bits depend on none of it."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tileinfer_b200.kernels import ops
    return ops


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("out,k", [(15, 8), (33, 504), (100, 512), (2000, 520), (5000, 1032), (4100, 2056), (260, 8 * 1037)])
def test_product_bits_do_not_depend_on_the_kernel(ops, dtype, out, k):
    """Weight streaming by 1 to 64 tokens (16 or 32 rows a block, shallow or deep rings), tiles, and rows that cannot be
    read 16 bytes at a time (staged in smaller pieces): one order of additions, so one set of bits."""
    g = torch.Generator().manual_seed(out + k)
    x = torch.randn(700, k, generator=g).to(dtype).cuda()
    w = (torch.randn(out, k, generator=g) * k ** -0.5).to(dtype).cuda()
    odd = torch.zeros(700, k + 1, dtype=dtype, device="cuda")
    odd[:, :k] = x
    want = x.double() @ w.double().t()
    # Two chains of 256 terms, their sum, and the segments' sums one after the other: so many roundings of partial sums.
    bound = (min(k, 512) / 2 + 1 + k / 512) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().t())
    first = None
    for n in (700, 300, 129, 128, 65, 64, 33, 32, 17, 16, 9, 8, 5, 4, 3, 2, 1):
        for rows in (x[:n], odd[:n, :k]):
            y = torch.full((n, out), float("nan"), dtype=torch.float32, device="cuda")
            ops.gemm_plain(y, rows, w, ops.EPI_F32_OUT)
            if first is None:
                first = y
                if dtype == torch.float32:
                    assert bool(((y.double() - want).abs() <= bound).all())
                else:                                    # one rounding to bfloat16 on top
                    assert bool(((y.double() - want).abs() <= bound + want.abs() * 2.0 ** -8).all())
            assert torch.equal(y, first[:n]), (n, rows.stride(0))


@pytest.mark.parametrize("D,nq,nkv", [(4, 3, 3), (20, 5, 1), (33, 4, 2), (64, 8, 1), (96, 4, 4), (128, 12, 2), (132, 2, 1), (256, 4, 2), (512, 2, 2)])
def test_attention_over_chunk_edges(ops, D, nq, nkv):
    """Positions on both sides of the 256-key chunks, alone and in one launch (the same bits), against 64-bit arithmetic; without a
    window, with one, with kept first positions, and in chunks of visibility."""
    page, last = 16, 800
    g = torch.Generator().manual_seed(D)
    pages = -(-last // page)
    k, v = (torch.randn(pages + 3, nkv, page, D, generator=g).cuda() for _ in range(2))
    order = torch.randperm(pages + 3, generator=g)[:pages]
    table = torch.zeros(2, pages, dtype=torch.int32)
    table[1] = order.int()
    table = table.cuda()
    positions = [0, 1, 30, 31, 32, 255, 256, 257, 511, 512, 600, 799]
    q = torch.randn(len(positions), nq, D, generator=g).cuda()
    keys, values = (c[order.cuda()].permute(0, 2, 1, 3).reshape(-1, nkv, D).double() for c in (k, v))
    scale = D ** -0.5
    for window, keep, chunk in ((0, 0, 0), (70, 0, 0), (300, 40, 0), (0, 0, 100)):
        def run(rows):
            pos = torch.tensor([positions[r] for r in rows], dtype=torch.int32, device="cuda")
            out = torch.empty(len(rows), nq * D, device="cuda")
            ops.attention_plain(out, q[rows].contiguous(), k, v, table, torch.ones_like(pos), pos, scale, nq, nkv, D, page, window, chunk=chunk, keep=keep)
            return out.view(len(rows), nq, D)
        together = run(list(range(len(positions))))
        for r, p in enumerate(positions):
            seen = torch.arange(p + 1, device="cuda")
            low = max(p + 1 - window if window else 0, p // chunk * chunk if chunk else 0)
            seen = seen[(seen >= low) | (seen < keep)] if window else seen[seen >= low]
            for h in range(nq):
                s = (keys[seen, h // (nq // nkv)] @ q[r, h].double()) * scale
                want = torch.softmax(s, 0) @ values[seen, h // (nq // nkv)]
                # Roundings: the score's D products scaled (its error enters as a factor), an exponential and a sum over the keys.
                size = float((q[r, h].abs().double() @ keys[seen, h // (nq // nkv)].abs().t()).max()) * scale
                bound = 2.0 ** -24 * (2 * D * size + 4 * math.sqrt(len(seen)) + 16) * float(values.abs().max())
                assert float((together[r, h].double() - want).abs().max()) <= bound, (p, h, window)
            assert torch.equal(run([r])[0], together[r])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D,nq,nkv", [(4, 3, 3), (33, 4, 2), (64, 10, 2), (100, 4, 2), (128, 4, 4), (128, 12, 2), (132, 3, 3), (192, 4, 2), (256, 6, 2), (260, 2, 2),
                                      (512, 4, 2), (512, 5, 1)])
def test_attention_of_many_tokens_has_the_bits_of_few(ops, dtype, D, nq, nkv):
    """A launch of many blocks takes the kernels that put more of them on an SM, with fewer loads in flight each: the same bits as in launches
    of few, for sets of one, two and up to four heads."""
    from tileinfer_b200.kernels import fast
    page, last = 16, 300
    g = torch.Generator(device="cuda").manual_seed(D + nq)
    pages = -(-last // page)
    k, v = (torch.randn(pages, nkv, page, D, generator=g, device="cuda").to(dtype) for _ in range(2))
    table = torch.randperm(pages, generator=g, device="cuda").int()[None]
    n = 3 * fast.sm_count() + 1                          # a block per token, KV head and set
    positions = torch.randint(0, last, (n,), generator=g, device="cuda").int()
    q = torch.randn(n, nq, D, generator=g, device="cuda").to(dtype)

    def run(lo, hi):
        out = torch.empty(hi - lo, nq * D, dtype=dtype, device="cuda")
        pos = positions[lo:hi].contiguous()
        ops.attention_plain(out, q[lo:hi].contiguous(), k, v, table, torch.zeros_like(pos), pos, D ** -0.5, nq, nkv, D, page)
        return out

    together = run(0, n)
    for lo in range(0, n, 37):
        hi = min(n, lo + 37)
        assert torch.equal(run(lo, hi), together[lo:hi]), lo


def test_attention_beyond_two_to_the_31_rows(ops):
    """A pool of one-element heads with more rows than a 32-bit integer counts: a sequence whose pages lie at its end gets what the same
    keys and values give in a pool of their own."""
    page, nkv, nq, keys = 16, 2, 4, 300
    g = torch.Generator().manual_seed(31)
    used = -(-keys // page)
    k, v = (torch.randn(used, nkv, page, 1, generator=g).bfloat16().cuda() for _ in range(2))
    q = torch.randn(3, nq, 1, generator=g).bfloat16().cuda()
    positions = torch.tensor([0, 255, keys - 1], dtype=torch.int32, device="cuda")

    def run(k_pool, v_pool, first):
        table = torch.arange(first, first + used, dtype=torch.int32, device="cuda")[None]
        out = torch.empty(3, nq, dtype=torch.bfloat16, device="cuda")
        ops.attention_plain(out, q, k_pool, v_pool, table, torch.zeros_like(positions), positions, 1.0, nq, nkv, 1, page)
        return out

    want = run(k, v, 0)
    pages = 2 ** 31 // (nkv * page) + used                # 4.3 GB each; only the last pages are written and read
    k_pool, v_pool = (torch.empty(pages, nkv, page, 1, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    k_pool[-used:], v_pool[-used:] = k, v
    assert torch.equal(run(k_pool, v_pool, pages - used), want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k", [40, 1031, 1042, 1544])      # one segment; an odd k; 2 modulo 8; several segments and a part of one, in 16-byte rows
def test_every_tile_shape_and_width_of_copy(ops, dtype, k):
    """Tiles of every shape with ragged edges, and steps of few tokens, with the operands' rows on 16 bytes, on 4, and on single elements:
    one order of additions, so the bits of a token alone in rows of 16 bytes, and its distance to 64-bit sums."""
    from tileinfer_b200.kernels import fast, lib
    choose = lib().handle.ti_gemm_plain_shape
    sizes = [(500, 4090), (390, 1999), (250, 2001), (100, 333), (1, 50), (7, 333), (13, 2001), (61, 100)]
    assert {choose(n, out, fast.sm_count()) for n, out in sizes[:4]} == {0, 1, 2, 3}
    g = torch.Generator(device="cuda").manual_seed(k)
    wide = -(-k // 8) * 8                                  # the same k terms and zeros, in rows of 16 bytes
    for n, out in sizes:
        x = torch.zeros(n, wide, device="cuda", dtype=dtype)
        w = torch.zeros(out, wide, device="cuda", dtype=dtype)
        x[:, :k] = torch.randn(n, k, generator=g, device="cuda")
        w[:, :k] = torch.randn(out, k, generator=g, device="cuda") * k ** -0.5
        want = torch.empty(n, out, device="cuda")
        for t in range(n):
            ops.gemm_plain(want[t:t + 1], x[t:t + 1], w, ops.EPI_F32_OUT)
        exact, mass = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
        bound = (min(k, 512) / 2 + 1 + k / 512) * 2.0 ** -24 * mass + (exact.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
        assert bool(((want.double() - exact).abs() <= bound).all())
        narrow = w[:, :k].contiguous()
        for pad, base in ((0, 0), (1, 0), (2, 0), (8, 0), (8, 1), (8, 2)):      # the tokens' row pitch beyond k, and the first row's place
            store = torch.full((base + n * (k + pad),), float("nan"), dtype=dtype, device="cuda")
            rows = store[base:].view(n, k + pad)[:, :k]
            rows.copy_(x[:, :k])
            y = torch.full((n + 1, out), 7.0, device="cuda")
            ops.gemm_plain(y[:n], rows, narrow, ops.EPI_F32_OUT)
            assert torch.equal(y[:n], want), (n, out, pad, base)
            assert bool((y[n] == 7.0).all())
