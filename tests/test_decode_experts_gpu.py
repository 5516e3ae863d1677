"""The routed units of a step of few tokens streamed by pair (csrc/expert_stream.cu), at the sizes where they can go wrong, against 64-bit
arithmetic on the same numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("units,out,k,tokens,per_token", [(3, 8, 8, 1, 2), (5, 24, 40, 3, 2), (34, 40, 264, 8, 5), (4, 56, 520, 16, 3), (64, 16, 1032, 2, 7),
                                                          (9, 136, 2048, 12, 4)])
@pytest.mark.parametrize("gated", [True, False])
def test_units_streamed_by_pair(units, out, k, tokens, per_token, gated):
    """Choices without a unit, units that more than 8 pairs share (the matrix goes over them again), fewer pairs than units and more,
    rows beyond the last tile; the score on the input or not; the squared rectifier; a second product with a row per pair."""
    from tileinfer_b200.kernels import fast
    g = torch.Generator().manual_seed(units * 1000 + k)
    x = torch.randn(tokens, k, generator=g).bfloat16()
    w = (torch.randn(units, (2 if gated else 1) * out, k, generator=g) * k ** -0.5).bfloat16()
    ids = torch.stack([torch.randperm(units, generator=g)[:per_token] if units >= per_token else torch.arange(per_token) % units for _ in range(tokens)]).int()
    ids[:, 0] = units - 1                                # one unit that every token takes
    if per_token > 2:
        ids[tokens // 2, 1] = -1
    scores = torch.rand(tokens, per_token, generator=g)
    limits = torch.full((units,), 1.5)
    pairs = tokens * per_token
    for scaled in (False, True):
        y = torch.full((pairs, out), 7.0, dtype=torch.bfloat16, device="cuda")
        rows = torch.full((tokens, per_token), 99, dtype=torch.int32, device="cuda")
        fast.grouped_stream(y, x.cuda(), w.cuda(), ids.cuda(), scores.cuda() if scaled else None, rows, per_token, gated=gated, relu2=not gated,
                            limits=limits.cuda(), slope=1.7, shift=1.0)
        assert torch.equal(rows.cpu().flatten(), torch.where(ids.flatten() >= 0, torch.arange(pairs), torch.tensor(-1)).int())
        for p in range(pairs):
            e, t = int(ids.flatten()[p]), p // per_token
            if e < 0:
                assert bool((y[p] == 7.0).all())
                continue
            row = (scores.flatten()[p] * x[t].float()).bfloat16() if scaled else x[t]
            z = w[e].to(F64) @ row.to(F64)
            # A 32-bit sum of k products off by k / 2 roundings of its terms at most, then one rounding to bfloat16.
            off = k / 2 * 2.0 ** -24 * (w[e].to(F64).abs() @ row.to(F64).abs()) + z.abs() * 2.0 ** -8
            if gated:
                a, b = z[:out].clamp(max=1.5), z[out:].clamp(-1.5, 1.5)
                want = a * torch.sigmoid(1.7 * a) * (b + 1.0)
                bound = off[:out] * 1.2 * (b + 1.0).abs() + off[out:] * a.abs()             # slopes: |d/da| <= 1.2 |b + 1|, |d/db| <= |a|
            else:
                want = torch.relu(z) ** 2
                bound = off * (2 * z.abs() + off)
            assert bool(((y[p].cpu().to(F64) - want).abs() <= bound + want.abs() * 2.0 ** -7 + 1e-6).all()), p
    down = (torch.randn(units, 24, out, generator=g) * out ** -0.5).bfloat16()
    y2, y3 = torch.zeros((pairs, 24), dtype=torch.bfloat16, device="cuda"), torch.zeros((pairs, 24), dtype=torch.bfloat16, device="cuda")
    fast.grouped_stream(y2, y, down.cuda(), ids.cuda())
    fast.grouped_stream(y3, y, down.cuda(), ids.cuda(), ahead=True)
    assert torch.equal(y2, y3)
    for p in range(pairs):
        e = int(ids.flatten()[p])
        if e >= 0:
            want = down[e].to(F64) @ y[p].cpu().to(F64)
            bound = out / 2 * 2.0 ** -24 * (down[e].to(F64).abs() @ y[p].cpu().to(F64).abs()) + want.abs() * 2.0 ** -8
            assert bool(((y2[p].cpu().to(F64) - want).abs() <= bound + 1e-7).all())


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("units,out,k,tokens,per_token", [(40, 1032, 72, 16, 2), (70, 24, 2056, 16, 4), (9, 40, 264, 16, 7), (300, 16, 40, 16, 20), (100, 16, 40, 16, 40),
                                                          (5, 4096, 40, 9, 13)])
def test_units_listed_by_warp_block_and_launch(units, out, k, tokens, per_token, gated):
    """32 pairs (listed by one warp), more, as many as a block's threads and more, and more than one launch lists; few units that many pairs chose;
    several tiles a block, and a block per unit and tile; rows longer and shorter than the k blocks in flight: every pair's result has the bits of
    the pair alone."""
    from tileinfer_b200.kernels import fast
    g = torch.Generator(device="cuda").manual_seed(units + k)
    x = torch.randn(tokens, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(units, (2 if gated else 1) * out, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    ids = torch.randint(-1, units, (tokens, per_token), generator=g, device="cuda").int()
    ids[::2, 0] = 3                                      # more than 8 pairs with one unit
    scores = torch.rand(tokens, per_token, generator=g, device="cuda")
    limits = torch.full((units,), 1.5, device="cuda")
    pairs = tokens * per_token

    def run(x, ids, scores, per_token):
        y = torch.full((ids.numel(), out), 7.0, dtype=torch.bfloat16, device="cuda")
        rows = torch.full(ids.shape, 99, dtype=torch.int32, device="cuda")
        fast.grouped_stream(y, x, w, ids, scores, rows, per_token, gated=gated, relu2=not gated, limits=limits, slope=1.7, shift=1.0)
        assert torch.equal(rows.flatten(), torch.where(ids.flatten() >= 0, torch.arange(ids.numel(), device="cuda"), -1).int())
        return y

    for s in (None, scores):
        together = run(x, ids, s, per_token)
        for p in range(pairs):
            t, j = divmod(p, per_token)
            one = run(x[t:t + 1].contiguous(), ids[t:t + 1, j:j + 1].contiguous(), s[t:t + 1, j:j + 1].contiguous() if s is not None else None, 1)
            assert torch.equal(one[0], together[p]), p


@pytest.mark.parametrize("heads,out,k", [(3, 40, 8), (16, 128, 64), (5, 24, 264), (2, 136, 2056), (64, 520, 128), (130, 264, 128)])
@pytest.mark.parametrize("n", [1, 8, 9, 16, 17])
def test_product_with_a_matrix_per_head(heads, out, k, n):
    """Streamed by head up to 16 tokens (a second pass over the matrices from 9 on), in tiles from 17 on and where the blocks would be too many;
    outputs that are no whole tiles."""
    from tileinfer_b200.kernels import fast
    g = torch.Generator(device="cuda").manual_seed(heads * 100 + n)
    x = torch.randn(n, heads, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(heads, out, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    y = torch.full((n + 1, heads, out), 7.0, dtype=torch.bfloat16, device="cuda")
    assert fast.head_linear(y[:n], x, w)
    fast.check_status()
    want, mass = (torch.einsum("hok,nhk->nho", a, b) for a, b in ((w.to(F64), x.to(F64)), (w.to(F64).abs(), x.to(F64).abs())))
    # 32-bit sums of k products in any order, then one rounding to bfloat16.
    assert bool(((y[:n].to(F64) - want).abs() <= k / 2 * 2.0 ** -24 * mass + want.abs() * 2.0 ** -8 + 1e-7).all())
    assert bool((y[n] == 7.0).all())
