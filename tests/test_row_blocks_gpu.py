"""Row kernels whose blocks depend on how many rows a step has, and the recurrences' scans beside their one-token kernels: a row's bits do not
depend on the step it is in. Their distance to 64-bit arithmetic is measured where the kernels are tested alone (test_fasodra_gpu.py)."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from tileinfer_b200.kernels import ops
    return ops


def _step(lengths, slots=None):
    cu = torch.tensor([0] + lengths).cumsum(0).int().cuda()
    return SimpleNamespace(cu_seqlens=cu, seq_slots=torch.tensor(slots or list(range(len(lengths)))).int().cuda(), n_seqs=len(lengths))


@pytest.mark.parametrize("size", [96, 1000, 1024, 2048, 4096, 5000])
@pytest.mark.parametrize("streams", [1, 2, 3, 8])
def test_stream_rows_in_small_and_large_steps(ops, size, streams):
    g = torch.Generator(device="cuda").manual_seed(size + streams)
    n = 400                                                # more rows than SMs
    R = lambda *s, dtype=torch.float32: torch.randn(*s, generator=g, device="cuda").to(dtype)     # noqa: E731
    x, delta, parts = R(n, streams * size), R(n, size, dtype=torch.bfloat16), R(3, n, size)
    w, b = R(size, dtype=torch.bfloat16), R(size, dtype=torch.bfloat16)
    mix, out, blend = ([0.3 + 0.1 * i for i in range(c)] for c in (streams * streams, streams, streams))
    a = torch.tensor(blend, device="cuda")

    def run(lo, hi):
        got = []
        for d in (delta[lo:hi].contiguous(), parts[:, lo:hi].contiguous()):
            for centred in (True, False):
                xs, h = x[lo:hi].clone(), torch.empty(hi - lo, size, dtype=torch.bfloat16, device="cuda")
                ops.streams_update(xs, d, mix, out, blend, h, w, b, 1e-6, centred)
                got += [xs, h]
        h = torch.empty(hi - lo, size, dtype=torch.bfloat16, device="cuda")
        ops.streams_read_norm(h, x[lo:hi].contiguous(), a, w, b, 1e-6)
        pairs = torch.empty(hi - lo, size, device="cuda")
        ops.pair_combine(pairs, delta[lo:hi].contiguous(), parts[:, lo:hi].contiguous(), w, b, 1e-6, 0.5, 2.0, torch.bfloat16)
        return got + [h, pairs]

    whole = run(0, n)
    want = torch.einsum("st,nsc->ntc", torch.tensor(mix).view(streams, streams).double().cuda(), x.double().view(n, streams, size))
    want = (want + torch.tensor(out).double().cuda()[:, None] * delta.double()[:, None, :]).reshape(n, -1)
    assert float((whole[0].double() - want).abs().max()) <= 16 * 2.0 ** -24 * float(want.abs().max())
    for lo, hi in ((0, 1), (3, 7), (100, 248)):
        for one, all_ in zip(run(lo, hi), whole):
            assert torch.equal(one, all_[lo:hi]), (lo, hi)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("W,K", [(40, 1), (257, 5), (2048, 5), (1024, 10)])
def test_blends_in_runs_of_tokens(ops, dtype, W, K):
    """Eight tokens a block and one: sequences that begin and end inside a run, rows before the step's first from the state."""
    g = torch.Generator(device="cuda").manual_seed(W)
    lengths = [1, 3, 900, 2, 7, 300, 1]
    n, slots = sum(lengths), [4, 0, 6, 2, 1, 3, 5]
    h = torch.randn(n, W, generator=g, device="cuda").to(dtype)
    mu = torch.randn(K, W, generator=g, device="cuda").to(dtype)
    prev = torch.randn(7, W, generator=g, device="cuda")

    def run(cuts):
        state, out = prev.clone(), torch.empty(K, n, W, dtype=dtype, device="cuda")
        for first, last in zip(cuts, cuts[1:]):              # sequences first .. last - 1 in one step
            lo, hi = sum(lengths[:first]), sum(lengths[:last])
            piece = torch.empty(K, hi - lo, W, dtype=dtype, device="cuda")
            ops.shift_blend(piece, h[lo:hi].contiguous(), mu, state, _step(lengths[first:last], slots[first:last]))
            out[:, lo:hi] = piece
        return out, state

    whole, state = run([0, 7])
    apart, state_apart = run([0, 2, 3, 5, 6, 7])
    assert torch.equal(whole, apart) and torch.equal(state, state_apart)
    at = 0
    for length, slot in zip(lengths, slots):
        rows = h[at:at + length].double()
        before = torch.cat([prev[slot].double()[None], rows[:-1]])
        want = rows[None] + (before - rows)[None] * mu.double()[:, None, :]
        bound = (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22) * float(want.abs().max())
        assert float((whole[:, at:at + length].double() - want).abs().max()) <= bound
        assert torch.equal(state[slot], h[at + length - 1].float())
        at += length


@pytest.mark.parametrize("taps", [0, 1, 3, 4, 7])
@pytest.mark.parametrize("G,D,HV", [(1, 24, 40), (3, 128, 384), (2, 300, 64), (4, 64, 1000)])
def test_delta_inputs_in_runs_of_tokens(ops, taps, G, D, HV):
    g = torch.Generator(device="cuda").manual_seed(D + taps)
    C, lengths = 2 * G * D + HV, [2, 2000, 1, 5]
    n, slots = sum(lengths), [2, 0, 3, 1]
    proj = torch.randn(n, C, generator=g, device="cuda").bfloat16()
    conv = torch.randn(C, max(1, taps), generator=g, device="cuda").bfloat16()
    hist = torch.randn(4, max(1, taps - 1) * C, generator=g, device="cuda")
    whole = torch.empty(n, C, device="cuda")
    ops.delta_inputs(whole, proj, conv, taps, hist, _step(lengths, slots), G, D, HV, 1e-6)
    at = 0
    for length, slot in zip(lengths, slots):
        rows = min(length, 40)                             # few tokens: one a block
        part = torch.empty(rows, C, device="cuda")
        ops.delta_inputs(part, proj[at:at + rows].contiguous(), conv, taps, hist, _step([rows], [slot]), G, D, HV, 1e-6)
        assert torch.equal(part, whole[at:at + rows])
        older = hist[slot, :max(0, taps - 1) * C].double().view(-1, C)
        x = torch.cat([older, proj[at:at + length].double()])
        y = x if taps == 0 else sum(conv[:, k].double() * x[k:k + length] for k in range(taps))
        y = y * torch.sigmoid(y)
        heads = y[:, :2 * G * D].view(length, 2 * G, D)
        heads = heads / torch.sqrt((heads * heads).sum(-1, keepdim=True) + 1e-6)
        heads[:, :G] *= D ** -0.5
        want = torch.cat([heads.reshape(length, -1), y[:, 2 * G * D:]], 1)
        # Sums of up to 7 products, an exponential, and sums over a head.
        assert float((whole[at:at + length].double() - want).abs().max()) <= 2.0 ** -24 * 64 * max(1.0, float(y.abs().max()))
        at += length


def test_rows_of_steps_with_sequences_without_tokens(ops):
    """As many sequences as tokens, some with none and some with several: the rows before are each sequence's own."""
    g = torch.Generator(device="cuda").manual_seed(5)
    W, G, D, HV, taps = 96, 1, 24, 48, 4
    for lengths in ([0, 2], [2, 0], [1, 0, 0, 3], [1, 2, 0, 1]):
        n, B = sum(lengths), len(lengths)
        h, mu = torch.randn(n, W, generator=g, device="cuda"), torch.randn(2, W, generator=g, device="cuda")
        prev, hist = torch.randn(B, W, generator=g, device="cuda"), torch.randn(B, (taps - 1) * W, generator=g, device="cuda")
        conv = torch.randn(W, taps, generator=g, device="cuda")
        state, out, rows = prev.clone(), torch.empty(2, n, W, device="cuda"), torch.empty(n, W, device="cuda")
        ops.shift_blend(out, h, mu, state, _step(lengths))
        ops.delta_inputs(rows, h, conv, taps, hist, _step(lengths), G, D, HV, 1e-6)
        at = 0
        for b, length in enumerate(lengths):
            if not length:
                assert torch.equal(state[b], prev[b])
                continue
            own = prev[b:b + 1].clone()
            one, part = torch.empty(2, length, W, device="cuda"), torch.empty(length, W, device="cuda")
            ops.shift_blend(one, h[at:at + length].contiguous(), mu, own, _step([length]))
            ops.delta_inputs(part, h[at:at + length].contiguous(), conv, taps, hist[b:b + 1].contiguous(), _step([length]), G, D, HV, 1e-6)
            assert torch.equal(out[:, at:at + length], one) and torch.equal(state[b], own[0]) and torch.equal(rows[at:at + length], part)
            at += length


@pytest.mark.parametrize("G,D,HV", [(0, 0, 300), (2, 0, 1000), (0, 24, 40), (0, 0, 0)])
def test_delta_inputs_without_heads(ops, G, D, HV):
    """Values alone: no head to norm, and none to divide a block's channels by."""
    proj = torch.randn(5, HV, generator=torch.Generator(device="cuda").manual_seed(HV), device="cuda")
    out = torch.empty(5, HV, device="cuda")
    ops.delta_inputs(out, proj, None, 0, None, _step([5]), G, D, HV, 1e-6)
    want = proj.double() * torch.sigmoid(proj.double())
    assert HV == 0 or float((out.double() - want).abs().max()) <= 2.0 ** -20 * float(want.abs().max())


@pytest.mark.parametrize("n,G,D,HV", [(1500, 1, 1534, 0), (1500, 1, 1536, 8), (1500, 1, 1540, 8), (3, 1, 12288, 0)])
def test_delta_inputs_of_rows_at_the_shared_memory_limit(ops, n, G, D, HV):
    """A block's rows and its table of tokens fill 48 KB, or a little less or more."""
    g = torch.Generator(device="cuda").manual_seed(D)
    proj = torch.randn(n, 2 * G * D + HV, generator=g, device="cuda").bfloat16()
    out = torch.empty(n, 2 * G * D + HV, device="cuda")
    ops.delta_inputs(out, proj, None, 0, None, _step([n]), G, D, HV, 1e-6)
    y = proj.double() * torch.sigmoid(proj.double())
    heads = y[:, :2 * G * D].view(n, 2 * G, D)
    heads = heads / torch.sqrt((heads * heads).sum(-1, keepdim=True) + 1e-6)
    heads[:, :G] *= D ** -0.5
    want = torch.cat([heads.reshape(n, -1), y[:, 2 * G * D:]], 1)
    # An exponential, a quotient, and a head's sum of squares: 2^-24 for each of its D / 32 additions in a row.
    assert float((out.double() - want).abs().max()) <= 2.0 ** -24 * (16 + D / 32) * float(y.abs().max())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [2, 300])
@pytest.mark.parametrize("fill", [11900, 12256, 12288, 12352])
def test_rows_that_fill_the_shared_memory_a_launch_may_have_unasked(ops, dtype, n, fill):
    """Kernels that keep ``fill`` floats of a row, or of two rows, in dynamic shared memory beside their static arrays, around 48 KB."""
    g = torch.Generator(device="cuda").manual_seed(fill + n)
    R = lambda *s, dtype=dtype: torch.randn(*s, generator=g, device="cuda").to(dtype)             # noqa: E731
    rms = lambda t: t / torch.sqrt((t * t).mean(-1, keepdim=True) + 1e-6)                          # noqa: E731
    step_of = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0

    def close(got, want, rounded):
        # Sums of squares over a row, a root, a quotient and a few products; where the result is of the element type, one rounding more.
        assert float(((got.double() - want).abs() - (step_of if rounded else 0.0) * want.abs()).max()) <= 2.0 ** -18 * float(want.abs().max())

    for op in ("streams", "branch", "sum"):
        x, d, w, w2, h = R(n, fill, dtype=torch.float32), R(n, fill), R(fill), R(fill), torch.empty(n, fill, dtype=dtype, device="cuda")
        was, D = x.double(), d.double()
        if op == "streams":
            ops.streams_read_norm(h, x, torch.ones(1, device="cuda"), w, None, 1e-6, centred=False)
            close(h, rms(was) * w.double(), True)
            ops.streams_update(x, d, [0.5], [2.0], [1.0], h, w, None, 1e-6, centred=False)
            want = 0.5 * was + 2.0 * D
        elif op == "branch":
            ops.branch_norm_add32(x, d, w2, 1e-6, 0.5, h=h, out_norm=(w, 1e-6, False))
            want = was + 0.5 * rms(D) * w2.double()
        else:
            ops.sum_add_norm32(x, d, None, h, w, 1e-6)
            want = was + D
        close(x, want, False)
        close(h, rms(want) * w.double(), True)
    half = fill // 2
    a, b, wa, wb, w, out = R(n, half), R(n, half), R(half), R(half), R(half), torch.empty(n, half, device="cuda")
    pair = 0.5 * rms(a.double()) * wa.double() + 2.0 * rms(b.double()) * wb.double()
    ops.pair_combine(out, a, b, wa, wb, 1e-6, 0.5, 2.0, dtype)
    close(out, pair, False)
    x, h = R(n, half, dtype=torch.float32), torch.empty(n, half, dtype=dtype, device="cuda")
    want = x.double() + pair
    ops.pair_add_norm32(x, a, b, wa, wb, 0.5, 2.0, 1e-6, 1.0, h, w, 1e-6)
    close(x, want, False)
    close(h, rms(want) * w.double(), True)
    rows, q = R(n, fill), torch.empty(n, fill // 4, 4, dtype=dtype, device="cuda")
    step = _step([n])
    step.positions, step.kv_lens = torch.arange(n, device="cuda").int(), torch.tensor([n], device="cuda").int()
    ops.conv_attention_inputs(rows, None, None, 0, None, None, None, 1e-6, None, q, None, None, step, None, fill // 4, 1, 4, 4, 4, 64, write_kv=False)
    assert torch.equal(q.view(n, fill), rows)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("size", [40, 1000, 2048, 4100, 9000, 12032, 12036, 12252, 12256, 12288, 12292])
def test_gated_rows_of_the_lightning_mixer_in_small_and_large_steps(ops, dtype, size):
    g = torch.Generator(device="cuda").manual_seed(size)
    n = 300                                                # more rows than SMs
    o, w = torch.randn(n, size, generator=g, device="cuda"), torch.randn(size, generator=g, device="cuda").to(dtype)
    gate = torch.randn(n, size, generator=g, device="cuda").to(dtype)
    for z in (gate, None):
        def run(lo, hi):
            y = torch.empty(hi - lo, size, dtype=dtype, device="cuda")
            ops.lightning_out(y, o[lo:hi].contiguous(), z[lo:hi] if z is not None else None, w, 1e-6)
            return y

        whole = run(0, n)
        want = o.double() / torch.sqrt((o.double() ** 2).mean(-1, keepdim=True) + 1e-6) * w.double() * (torch.sigmoid(z.double()) if z is not None else 1.0)
        # A sum of squares, a root, a quotient, an exponential; one rounding to the element type.
        assert bool(((whole.double() - want).abs() <= want.abs() * ((2.0 ** -8 if dtype == torch.bfloat16 else 0) + 2.0 ** -18) + 1e-9).all())
        for lo, hi in ((0, 1), (5, 9), (100, 248)):
            assert torch.equal(run(lo, hi), whole[lo:hi])


@pytest.mark.parametrize("tile", [32, 128])
@pytest.mark.parametrize("n,per,units", [(1, 1, 1), (3, 2, 40), (2048, 6, 34), (1500, 8, 1000), (5000, 4, 65)])
def test_plan_of_units(ops, n, per, units, tile):
    """Up to as many pairs as the threads keep and more, experts beyond a warp's 32, units without pairs, choices without a unit."""
    g = torch.Generator(device="cuda").manual_seed(n + units)
    ids = torch.randint(-1, units, (n, per), generator=g, device="cuda").int()
    ids[ids % 3 == 1] = units - 1
    most, capacity = ops.expert_plan_sizes(n * per, units, tile)
    pair_row, row_pair = torch.full((n, per), 77, dtype=torch.int32, device="cuda"), torch.full((capacity,), 77, dtype=torch.int32, device="cuda")
    plan = torch.full((1 + most,), 77, dtype=torch.int32, device="cuda")
    ops.expert_plan(ids, units, tile, pair_row, row_pair, plan)
    flat, rows = ids.flatten().cpu(), pair_row.flatten().cpu()
    counts = torch.bincount(flat[flat >= 0], minlength=units)
    tiles = (counts + tile - 1) // tile
    assert int(plan[0]) == int(tiles.sum())
    assert torch.equal(plan[1:1 + int(tiles.sum())].cpu().long(), torch.repeat_interleave(torch.arange(units), tiles))
    assert bool((rows[flat < 0] == -1).all())
    has = flat >= 0
    assert len(set(rows[has].tolist())) == int(has.sum())
    assert torch.equal(plan[1:].cpu()[(rows[has] // tile).long()], flat[has])
    back = torch.full((capacity,), -1, dtype=torch.int32)
    back[rows[has].long()] = torch.arange(n * per, dtype=torch.int32)[has]
    assert torch.equal(row_pair.cpu(), back)


@pytest.mark.parametrize("H,D,G,V", [(3, 5, 3, 8), (2, 33, 2, 36), (32, 64, 32, 67), (1, 64, 1, 67), (5, 100, 5, 103), (2, 129, 2, 132), (1, 256, 1, 259),
                                     (4, 16, 2, 64), (4, 128, 2, 128), (1, 128, 1, 132), (2, 256, 1, 64), (8, 192, 4, 36), (64, 64, 32, 64), (24, 128, 12, 128), (24, 256, 12, 128)])
def test_scans_have_the_bits_of_single_tokens(ops, H, D, G, V):
    """Batches of tokens, a batch's remainder and tokens one by one: the same bits, for every number of row groups and blocks of all sizes, the state
    straight into the lanes and through shared memory, rows of the delta rule in pieces of 16 bytes and of 4, heads that share queries and keys."""
    g = torch.Generator(device="cuda").manual_seed(D)
    R = lambda *s: torch.randn(*s, generator=g, device="cuda")                                     # noqa: E731
    lengths = [37, 16, 1, 30]
    n = sum(lengths)
    rkv, dlog, w0, u = R(n, 3 * H * D).bfloat16(), R(n, H * D), R(H * D) - 2, R(H * D)
    qkv = R(n, 2 * G * D + H * V) * D ** -0.5
    ba, a_log, dt = R(n, 2 * H), R(H) * 0.5, R(H) - 1

    def run(portions):
        s1, s2 = torch.zeros(4, H * D * D, device="cuda"), torch.zeros(4, H * D * V, device="cuda")
        o1, o2 = torch.empty(n, H * D, device="cuda"), torch.empty(n, H * V, device="cuda")
        fed = [0] * 4
        starts = [sum(lengths[:b]) for b in range(4)]
        for p in portions:
            live = [b for b in range(4) if fed[b] < lengths[b]]
            if not live:
                break
            take = [min(p, lengths[b] - fed[b]) for b in live]
            rows = torch.cat([torch.arange(starts[b] + fed[b], starts[b] + fed[b] + m) for b, m in zip(live, take)]).cuda()
            a, c = torch.empty(len(rows), H * D, device="cuda"), torch.empty(len(rows), H * V, device="cuda")
            ops.decay_scan(a, rkv[rows].contiguous(), 0, H * D, 2 * H * D, dlog[rows].contiguous(), w0, u, s1, _step(take, live), H, D)
            ops.delta_scan(c, qkv[rows].contiguous(), ba[rows].contiguous(), a_log, dt, s2, _step(take, live), H, G, D, V)
            o1[rows], o2[rows] = a, c
            for b, m in zip(live, take):
                fed[b] += m
        return o1, o2, s1, s2

    whole = run([100])
    for portions in ([17] * 4, [1] * 40):
        for got, want in zip(run(portions), whole):
            assert torch.equal(got, want)


@pytest.mark.parametrize("out,k", [(248, 72), (256, 8), (264, 136), (520, 264), (1024, 2056), (2048, 128)])
def test_grouped_products_on_pairs_of_sms(ops, out, k):
    """Token tiles of 128 rows of one matrix each: from 256 weight rows on two SMs share a tile. Matrices without a tile and with several, fewer
    tiles in use than there is room for, weight rows that are no whole tiles (the next matrix's lie behind them), k that ends inside a stage."""
    from tileinfer_b200.kernels import fast
    g = torch.Generator(device="cuda").manual_seed(out + k)
    matrices, used, room = 5, [4, 0, 0, 2, 2, 2, 3], 12
    x = torch.randn(room * 128, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(matrices, out, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    y = torch.full((room * 128, out), 7.0, dtype=torch.bfloat16, device="cuda")
    plan = torch.tensor([len(used)] + used + [99] * (room - len(used)), dtype=torch.int32, device="cuda")
    assert fast.grouped_linear(y, x, w, plan, 128)
    fast.check_status()
    for t, m in enumerate(used):
        rows = x[t * 128:(t + 1) * 128].double()
        want, mass = rows @ w[m].double().t(), rows.abs() @ w[m].double().abs().t()
        # 32-bit sums of k products in any order, then one rounding to bfloat16.
        assert bool(((y[t * 128:(t + 1) * 128].double() - want).abs() <= k / 2 * 2.0 ** -24 * mass + want.abs() * 2.0 ** -8 + 1e-7).all()), t
    assert bool((y[len(used) * 128:] == 7.0).all())


@pytest.mark.parametrize("D,nq,nkv,B", [(128, 8, 8, 50), (128, 40, 4, 100), (256, 16, 8, 45), (128, 6, 6, 90)])
def test_decode_attention_of_many_unsplit_sequences(D, nq, nkv, B):
    """A block per sequence and KV head, more of them than places: lengths on both sides of a page's end and of a warp's keys, a window, kept
    first positions, a sink; against 64-bit arithmetic."""
    from tileinfer_b200.kernels import fast
    from tileinfer_b200.kernels.library import lib
    g = torch.Generator(device="cuda").manual_seed(D + B)
    R = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()                          # noqa: E731
    lengths = [(1, 31, 32, 33, 63, 64, 65, 96, 97, 128, 129, 200)[i % 12] for i in range(B)]
    pages = 4
    k, v, q = R(B * pages, nkv, 64, D), R(B * pages, nkv, 64, D), R(B, nq, D)
    table = torch.randperm(B * pages, generator=g, device="cuda").int().view(B, pages).contiguous()
    slots, kv = torch.arange(B, device="cuda").int(), torch.tensor(lengths, device="cuda").int()
    sink = torch.randn(nq, generator=g, device="cuda")
    for window, keep, with_sink in ((0, 0, False), (40, 0, True), (70, 5, False)):
        out = torch.empty(B, nq * D, dtype=torch.bfloat16, device="cuda")
        rc = lib().ti_attention_decode_kept(out.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), table.data_ptr(), pages, slots.data_ptr(), kv.data_ptr(), None, None, None,
                                            None, D ** -0.5, B, nq, nkv, D, 64, 1, window, sink.data_ptr() if with_sink else None, 0, None, 0, 0.0, None, keep, fast._stream())
        assert rc == 0
        for b, n in enumerate(lengths):
            keys, values = (c[table[b].long()].permute(1, 0, 2, 3).reshape(nkv, -1, D)[:, :n].double().repeat_interleave(nq // nkv, 0) for c in (k, v))
            s = torch.einsum("hd,hnd->hn", q[b].double(), keys) * D ** -0.5
            at = torch.arange(n, device="cuda")
            if window:
                s = s.masked_fill(~((at >= n - window) | (at < keep)), -float("inf"))
            if with_sink:
                s = torch.cat([s, sink.double()[:, None]], 1)
            p = torch.softmax(s, -1)[:, :n]
            want = torch.einsum("hn,hnd->hd", p, values)
            # P is rounded to bfloat16, the result once more; scores and sums are 32-bit.
            bound = 2.0 ** -8 * (torch.einsum("hn,hnd->hd", p, values.abs()) + want.abs()) + 1e-5
            assert bool(((out[b].view(nq, D).double() - want).abs() <= bound).all()), (b, n, window)
