"""Row kernels that keep a row's quads in registers, at the sizes where a thread's share changes, against 64-bit arithmetic."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _rms(v, w, eps):
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps) * w.to(F64)


@pytest.mark.parametrize("size", [4, 60, 2044, 2048, 2052, 4096, 4100])
@pytest.mark.parametrize("form", ["rows", "partials", "gather"])
@pytest.mark.parametrize("centred", [False, True])
def test_branch_norm(size, form, centred):
    """One quad a thread, two, and the kernel of longer rows; a step of few rows and one of more than fill the device, whose kernel reads
    its weights and the stream late: the same bits."""
    from tileinfer_b200.kernels import fast, ops
    g = torch.Generator(device="cuda").manual_seed(size)
    n = 2 * fast.sm_count() + 5
    w, w_out, bias = ((torch.randn(size, generator=g, device="cuda") * 0.1 + c).bfloat16() for c in (1.0, 1.0, 0.0))
    x0 = torch.randn(n, size, generator=g, device="cuda")
    index = torch.randint(0, n + 2, (n, 3), generator=g, device="cuda").int()
    delta = {"rows": lambda: torch.randn(n, size, generator=g, device="cuda").bfloat16(), "partials": lambda: torch.randn(3, n, size, generator=g, device="cuda"),
             "gather": lambda: torch.randn(n + 2, size, generator=g, device="cuda").bfloat16()}[form]()
    d = {"rows": lambda: delta.to(F64), "partials": lambda: delta.to(F64).sum(0), "gather": lambda: delta.to(F64)[index.long()].sum(1)}[form]()

    def run(rows):
        x, h = x0[:rows].clone(), torch.empty(rows, size, dtype=torch.bfloat16, device="cuda")
        part = delta[:rows] if form == "rows" else delta[:, :rows].contiguous() if form == "partials" else delta
        ops.branch_norm_add32(x, part, w, 1e-6, 0.5, offset=ops.NORM_CENTRED if centred else 0, h=h, out_norm=(w_out, 1e-6, ops.NORM_CENTRED if centred else 0),
                              gather=index[:rows].contiguous() if form == "gather" else None, bias=bias)
        return x, h
    x, h = run(n)
    norm = (lambda v, g_: _rms(v - v.mean(-1, keepdim=True), g_, 1e-6)) if centred else (lambda v, g_: _rms(v, g_, 1e-6))
    new = x0.to(F64) + 0.5 * norm(d + bias.to(F64), w)
    want = norm(new, w_out)
    # Chains of a few 32-bit operations on numbers of size 6; a norm over 4 centred numbers may have a small root. The row is rounded to
    # bfloat16 once.
    assert float((x.to(F64) - new).abs().max()) <= (4e-6 if size > 4 else 4e-5)
    assert bool(((h.to(F64) - want).abs() <= want.abs() * 2.0 ** -8 + (1e-5 if size > 4 else 1e-3)).all())
    few = run(5)
    assert torch.equal(few[0], x[:5]) and torch.equal(few[1], h[:5])


# 24 + 40: one quad a thread; 336, 512 quads: two; 513, and ranks that are no whole quads: the general kernel.
@pytest.mark.parametrize("q_rank,kv_rank,rot,spare", [(24, 40, 0, 0), (24, 40, 8, 4), (768, 512, 64, 0), (0, 512, 64, 8), (1536, 512, 0, 0), (1532, 448, 68, 0),
                                                      (1536, 452, 64, 0), (1022, 130, 0, 0), (4, 4, 4, 4)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("form", ["rows", "partials"])
@pytest.mark.parametrize("interleaved", [False, True])
def test_latent_inputs(q_rank, kv_rank, rot, spare, dtype, form, interleaved):
    """A row's quads in registers and the general kernel (also the same numbers in rows off 4 elements), latents and the rotated key part."""
    from tileinfer_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(q_rank + kv_rank + rot)
    n, size, pool_row = 5, q_rank + kv_rank + rot, kv_rank + rot + spare
    rows = torch.randn(n, size, generator=g, device="cuda").to(dtype) if form == "rows" else torch.randn(3, n, size, generator=g, device="cuda")
    raw = rows.to(F64) if form == "rows" else rows.to(F64).sum(0)
    mass = raw.abs() if form == "rows" else rows.to(F64).abs().sum(0)
    wq, wkv = (torch.randn(r, generator=g, device="cuda").to(dtype) if r else None for r in (q_rank, kv_rank))
    slots = torch.tensor([6, 0, 3, 8, 1], dtype=torch.int32, device="cuda")
    positions = torch.tensor([2, 0, 7, 1, 5], dtype=torch.int32, device="cuda")
    angles = torch.rand(8, max(rot // 2, 1), generator=g, device="cuda") * 6
    table = torch.stack([angles.cos(), angles.sin()], -1).contiguous()
    rotation = SimpleNamespace(rotary_dim=rot, cos_sin=table, interleaved=interleaved) if rot else None
    off = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0

    def check(given):
        cq = torch.full((n, q_rank), 7.0, dtype=dtype, device="cuda") if q_rank else None
        pool = torch.full((9, pool_row), 7.0, dtype=dtype, device="cuda")
        ops.latent_inputs(given, cq, pool, wq, wkv, 1e-6, slots, q_rank, kv_rank, rotation=rotation, positions=positions if rot else None, pool_row=pool_row)
        parts = [(pool[slots.long(), :kv_rank], slice(q_rank, q_rank + kv_rank), wkv)]
        if q_rank:
            parts.append((cq, slice(0, q_rank), wq))
        for got, where, w in parts:
            want = _rms(raw[:, where], w, 1e-6)
            # An element's own sum of three terms off by two roundings of its terms; the root and the product by a few of the result.
            bound = want.abs() * (off + 16 * 2.0 ** -24) + mass[:, where] / raw[:, where].pow(2).mean(-1, keepdim=True).sqrt() * w.to(F64).abs() * 2.0 ** -22
            assert bool(((got.to(F64) - want).abs() <= bound).all())
        if rot:
            key, m, cs = raw[:, q_rank + kv_rank:], mass[:, q_rank + kv_rank:], table[positions.long()].to(F64)
            first, second = (slice(0, rot, 2), slice(1, rot, 2)) if interleaved else (slice(0, rot // 2), slice(rot // 2, rot))
            want, bound = torch.empty_like(key), torch.empty_like(key)
            want[:, first] = key[:, first] * cs[..., 0] - key[:, second] * cs[..., 1]
            want[:, second] = key[:, second] * cs[..., 0] + key[:, first] * cs[..., 1]
            bound[:, first] = bound[:, second] = (m[:, first] + m[:, second]) * 2.0 ** -22
            got = pool[slots.long(), kv_rank:kv_rank + rot].to(F64)
            assert bool(((got - want).abs() <= bound + want.abs() * off).all())
        assert bool((pool[slots.long(), kv_rank + rot:] == 0).all())
        assert bool((pool[[2, 4, 5, 7]] == 7.0).all())

    check(rows)
    if form == "rows":                                   # rows a whole number of elements apart, but not of quads
        wide = torch.zeros(n, size + 3, dtype=dtype, device="cuda")
        wide[:, :size] = rows
        check(wide[:, :size])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,D,taps,norm", [(16, 4, 128, 4, True), (32, 8, 64, 0, True), (6, 2, 36, 3, False), (5, 1, 256, 2, True)])
def test_convolved_attention_inputs_shared_out(nq, nkv, D, taps, norm, dtype):
    """A token's heads by one block, by a few in quads and by many channel by channel: the same bits, and those of 64-bit arithmetic within the
    roundings."""
    from tileinfer_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(nq * D)
    n, page, C = 260, 16, (nq + 2 * nkv) * D
    rows = torch.randn(n, C, generator=g, device="cuda").to(dtype)
    bias = torch.randn(C, generator=g, device="cuda").to(dtype)
    conv = torch.randn(C, taps, generator=g, device="cuda").to(dtype) if taps else None
    state = torch.randn(n, taps - 1, C, generator=g, device="cuda").to(dtype).float() if taps else None
    wq, wk = ((torch.randn(D, generator=g, device="cuda") * 0.1 + 1).to(dtype) for _ in range(2)) if norm else (None, None)

    def run(count):
        q = torch.empty(count, nq, D, dtype=dtype, device="cuda")
        k, v = (torch.empty(-(-count // page), nkv, page, D, dtype=dtype, device="cuda") for _ in range(2))
        index = torch.arange(count + 1, device="cuda").int()
        step = SimpleNamespace(positions=torch.full((count,), 9, dtype=torch.int32, device="cuda"), cu_seqlens=index, seq_slots=index[:count],
                               kv_lens=torch.full((count,), 10, dtype=torch.int32, device="cuda"), n_seqs=count)
        ops.conv_attention_inputs(rows[:count], bias, conv, taps, state, wq, wk, 1e-6, None, q, k, v, step, index[:count].contiguous(), nq, nkv, D, D, D, page,
                                  head_norm=norm)
        keys, values = (c.permute(0, 2, 1, 3).reshape(-1, nkv, D)[:count] for c in (k, v))
        return torch.cat([q, keys, values], 1)

    whole = run(n)
    for count in (1, 8, 33, 70, 150):
        assert torch.equal(run(count), whole[:count]), count
    low = dtype == torch.bfloat16
    own = (rows.to(F64) + bias.to(F64)).to(dtype).to(F64)
    if taps:
        own = ((state.to(F64) * conv.to(F64).T[:taps - 1]).sum(1) + own * conv.to(F64).T[taps - 1]).to(dtype).to(F64)
    want = own.view(n, nq + 2 * nkv, D)
    if norm:
        want = torch.cat([_rms(want[:, :nq], wq, 1e-6), _rms(want[:, nq:nq + nkv], wk, 1e-6), want[:, nq + nkv:]], 1)
    # bfloat16: a rounding before the last one may fall the other way, two units in the last place together; 32-bit: a few roundings of terms
    # of up to 64.
    assert bool(((whole.to(F64) - want).abs() <= (2.0 ** -6 if low else 2.0 ** -17) * want.abs().clamp(min=1.0)).all())
