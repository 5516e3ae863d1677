"""Prompts through the recurrences in chunks of 64 tokens, side by side, against the recurrences run token by token in 64-bit."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64
LENGTHS = [130, 1, 64, 65, 127]


def _step(lengths, slots):
    cu = torch.tensor([sum(lengths[:i]) for i in range(len(lengths) + 1)], dtype=torch.int32, device="cuda")
    return SimpleNamespace(cu_seqlens=cu, seq_slots=torch.tensor(slots, dtype=torch.int32, device="cuda"), n_seqs=len(lengths))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,D,V,act", [(3, 12, 20, True), (2, 128, 128, True), (1, 132, 264, False), (5, 33, 7, True)])
def test_lightning_in_chunks(dtype, H, D, V, act):
    from tileinfer_b200.kernels import ops
    g = torch.Generator().manual_seed(D + V)
    n, slots = sum(LENGTHS), [3, 1, 5, 0, 2]
    rows = torch.randn(n, 2 * H * D + H * V + 8, generator=g).to(dtype)
    decay = torch.rand(H, generator=g) * 0.6 + 0.399
    state0 = torch.randn(6, H, D, V, generator=g)
    state, o = state0.clone().cuda(), torch.empty(n, H * V, device="cuda")
    cu = torch.tensor([0] + list(np.cumsum(LENGTHS)), dtype=torch.int32, device="cuda")
    chunks, floats = ops.memory_chunk_sizes(LENGTHS, H, D, V)
    space = (chunks, torch.full((floats,), float("nan"), device="cuda"), torch.full((chunks, H), float("nan"), device="cuda"))
    ops.lightning_scan(o, rows.cuda(), 0, H * D, 2 * H * D, state, decay.cuda(), cu, torch.tensor(slots, dtype=torch.int32, device="cuda"), 5, H, D, V,
                       act=act, chunked=space)
    x = rows.to(F64).cuda()
    f = (lambda z: (z * torch.sigmoid(z)).to(dtype).to(F64)) if act else (lambda z: z)
    q, k, v = (f(x[:, a:b]).view(n, H, -1) for a, b in ((0, H * D), (H * D, 2 * H * D), (2 * H * D, 2 * H * D + H * V)))
    want, at, a = torch.zeros(n, H, V, dtype=F64, device="cuda"), 0, decay.to(F64).cuda()[:, None, None]
    for b, m in enumerate(LENGTHS):
        S = state0[slots[b]].to(F64).cuda()
        for t in range(at, at + m):
            S = a * S + k[t][:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hdv,hd->hv", S, q[t])
        at += m
        assert float((state[slots[b]].to(F64) - S).abs().max()) <= 1e-4 * max(1.0, float(S.abs().max()))
    # The activation's rounding to bfloat16 may fall the other way where the 32-bit and the 64-bit sigmoid part.
    tol = 1e-4 if dtype == torch.float32 else 4e-3
    assert float((o.to(F64).view(n, H, V) - want).abs().max()) <= tol * max(1.0, float(want.abs().max()))
    assert torch.equal(state[4].cpu(), state0[4])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D,V", [(12, 20), (128, 128)])
def test_an_infinity_does_not_reach_the_tokens_ahead_of_it(dtype, D, V):
    """A query, key or value that is infinite or NaN, at every place of a group of four tokens: the outputs of earlier tokens of the sequence
    and of the other sequences are the bits that they are without it; its own and later ones are not finite."""
    from tileinfer_b200.kernels import ops
    H, lengths = 2, [70, 130, 66]
    g = torch.Generator().manual_seed(D)
    n = sum(lengths)
    clean = torch.randn(n, 2 * H * D + H * V, generator=g).to(dtype)
    decay = torch.tensor([0.9, 0.998], device="cuda")
    sp = _step(lengths, [0, 1, 2])
    chunks, floats = ops.memory_chunk_sizes(lengths, H, D, V)

    def run(rows):
        state, o = torch.zeros(3, H, D, V, device="cuda"), torch.empty(n, H * V, device="cuda")
        space = (chunks, torch.empty(floats, device="cuda"), torch.empty(chunks, H, device="cuda"))
        ops.lightning_scan(o, rows.cuda(), 0, H * D, 2 * H * D, state, decay, sp.cu_seqlens, sp.seq_slots, 3, H, D, V, act=False, chunked=space)
        return o
    want = run(clean)
    for t in (1, 2, 3, 4, 63, 65, 66, 67):                # places in the second sequence: first chunk, its last token, second chunk
        for column, bad in ((2 * H * D + 1, float("inf")), (2 * H * D + 1, float("nan")), (H * D + 1, float("inf")), (1, float("nan"))):
            rows = clean.clone()
            rows[lengths[0] + t, column] = bad
            got, at = run(rows), lengths[0] + t
            assert torch.equal(got[:at], want[:at]), (t, column, bad)
            assert torch.equal(got[lengths[0] + lengths[1]:], want[lengths[0] + lengths[1]:])
            assert not bool(torch.isfinite(got[at, :V]).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D,V", [(128, 128), (32, 36), (9, 7)])          # the state moved on four elements at a time, and one
def test_a_state_carried_over_many_chunks(dtype, D, V):
    """65 chunks, the last one ragged, of zero keys: the state only fades, by its decay's power. Every chunk rounds an element once, this
    way or that, so their mean is off by far less than a factor rounded to one float, the same at every chunk, would make it."""
    from tileinfer_b200.kernels import ops
    decay = torch.tensor([0.9961, 0.998, 0.9995, 0.99975, 0.9999], dtype=torch.float32)       # something is left after so many tokens
    H, tokens = len(decay), 64 * 64 + 37
    sp = _step([tokens], [0])
    chunks, floats = ops.memory_chunk_sizes([tokens], H, D, V)
    g = torch.Generator().manual_seed(D)
    state0 = torch.rand(1, H, D, V, generator=g) + 0.5
    state, o = state0.clone().cuda(), torch.empty(tokens, H * V, device="cuda")
    rows = torch.zeros(tokens, 2 * H * D + H * V, dtype=dtype, device="cuda")
    ops.lightning_scan(o, rows, 0, H * D, 2 * H * D, state, decay.cuda(), sp.cu_seqlens, sp.seq_slots, 1, H, D, V, act=True,
                       chunked=(chunks, torch.empty(floats, device="cuda"), torch.empty(chunks, H, device="cuda")))
    want = state0.to(F64) * (decay.to(F64) ** tokens)[None, :, None, None]
    off = (state.cpu().to(F64) - want) / want
    assert float(off.abs().max()) <= chunks * 2.0 ** -24 * 1.1
    # The mean over n elements of sums of 65 roundings of up to half a unit (2^-24 of the element at most): their spread is below
    # sqrt(65 / 3) 2^-24 = 2.8e-7 each; six times that over sqrt(n), and 2e-9 for the second float's own rounding. One float per factor
    # is off by 65 times up to 2^-25 of it: 1e-7 to 2.6e-6 for these decays.
    bound = 6 * 2.8e-7 / (D * V) ** 0.5 + 2e-9
    assert float(off[0].flatten(1).mean(1).abs().max()) <= bound
    powers = decay.to(F64) ** 64
    assert float(((powers.float().to(F64) - powers) / powers * 65).abs().max()) > (2 * bound if D * V > 1000 else 0)


@pytest.mark.parametrize("lengths", [[64 * 10 + 37], [130, 577]])
def test_outputs_with_slow_decays(lengths):
    """128 x 128 heads with the decays that the design has, more than eight chunks: within a few 1e-7 of 64-bit arithmetic in 32-bit."""
    from tileinfer_b200.kernels import ops
    H, D = 8, 128
    decay = torch.tensor([np.exp(-2.0 ** -k) for k in range(1, 9)], dtype=torch.float32)
    sp = _step(lengths, [1, 0][:len(lengths)])
    n = sum(lengths)
    g = torch.Generator(device="cuda").manual_seed(n)
    rows = torch.randn(n, 3 * H * D, generator=g, device="cuda")
    chunks, floats = ops.memory_chunk_sizes(lengths, H, D, D)
    state, o = torch.zeros(2, H, D, D, device="cuda"), torch.empty(n, H * D, device="cuda")
    ops.lightning_scan(o, rows, 0, H * D, 2 * H * D, state, decay.cuda(), sp.cu_seqlens, sp.seq_slots, len(lengths), H, D, D, act=False,
                       chunked=(chunks, torch.empty(floats, device="cuda"), torch.empty(chunks, H, device="cuda")))
    q, k, v = (x.to(F64).view(n, H, D) for x in rows.split(H * D, 1))
    want, at = torch.zeros(n, H, D, dtype=F64, device="cuda"), 0
    for b, m in enumerate(lengths):
        S = torch.zeros(H, D, D, dtype=F64, device="cuda")
        for t in range(at, at + m):
            S = decay.to(F64).cuda()[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
            want[t] = torch.einsum("hdv,hd->hv", S, q[t])
        at += m
        assert float((state[sp.seq_slots[b]].to(F64) - S).norm() / S.norm()) <= 2e-7
    # Sums of 128 and 64 products in groups of 16, a handful of roundings of 2^-25 on average: 8e-8 measured, the walk token by token 9e-8.
    assert float((o.to(F64).view(n, H, D) - want).norm() / want.norm()) <= 2e-7
