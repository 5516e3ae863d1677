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
