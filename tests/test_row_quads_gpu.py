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
