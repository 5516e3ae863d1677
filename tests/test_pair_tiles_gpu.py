"""The product on pairs of SMs in token tiles of every width that it takes, with a ragged last tile, against 64-bit arithmetic."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (tokens, out): widths of 128 (257 and 384 tokens), 160, 192, 224 and 256, by what fills 74 pairs best; 4,097 tokens: full tiles and one row more.
@pytest.mark.parametrize("n,out", [(257, 4096), (272, 6144), (300, 6160), (384, 6144), (411, 9216), (512, 6144), (700, 4096), (1000, 4096), (1283, 4096),
                                   (1283, 6144), (1500, 264), (2049, 2048), (4097, 512)])
@pytest.mark.parametrize("k", [200, 1024])
def test_product_in_tiles_of_every_width(n, out, k):
    from tileinfer_b200.kernels import fast, lib
    from tileinfer_b200.kernels.library import check, current_stream
    g = torch.Generator(device="cuda").manual_seed(n + out)
    x = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    w = torch.randn(out, k, generator=g, device="cuda").bfloat16()
    want, mass = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    bound = k * 2.0 ** -24 * mass                       # 32-bit sums of k products in any order
    for splits, epilogue in ((1, 0), (2, 3)):           # rounded rows; two slices of k as 32-bit partial sums
        dtype = torch.bfloat16 if splits == 1 else torch.float32
        y = torch.full((splits * n + 1, out), 7.0, dtype=dtype, device="cuda")
        check(lib().ti_gemm_tcgen05(y.data_ptr(), out, x.data_ptr(), k, w.data_ptr(), n, out, k, splits, epilogue, 0.0, 0.0, 0.0, 0.0,
                                    fast.status_word().data_ptr(), current_stream()), "gemm_tcgen05")
        fast.check_status()
        got = y[:splits * n].double().view(splits, n, out).sum(0)
        assert bool(((got - want).abs() <= bound + (want.abs() * 2.0 ** -8 if splits == 1 else 0.0)).all())
        assert bool((y[splits * n] == 7.0).all())


@pytest.mark.parametrize("n,out,k", [(769, 1536, 6144), (800, 2048, 8192), (982, 2048, 8192), (1283, 4096, 21504)])
def test_sums_of_a_cut_product_are_not_rounded(n, out, k):
    """A product that a 32-bit stream's update adds up (``allow_partials``) and that is cut over k leaves 32-bit sums, also above 768 tokens:
    a rounding to bfloat16 would be a hundred times the bound."""
    from types import SimpleNamespace
    from tileinfer_b200.kernels import fast, ops
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(n, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(out, k, generator=g, device="cuda") * k ** -0.5).bfloat16()
    rt = SimpleNamespace(buffer=lambda name, shape, dtype: torch.empty(shape, dtype=dtype, device="cuda"))
    lin = SimpleNamespace(weight=w, out_features=out, in_features=k, rt=rt, partials_name="linear.partials")
    y = fast.linear(lin, x, torch.empty(n, out, dtype=torch.bfloat16, device="cuda"), ops.EPI_NONE, (0.0, 0.0, 0.0, 0.0), allow_partials=True)
    fast.check_status()
    assert y.dtype == torch.float32 and tuple(y.shape[1:]) == (n, out) and y.shape[0] > 1
    want, mass = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # 32-bit sums of k products: off by a share of the terms' magnitudes, and far less than a bfloat16 rounding (2^-9 of the result) together.
    assert bool(((y.double().sum(0) - want).abs() <= k * 2.0 ** -24 * mass).all())
    assert float((y.double().sum(0) - want).norm() / want.norm()) <= 2.0 ** -16
