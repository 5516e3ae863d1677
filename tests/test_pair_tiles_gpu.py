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
