"""Products of more than 64 rows on pairs of CTAs (tiles of 256 rows x 256 or 128 columns) and on single CTAs: rows and columns at the edges of the
tiles, K tails, one and several rounds, the three kernels that the dispatch chooses from.

Against 64 bits.  fp32 accumulation of K <= 1024 products of order 1/sqrt(K): rounding of order sqrt(K) 2^-24, far below 1e-4;
16-bit outputs carry one bf16 rounding (2^-9 relative) on top."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(8, 72), (112, 1024), (304, 456), (1000, 520), (11264, 64)])
@pytest.mark.parametrize("M", [65, 128, 129, 256, 257, 300, 513, 1000, 2305])
def test_pairs(cuda, M, N, K):
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    x = torch.randn(M, K + 8, generator=g, device=cuda).bfloat16()[:, :K]
    w = (torch.randn(N, K, generator=g, device=cuda) / K ** 0.5).bfloat16()
    want = x.double() @ w.double().T
    h = torch.randn(M, N, generator=g, device=cuda)
    gain, copy, sum64 = torch.rand(N, generator=g, device=cuda), torch.empty(M, N, dtype=torch.bfloat16, device=cuda), h.double() + want
    capi.linear_ex(x, w, h, epilogue=capi.EPI_ADD_F32, scaled_copy=copy, copy_scale=gain)
    assert (h.double() - sum64).abs().max().item() < 1e-4
    assert torch.equal(copy, (h * gain).bfloat16())
    scale = torch.rand(M, generator=g, device=cuda)
    y = torch.empty(M, N, device=cuda)
    capi.linear_ex(x, w, y, epilogue=capi.EPI_F32, row_scale=scale)
    assert (y.double() - want * scale.double()[:, None]).abs().max().item() < 1e-4
    wide = torch.full((M, N + 8), 3.0, dtype=torch.bfloat16, device=cuda)
    capi.linear_ex(x, w, wide[:, :N], epilogue=capi.EPI_BF16)
    assert ((wide[:, :N].double() - want).abs() - want.abs() / 256).max().item() < 1e-4
    assert bool((wide[:, N:] == 3.0).all())
    if N % 16 == 0:
        z = torch.empty(M, N // 2, dtype=torch.bfloat16, device=cuda)
        capi.linear_ex(x, w, z, epilogue=capi.EPI_SWIGLU)
        gated = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
        assert ((z.double() - gated).abs() - gated.abs() / 256).max().item() < 1e-4
    capi.check_kernel_status(0)


@pytest.mark.parametrize("K", [456, 1032])
@pytest.mark.parametrize("M,N", [(2305, 11264), (1000, 19008)])
def test_pairs_over_several_tiles(cuda, M, N, K):
    """Several tiles per pair with more blocks of 64 columns than the ring has stages, and not a multiple of them: stages and their parities carry over
    from tile to tile while the accumulators alternate."""
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g, device=cuda).bfloat16()
    w = (torch.randn(N, K, generator=g, device=cuda) / K ** 0.5).bfloat16()
    want = x.double() @ w.double().T
    h = torch.randn(M, N, generator=g, device=cuda)
    sum64 = h.double() + want
    capi.linear_ex(x, w, h, epilogue=capi.EPI_ADD_F32)
    assert (h.double() - sum64).abs().max().item() < 1e-4
    z = torch.empty(M, N // 2, dtype=torch.bfloat16, device=cuda)
    capi.linear_ex(x, w, z, epilogue=capi.EPI_SWIGLU)
    gated = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
    assert ((z.double() - gated).abs() - gated.abs() / 256).max().item() < 1e-4
    capi.check_kernel_status(0)


def test_product_longer_than_a_wait(cuda):
    """The limit of a wait inside the kernel (2e9 cycles) is for one hand-over; a product that takes longer than that as a whole is computed in full.
    2 n^3 operations at 148 x 8192 per cycle, the most that bf16 can do, take 2.1e9 cycles."""
    import torch
    from vesper_b200 import capi
    n = 108544
    if torch.cuda.mem_get_info(cuda)[0] < 80e9:
        pytest.skip("three matrices of 24 GB")
    x = torch.full((n, n), 1.0, dtype=torch.bfloat16, device=cuda)
    w = torch.full((n, n), 2.0 ** -17, dtype=torch.bfloat16, device=cuda)
    out = torch.zeros(n, n, dtype=torch.bfloat16, device=cuda)
    capi.linear_ex(x, w, out)
    capi.check_kernel_status(0)
    del x, w
    assert all(bool((part == n * 2.0 ** -17).all()) for part in out.split(8192))       # every partial sum is a multiple of 2^-17 below 1: exact
    del out
    torch.cuda.empty_cache()
