"""The K slices of a product of up to 64 rows, summed across a thread-block cluster: every number of slices, with row counts at the
edges of what a CTA of the cluster finishes (1, 2 or a multiple of 4 rows), slices that get no K block, and N and K tails.

Against 64 bits.  fp32 accumulation of K <= 2048 products of order 1/sqrt(K): rounding of order sqrt(K) 2^-24, far below 1e-4;
a gated output carries one bf16 rounding (2^-9 relative) on top."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [0, 1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("M", [1, 2, 5, 8, 9, 16, 17, 31, 32, 33, 63, 64])
def test_cluster_sum(cuda, M, splits):
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(100 * M + splits)
    for N, K in ((304, 456), (128, 64), (112, 2048)):
        x = torch.randn(M, K, generator=g, device=cuda).bfloat16()
        w = (torch.randn(N, K, generator=g, device=cuda) / K ** 0.5).bfloat16()
        want = x.double() @ w.double().T
        h = torch.randn(M, N, generator=g, device=cuda)
        gain, copy, sum64 = torch.rand(N, generator=g, device=cuda), torch.empty(M, N, dtype=torch.bfloat16, device=cuda), h.double() + want
        capi.linear_ex(x, w, h, epilogue=capi.EPI_ADD_F32, splits=splits, scaled_copy=copy, copy_scale=gain)
        assert (h.double() - sum64).abs().max().item() < 1e-4
        assert torch.equal(copy, (h * gain).bfloat16())
        rows = torch.randn(M, 512, generator=g, device=cuda)
        y = torch.empty(M, N, device=cuda)
        capi.linear_ex(x, w, y, epilogue=capi.EPI_F32, splits=splits, rms_rows=rows, rms_eps=1e-6)
        assert (y.double() - want * torch.rsqrt(rows.double().square().mean(1, keepdim=True) + 1e-6)).abs().max().item() < 1e-4
        z = torch.empty(M, N // 2, dtype=torch.bfloat16, device=cuda)
        capi.linear_ex(x, w, z, epilogue=capi.EPI_SWIGLU, splits=splits)
        gated = torch.nn.functional.silu(want[:, 0::2]) * want[:, 1::2]
        assert ((z.double() - gated).abs() - gated.abs() / 256).max().item() < 1e-4
    capi.check_kernel_status(0)


@pytest.mark.parametrize("N,K", [(2048, 2048), (3072, 2048), (11264, 2048), (8448, 2048), (2048, 5632), (160, 4096), (32000, 512), (8960, 2240), (304, 456)])
@pytest.mark.parametrize("M", [1, 8, 17, 40])
def test_default_slices(cuda, M, N, K):
    """The slices that the library chooses fix the order of a product's sums, and with it every bit of the result: one per SM and tile of 128
    weight rows, up to 8 (5 above 32 rows), the next larger number that divides the blocks of 64 columns where there is one."""
    import torch
    from vesper_b200 import capi
    tiles, blocks, most = -(-N // 128), -(-K // 64), 5 if M > 32 else 8
    want = max(1, min(-(-torch.cuda.get_device_properties(cuda).multi_processor_count // tiles), most, blocks))
    want = next((s for s in range(want, min(most, blocks) + 1) if blocks % s == 0), want)
    g = torch.Generator(device=cuda).manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g, device=cuda).bfloat16(), torch.randn(N, K, generator=g, device=cuda).bfloat16()
    chosen, stated = torch.empty(M, N, device=cuda), torch.empty(M, N, device=cuda)
    capi.linear_ex(x, w, chosen, epilogue=capi.EPI_F32)
    capi.linear_ex(x, w, stated, epilogue=capi.EPI_F32, splits=want)
    assert torch.equal(chosen, stated)
    capi.check_kernel_status(0)
