"""x += rms_norm(y) * w at the widths where the kernel's registers end: rows that fit the narrow form, the wide form, and rows gathered twice.

Against 64 bits: a sum of `dim` squares in fp32 and a handful of roundings, relative error below 1e-5; the copy is one bf16 rounding of the result."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [8, 1024, 2040, 2048, 2056, 8192, 8200])
@pytest.mark.parametrize("M", [1, 3, 300])
def test_norm_add(cuda, M, dim):
    import torch
    from vesper_b200 import hybrid_capi
    g = torch.Generator(device=cuda).manual_seed(dim + M)
    x, y = (torch.randn(M, dim, generator=g, device=cuda) for _ in range(2))
    w, scale = (torch.rand(dim, generator=g, device=cuda) for _ in range(2))
    rows = torch.randn(2 * M, dim, generator=g, device=cuda).bfloat16()
    gather = torch.randint(0, 2 * M, (M, 2), generator=g, device=cuda, dtype=torch.int32)
    for with_rows in (False, True):
        v = y.double() + (rows[gather.long()].double().sum(1) if with_rows else 0.0)
        want = x.double() + v * torch.rsqrt(v.square().mean(1, keepdim=True) + 1e-6) * w.double()
        got = x.clone()
        copy = hybrid_capi.norm_add(got, y, w, 1e-6, rows=rows if with_rows else None, gather=gather if with_rows else None, scale=scale, copy=True)
        assert ((got.double() - want).abs() <= 1e-5 * (1.0 + want.abs())).all()
        assert torch.equal(copy, (got * scale).bfloat16())
