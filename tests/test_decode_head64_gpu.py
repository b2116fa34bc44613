"""Decode with head_dim 64 on the tensor cores against the general kernel (the same call on cache rows with a stride takes that one).

Compared are the fp32 partial records.  Weights and queries enter the products as hi + lo halves: bf16 keeps 16 significand bits of
each, 2^-17 relative per factor; exponentials are accurate to 2^-22.  2^-14 of the largest output leaves a factor of four."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("lens,layout", [([0, 1, 62, 63], "bhsd"), ([64, 65, 127, 500], "bhsd"), ([15, 16, 17, 2100], "wide"), ([300], "single"), ([4095, 700], "bhsd")])
def test_matches_the_general_kernel(cuda, dtype, group, lens, layout):
    import torch
    from vesper_b200 import capi
    dt, D, Hkv, B = getattr(torch, dtype), 64, 3, len(lens)
    g = torch.Generator(device=cuda).manual_seed(group + sum(lens))
    cap = max(lens) + 5
    r = lambda *s: torch.randn(*s, generator=g, device=cuda).to(dt)
    q, kn, vn = r(B, Hkv * group, 1, D), r(B, Hkv, 1, D), r(B, Hkv, 1, D)
    k, v = r(B, Hkv, cap, D), r(B, Hkv, cap, D)
    for c in (k, v):
        for b, n in enumerate(lens):
            c[b, :, n + 1:] = float("nan")                      # rows that nothing may read into a result
    seq = torch.tensor(lens, dtype=torch.int32, device=cuda)

    def run(kc, vc):
        part = torch.empty(B, Hkv * group, D + 2, device=cuda)
        capi.decode(q, None, kc, vc, scale=D ** -0.5, k_new=kn, v_new=vn, theta=10000.0, seq_lens=seq, max_len=max(lens) + 1, partial_out=part)
        return part

    def strided(c):
        big = torch.zeros(B, Hkv, cap, 2 * D, dtype=dt, device=cuda)
        big[..., :D] = c
        return big[..., :D]
    kg, vg = strided(k), strided(v)
    want = run(kg, vg)
    if layout == "wide":                                        # heads of a larger cache, sequences far apart
        def view(c):
            big = torch.zeros(B, 2 * Hkv, cap + 3, D, dtype=dt, device=cuda)
            big[:, ::2, :cap] = c
            return big[:, ::2, :cap]
        k, v = view(k), view(v)
    elif layout == "single":                                    # one sequence: its stride may be anything
        k, v = k[0].expand(1, Hkv, cap, D), v[0].expand(1, Hkv, cap, D)
    got = run(k, v)
    capi.check_kernel_status(0)
    scale = want[..., :D].abs().max()
    assert (got[..., :D] - want[..., :D]).abs().max() <= 2 ** -14 * scale
    lse = lambda x: x[..., D] + x[..., D + 1].log()
    assert (lse(got) - lse(want)).abs().max() <= 2e-5 * max(1.0, lse(want).abs().max())
    for a, b in ((k, kg), (v, vg)):                             # the appended rows
        for i, n in enumerate(lens):
            assert torch.equal(a[i, :, n], b[i, :, n])


def test_repeated_cache_heads_stay_on_the_general_kernel(cuda):
    """A cache whose heads share one row block (stride 0) cannot be described by a tensor map."""
    import torch
    from vesper_b200 import capi
    D, cap = 64, 200
    g = torch.Generator(device=cuda).manual_seed(1)
    q = torch.randn(2, 8, 1, D, generator=g, device=cuda).bfloat16()
    k, v = (torch.randn(2, 1, cap, D, generator=g, device=cuda).bfloat16() for _ in range(2))

    def run(kc, vc):
        part = torch.empty(2, 8, D + 2, device=cuda)
        capi.decode(q, None, kc, vc, scale=D ** -0.5, uniform_len=150, max_len=150, append_enabled=False, partial_out=part)
        return part
    got, want = run(k.expand(2, 2, cap, D), v.expand(2, 2, cap, D)), run(k.repeat(1, 2, 1, 1), v.repeat(1, 2, 1, 1))
    assert (got[..., :D] - want[..., :D]).abs().max() <= 2 ** -14 * want[..., :D].abs().max()
