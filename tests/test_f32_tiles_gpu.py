"""The tiled fp32 attention kernels at the edges of their 64 x 64 tiles, against fp64 PyTorch.

Bound: a score and an output are sums of at most D + N fp32 products, each rounded once; with N(0, 1) operands the rounding errors
add like a random walk, sqrt(D + N) * 2^-24 of the largest partial sum, and the backward chains three such sums: 2e-5 of the
largest value is about ten times that at the sizes here."""
import math

import pytest

pytestmark = pytest.mark.gpu


def _reference(q, k, v, start, causal, d_out=None):
    import torch
    q, k, v = q.double(), k.double(), v.double()
    scale, group = q.shape[-1] ** -0.5, q.shape[1] // k.shape[1]
    k, v = k.repeat_interleave(group, 1), v.repeat_interleave(group, 1)
    s = q @ k.transpose(2, 3) * scale
    if causal:
        at = torch.arange(k.shape[2], device=q.device)
        s = s.masked_fill(at[None] > start + torch.arange(q.shape[2], device=q.device)[:, None], -math.inf)
    p = torch.softmax(s, -1)
    o = p @ v
    if d_out is None:
        return o, torch.logsumexp(s, -1)
    g = d_out.double()
    ds = p * (g @ v.transpose(2, 3) - (g * o).sum(-1, keepdim=True)) * scale
    return ds @ k, ds.transpose(2, 3) @ q, p.transpose(2, 3) @ g


def _close(got, want):
    assert (got.double() - want).abs().max() <= 2e-5 * max(1.0, want.abs().max().item())


@pytest.mark.parametrize("D", [8, 40, 64, 72, 128])
@pytest.mark.parametrize("T,start,causal", [(1, 0, True), (63, 0, True), (64, 0, False), (65, 0, True), (130, 0, True), (70, 61, True), (65, 0, False)])
def test_forward_edges(cuda, D, T, start, causal):
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(T * D + start)
    B, Hq, Hkv = 2, 4, 2
    rows = [torch.randn(B, T, h, D, generator=g, device=cuda).transpose(1, 2) for h in (Hq, Hkv, Hkv)]      # [B, T, H, D] memory
    q, k, v = rows
    o, lse = torch.empty_like(q), torch.empty(B, Hq, T, device=cuda)
    kw = {}
    if start:
        cache = [torch.randn(B, Hkv, start + T + 3, D, generator=g, device=cuda) for _ in range(2)]
        kw = dict(k_cache=cache[0], v_cache=cache[1], start_pos=start)
    capi.prefill(q, k, v, o, lse, scale=D ** -0.5, causal=causal, **kw)
    if start:
        k, v = (torch.cat([c[:, :, :start], x], 2) for c, x in zip(cache, (k, v)))
    want_o, want_lse = _reference(q, k, v, start, causal)
    _close(o, want_o)
    _close(lse, want_lse)


@pytest.mark.parametrize("D", [8, 40, 64, 72, 128])
@pytest.mark.parametrize("N,causal", [(1, True), (63, True), (64, False), (65, True), (191, False), (200, True)])
def test_backward_edges(cuda, D, N, causal):
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(N * D)
    q, k, v, do = (torch.randn(2, 3, N, D, generator=g, device=cuda) for _ in range(4))
    want_o, want_lse = _reference(q, k, v, 0, causal)
    got = capi.attention_bwd(do, q, k, v, want_o.float(), want_lse.float(), scale=D ** -0.5, causal=causal)
    for x, want in zip(got, _reference(q, k, v, 0, causal, do)):
        _close(x, want)


@pytest.mark.parametrize("D,shift", [(33, 0), (64, 1)])
def test_backward_without_16_byte_rows(cuda, D, shift):
    """Rows or base pointers that are not multiples of 16 bytes take the general kernels."""
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(D)
    n = 2 * 70 * D
    q, k, v, do = (torch.randn(n + shift, generator=g, device=cuda)[shift:].view(1, 2, 70, D) for _ in range(4))
    o, lse = _reference(q, k, v, 0, True)
    got = capi.attention_bwd(do, q, k, v, o.float(), lse.float(), scale=D ** -0.5, causal=True)
    for x, want in zip(got, _reference(q, k, v, 0, True, do)):
        _close(x, want)


@pytest.mark.parametrize("D", [40, 64, 128])
@pytest.mark.parametrize("at", [0, 70, 100])
@pytest.mark.parametrize("which", ["d_out", "q", "k", "v"])
def test_backward_infinite_rows_stay_where_they_are_seen(cuda, D, at, which):
    """Causal, 130 positions: an infinite row of one operand reaches only the gradients that depend on it; a masked position adds nothing, not 0 * inf."""
    import torch
    from vesper_b200 import capi
    N = 130
    g = torch.Generator(device=cuda).manual_seed(D + at)
    t = dict(zip(("q", "k", "v", "d_out"), (torch.randn(1, 2, N, D, generator=g, device=cuda) for _ in range(4))))
    o, lse = _reference(t["q"], t["k"], t["v"], 0, True)
    want = _reference(t["q"], t["k"], t["v"], 0, True, t["d_out"])
    t[which][:, :, at, ::2] = math.inf
    if which in ("q", "k", "v"):                     # what a forward pass gives: rows that see the position are not finite
        first, last = at, at + 1 if which == "q" else N
        o[:, :, first:last], lse[:, :, first:last] = math.nan, math.nan
    got = capi.attention_bwd(t["d_out"], t["q"], t["k"], t["v"], o.float(), lse.float(), scale=D ** -0.5, causal=True)
    row = which in ("d_out", "q")                    # a row of queries: its own dq, and dk and dv of the keys up to it
    clean = [[i for i in range(N) if (i != at if row else i < at)]] + [[j for j in range(N) if j > at] if row else []] * 2
    for x, y, keep in zip(got, want, clean):
        _close(x[:, :, keep], y[:, :, keep]) if keep else None


@pytest.mark.parametrize("D", [8, 32, 36, 64, 128])
@pytest.mark.parametrize("heads", [1, 160, 400])
@pytest.mark.parametrize("N", [16, 17, 32, 33, 65, 96, 97])
def test_backward_on_either_side_of_the_dispatch(cuda, D, heads, N):
    """Short sequences of few and of many heads: the general kernels or the tiled ones."""
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(N * D + heads)
    q, k, v, do = (torch.randn(1, heads, N, D, generator=g, device=cuda) for _ in range(4))
    o, lse = _reference(q, k, v, 0, True)
    got = capi.attention_bwd(do, q, k, v, o.float(), lse.float(), scale=D ** -0.5, causal=True)
    for x, want in zip(got, _reference(q, k, v, 0, True, do)):
        _close(x, want)


@pytest.mark.parametrize("D", [40, 64, 128])
@pytest.mark.parametrize("heads,T", [(150, 128), (150, 129), (40, 700), (150, 200)])
def test_forward_on_either_side_of_the_dispatch(cuda, D, heads, T):
    """Grids and lengths on both sides of the rule for four or eight query rows per thread."""
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(T * D + heads)
    q, k, v = (torch.randn(1, heads, T, D, generator=g, device=cuda) for _ in range(3))
    o, lse = torch.empty_like(q), torch.empty(1, heads, T, device=cuda)
    capi.prefill(q, k, v, o, lse, scale=D ** -0.5)
    want_o, want_lse = _reference(q, k, v, 0, True)
    _close(o, want_o)
    _close(lse, want_lse)
