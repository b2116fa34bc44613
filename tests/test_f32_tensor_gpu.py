"""fp32 attention on the tensor cores (head_dim 64 and 128, more than 64 keys), at the edges of its 128 x 64 tiles.

Bound: fp64 PyTorch, relative 2-norm.  An operand's three bf16 terms hold it exactly, six of the nine products of terms miss 2^-26 of a product, and
an addition in fp32 loses at most 2^-23 of the partial sum where it truncates and 2^-24 where it rounds.  A score is D / 16 such additions, an
output N / 64 sums of four more, the backward two of these in a chain: 5 * 2^-23 = 6e-7 is above the sum of their root mean squares at the
sizes here (and below what the CUDA cores' longer chains give at the largest)."""
import ctypes as C
import math

import pytest

pytestmark = pytest.mark.gpu
BOUND = 6e-7


def _reference(q, k, v, g, start, causal):
    import torch
    scale, group = q.shape[-1] ** -0.5, q.shape[1] // k.shape[1]
    q, k, v = q.double(), k.double().repeat_interleave(group, 1), v.double().repeat_interleave(group, 1)
    s = q @ k.transpose(2, 3) * scale
    if causal:
        s = s.masked_fill(torch.arange(k.shape[2], device=q.device)[None] > start + torch.arange(q.shape[2], device=q.device)[:, None], -math.inf)
    p = torch.softmax(s, -1)
    o = p @ v
    if g is None:
        return o, torch.logsumexp(s, -1)
    ds = p * (g.double() @ v.transpose(2, 3) - (g.double() * o).sum(-1, keepdim=True)) * scale
    return o, torch.logsumexp(s, -1), ds @ k, ds.transpose(2, 3) @ q, p.transpose(2, 3) @ g.double()


def _off(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("N,causal", [(65, True), (65, False), (127, True), (128, True), (129, False), (192, True), (193, True), (320, False), (1025, True)])
def test_edges_of_the_tiles(cuda, D, N, causal):
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(N * D)
    q, k, v, do = (torch.randn(2, 2, N, D, generator=g, device=cuda) for _ in range(4))
    o, lse = torch.empty_like(q), torch.empty(2, 2, N, device=cuda)
    capi.prefill(q, k, v, o, lse, scale=D ** -0.5, causal=causal)
    got = (o, lse) + tuple(capi.attention_bwd(do, q, k, v, o, lse, scale=D ** -0.5, causal=causal))
    for x, want in zip(got, _reference(q, k, v, do, 0, causal)):
        assert _off(x, want) <= BOUND


def _rows(kind, g, D, cuda):
    """q, k, v, dO whose sums differ from those of standard normal rows, which the factors in the kernel are fitted to."""
    import torch
    r = [torch.randn(2, 4, 320, D, generator=g, device=cuda) for _ in range(4)]
    if kind == "offset":
        return [x + 1 for x in r]
    if kind == "positive":
        return [x.abs() for x in r]
    if kind == "whole":                              # sums that lose nothing, scores to 40 and more
        return [x.mul(f).round() for x, f in zip(r, (2, 2, 4, 4))]
    if kind == "large":                              # scores to 100
        return [x * f for x, f in zip(r, (4, 4, 1, 1))]
    half = [x[..., :D // 2] for x in r[:2]]          # scores of two sums that cancel to a hundredth
    return [torch.cat([half[0] * 30, half[0] * 30 + 0.1 * r[0][..., D // 2:]], -1), torch.cat([half[1], -half[1]], -1), *r[2:]]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kind", ["offset", "positive", "whole", "large", "cancelling"])
def test_rows_of_other_distributions(cuda, D, kind):
    """No further from 64 bits than the CUDA cores (which a call without the whole workspace takes): at most a quarter more, what two runs of such
    rows differ by, and one rounding of a score, the factor that is given back where nothing was lost."""
    import torch
    from vesper_b200 import capi
    q, k, v, do = _rows(kind, torch.Generator(device=cuda).manual_seed(D), D, cuda)
    want = _reference(q, k, v, do, 0, True)
    off = []
    for whole in (True, False):
        o, lse = torch.empty_like(q), torch.empty(2, 4, 320, device=cuda)
        a = capi.prefill_args(q, k, v, o, lse, scale=D ** -0.5, causal=True)
        ws = torch.empty(capi.load().vb200_prefill_workspace_bytes(C.byref(a)), dtype=torch.uint8, device=cuda)
        if whole:
            a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
        capi.check(capi.load().vb200_prefill_fwd(C.byref(a)))
        got = (o, lse) + tuple(_backward(do, q, k, v, o, lse, whole))
        off.append([_off(x, w) for x, w in zip(got, want)])
    for tensor, cuda_cores in zip(*off):
        assert tensor <= 1.25 * cuda_cores + 2 ** -23


def _backward(do, q, k, v, o, lse, whole):
    """vb200_attention_bwd with its whole workspace, or with a float per row."""
    import torch
    from vesper_b200 import capi
    B, H, N, D = q.shape
    a = capi.AttnBwdArgs()
    a.struct_size, a.device, a.stream, a.dtype = C.sizeof(capi.AttnBwdArgs), 0, capi._stream_ptr(None), capi.dtype_code(q)
    a.B, a.H, a.N, a.D, a.causal, a.scale = B, H, N, D, 1, D ** -0.5
    out = [torch.empty_like(q) for _ in range(3)]
    need = capi.load().vb200_attention_bwd_workspace_bytes(C.byref(a)) if whole else 4 * B * H * N
    ws = torch.empty(need, dtype=torch.uint8, device=q.device)
    for name, t in zip(("d_out", "q", "k", "v", "out", "lse", "dq", "dk", "dv", "workspace"), (do, q, k, v, o, lse, *out, ws)):
        setattr(a, name, t.data_ptr())
    a.workspace_bytes = need
    capi.check(capi.load().vb200_attention_bwd(C.byref(a)))
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T,start,rotate", [(1, 64, False), (5, 200, True), (129, 62, False), (130, 0, True)])
def test_portions_of_a_prompt(cuda, D, T, start, rotate):
    """Groups of query heads, rows of a [B, T, H, D] tensor, keys behind cached ones, rotated queries: against the CUDA cores, which a call without
    the whole workspace takes."""
    import torch
    from vesper_b200 import capi
    L = capi.load()
    g = torch.Generator(device=cuda).manual_seed(T * D + start)
    q, k, v = (torch.randn(2, T, h, D, generator=g, device=cuda).transpose(1, 2) for h in (6, 2, 2))
    cache = [torch.randn(2, 2, start + T + 3, D, generator=g, device=cuda) for _ in range(2)]
    out = []
    for whole in (True, False):
        kc, vc = (c.clone() for c in cache)
        o, lse = torch.empty(2, T, 6, D, device=cuda).transpose(1, 2), torch.empty(2, 6, T, device=cuda)
        a = capi.prefill_args(q, k, v, o, lse, scale=D ** -0.5, causal=True, start_pos=start, theta=1e4 if rotate else None, k_cache=kc, v_cache=vc)
        need = L.vb200_prefill_workspace_bytes(C.byref(a))
        assert need > 2 * 2 * (start + T) * D * 12
        ws = torch.empty(need if whole else need - 256, dtype=torch.uint8, device=cuda)
        a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
        capi.check(L.vb200_prefill_fwd(C.byref(a)))
        torch.cuda.synchronize()
        capi.check_kernel_status(0)
        out.append((o, lse, kc, vc))
    for x, y in zip(*out):
        assert _off(x, y.double()) <= 2 * BOUND


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_masked_columns_of_huge_scores(cuda, D, causal):
    """Scores of both signs around 1e10, where a float's neighbours are 1024 apart: masked columns and those past the end weigh nothing.

    A row's weights are 1 for its largest score and 0 for the others, unless its two largest lie within the error of a score
    (D / 16 + 8 additions of 2^-23 of the largest sum of magnitudes); such rows, about one in 10^5, are left out."""
    import torch
    from vesper_b200 import capi
    N = 201
    g = torch.Generator(device=cuda).manual_seed(D)
    q, k, v = (torch.randn(1, 4, N, D, generator=g, device=cuda) * f for f in (3e5, 3e5, 1))
    o, lse = torch.empty_like(q), torch.empty(1, 4, N, device=cuda)
    capi.prefill(q, k, v, o, lse, scale=D ** -0.5, causal=causal)
    want, want_lse = _reference(q, k, v, None, 0, causal)
    s = q.double() @ k.double().transpose(2, 3) * D ** -0.5
    if causal:
        s = s.masked_fill(torch.ones(N, N, dtype=torch.bool, device=cuda).triu(1), -math.inf)
    two = s.topk(2, -1).values
    error = (D / 16 + 8) * 2 ** -23 * (q.double().abs() @ k.double().abs().transpose(2, 3)).amax(-1) * D ** -0.5
    sure = two[..., 0] - two[..., 1] > 2 * error + 100
    assert sure.float().mean() > 0.99
    assert _off(o[sure], want[sure]) <= BOUND and ((lse.double() - want_lse).abs() <= error)[sure].all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("value", [math.nan, math.inf, 3.4e38, 1e-33])
def test_values_that_three_terms_do_not_hold(cuda, D, value):
    """Four columns of one row of V outside the range: what does not depend on them is as before, and the others hold what fp32 gives."""
    import torch
    from vesper_b200 import capi
    N, at = 200, 130
    g = torch.Generator(device=cuda).manual_seed(D)
    q, k, v = (torch.randn(1, 2, N, D, generator=g, device=cuda) for _ in range(3))
    want, want_lse = _reference(q, k, v, None, 0, True)
    v[:, :, at, :4] = value
    o, lse = torch.empty_like(q), torch.empty(1, 2, N, device=cuda)
    capi.prefill(q, k, v, o, lse, scale=D ** -0.5, causal=True)
    assert _off(o[:, :, :at], want[:, :, :at]) <= BOUND and _off(o[..., 4:], want[..., 4:]) <= BOUND and _off(lse, want_lse) <= BOUND
    seen = o[:, :, at:, :4]
    if value == 3.4e38:
        p = torch.softmax((q.double() @ k.double().transpose(2, 3) * D ** -0.5).masked_fill(torch.ones(N, N, dtype=torch.bool, device=cuda).triu(1), -math.inf), -1)
        assert _off(seen, (p[:, :, at:] @ v.double())[..., :4]) <= BOUND
    elif value == 1e-33:
        v[:, :, at, :4] = 0                          # (the row adds less than a rounding)
        assert _off(seen, _reference(q, k, v, None, 0, True)[0][:, :, at:, :4]) <= BOUND
    else:
        assert (seen.isnan() if math.isnan(value) else seen.isinf()).all()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("tiny", ["q", "k", "v", "do"])
def test_one_tiny_column_beside_normal_ones(cuda, D, tiny):
    """Column 5 of one operand at 1e-37, whose second and third bf16 terms are subnormal: that column of the results it makes
    (V: O, dO: dV, K: dQ, Q: dK) keeps what fp32 gives there, 1e-5 as for the gradient below, and the other columns are as before."""
    import torch
    from vesper_b200 import capi
    N = 200
    g = torch.Generator(device=cuda).manual_seed(D)
    t = {n: torch.randn(1, 2, N, D, generator=g, device=cuda) for n in ("q", "k", "v", "do")}
    t[tiny][..., 5] *= 1e-37
    o, lse = torch.empty_like(t["q"]), torch.empty(1, 2, N, device=cuda)
    capi.prefill(t["q"], t["k"], t["v"], o, lse, scale=D ** -0.5, causal=True)
    got = dict(zip(("o", "dq", "dk", "dv"), (o, *capi.attention_bwd(t["do"], t["q"], t["k"], t["v"], o, lse, scale=D ** -0.5, causal=True))))
    want = _reference(t["q"], t["k"], t["v"], t["do"], 0, True)
    want = dict(zip(("o", "dq", "dk", "dv"), (want[0], *want[2:])))
    made = {"v": "o", "do": "dv", "k": "dq", "q": "dk"}[tiny]
    assert _off(got[made][..., 5], want[made][..., 5]) <= 1e-5
    for n in got:
        assert _off(got[n], want[n]) <= 2 * BOUND


@pytest.mark.parametrize("D", [64, 128])
def test_a_gradient_far_below_the_range(cuda, D):
    """dO of 1e-33: its second and third terms would be subnormal; 1e-5 as fp32 rounds numbers of 1e-36."""
    import torch
    from vesper_b200 import capi
    N = 200
    g = torch.Generator(device=cuda).manual_seed(D)
    q, k, v, do = (torch.randn(1, 2, N, D, generator=g, device=cuda) for _ in range(4))
    do = do * 1e-33
    o, lse, *want = _reference(q, k, v, do, 0, True)
    for x, y in zip(capi.attention_bwd(do, q, k, v, o.float(), lse.float(), scale=D ** -0.5, causal=True), want):
        assert _off(x, y) <= 1e-5


@pytest.mark.parametrize("backward", [False, True])
def test_more_heads_than_the_workspace_holds_at_a_time(cuda, backward):
    import torch
    from vesper_b200 import capi
    L = capi.load()
    H, N, D = (5500 if backward else 11000), 66, 64
    g = torch.Generator(device=cuda).manual_seed(1)
    q, k, v, do = (torch.randn(1, H, N, D, generator=g, device=cuda) for _ in range(4))
    o, lse = torch.empty_like(q), torch.empty(1, H, N, device=cuda)
    ws = capi.prefill(q, k, v, o, lse, scale=D ** -0.5)
    assert ws.numel() <= (1 << 30) + (1 << 20)
    some = [0, 1, H // 2, H - 1]
    got = [x[:, some] for x in ((o, lse) + (tuple(capi.attention_bwd(do, q, k, v, o, lse, scale=D ** -0.5)) if backward else ()))]
    for x, want in zip(got, _reference(q[:, some], k[:, some], v[:, some], do[:, some], 0, True)):
        assert _off(x, want) <= BOUND
