"""Decode with head_dim 64 on contiguous cache rows: fp32 throughout, against 64 bits and against the general kernel (the same call on cache
rows with a stride takes that one).

Compared are the fp32 partial records.  A score is a sum of 64 products whose partial sums stay below 16 in log2 units here: sqrt(64) roundings of
2^-25 * 16 move a weight by 64 * 2^-21 * ln 2 / 8 = 2.6e-6, the exponential by 2^-22; both are averaged over the keys of a row.  3e-6 of the largest output.
(16 significand bits in a query or a weight give 4e-6 to 1.2e-5.)"""
import math

import pytest

pytestmark = pytest.mark.gpu

D, BOUND = 64, 3e-6


def _rotate(x, pos, theta):
    """Rotation of adjacent pairs by the fp32 angle pos * freq."""
    import torch
    from vesper_b200 import capi
    if theta is None:
        return x.double()
    freq = torch.tensor(list(capi.inv_freq(theta, D))[: D // 2], dtype=torch.float32, device=x.device)
    angle = (torch.tensor(float(pos), device=x.device) * freq).double()
    a, b = x.double()[..., 0::2], x.double()[..., 1::2]
    return torch.stack((a * angle.cos() - b * angle.sin(), a * angle.sin() + b * angle.cos()), -1).flatten(-2)


def _exact(q, k, v, kn, vn, lens, scale, theta):
    import torch
    group, rows, lses = q.shape[1] // k.shape[1], [], []
    for b, n in enumerate(lens):
        keys = torch.cat((k[b, :, :n].double(), _rotate(kn[b], n, theta)), 1).repeat_interleave(group, 0)
        values = torch.cat((v[b, :, :n], vn[b]), 1).double().repeat_interleave(group, 0)
        s = (_rotate(q[b], n, theta) * keys).sum(-1) * scale
        rows.append(torch.where(s[..., None] == -math.inf, 0.0, torch.softmax(s, -1)[..., None] * values).sum(1))
        lses.append(torch.logsumexp(s, -1))
    return torch.stack(rows), torch.stack(lses)


def _partial(q, k, v, kn, vn, lens, scale, theta, **kw):
    import torch
    from vesper_b200 import capi
    part = torch.empty(q.shape[0], q.shape[1], D + 2, device=q.device)
    seq = torch.tensor(lens, dtype=torch.int32, device=q.device)
    capi.decode(q, None, k, v, scale=scale, k_new=kn, v_new=vn, theta=theta, seq_lens=seq, max_len=max(lens) + 1, partial_out=part, **kw)
    capi.check_kernel_status(0)
    return part[..., :D], part[..., D] + part[..., D + 1].log()


def _inputs(device, dtype, lens, heads, kv_heads, seed, spread=1.0):
    import torch
    g = torch.Generator(device=device).manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device=device).to(getattr(torch, dtype))
    B, cap = len(lens), max(lens) + 5
    return [r(B, heads, 1, D) * spread, r(B, kv_heads, cap, D), r(B, kv_heads, cap, D), r(B, kv_heads, 1, D), r(B, kv_heads, 1, D)]


def _close(got, want):
    assert (got.double() - want).abs().max() <= BOUND * want.abs().max()


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("lens,layout", [([0, 1, 62, 63], "bhsd"), ([64, 65, 127, 500], "bhsd"), ([15, 16, 17, 2100], "wide"), ([300], "single"), ([4095, 700], "bhsd")])
def test_matches_the_general_kernel(cuda, dtype, group, lens, layout):
    import torch
    Hkv, B, cap = 3, len(lens), max(lens) + 5
    q, k, v, kn, vn = _inputs(cuda, dtype, lens, Hkv * group, Hkv, group + sum(lens))
    for c in (k, v):
        for b, n in enumerate(lens):
            c[b, :, n + 1:] = float("nan")                      # rows that nothing may read into a result

    def strided(c):
        big = torch.zeros(B, Hkv, cap, 2 * D, dtype=c.dtype, device=cuda)
        big[..., :D] = c
        return big[..., :D]
    kg, vg = strided(k), strided(v)
    want = _partial(q, kg, vg, kn, vn, lens, D ** -0.5, 10000.0)
    if layout == "wide":                                        # heads of a larger cache, sequences far apart
        def view(c):
            big = torch.zeros(B, 2 * Hkv, cap + 3, D, dtype=c.dtype, device=cuda)
            big[:, ::2, :cap] = c
            return big[:, ::2, :cap]
        k, v = view(k), view(v)
    elif layout == "single":                                    # one sequence: its stride may be anything
        k, v = k[0].expand(1, Hkv, cap, D), v[0].expand(1, Hkv, cap, D)
    got = _partial(q, k, v, kn, vn, lens, D ** -0.5, 10000.0)
    _close(got[0], want[0].double())
    assert (got[1] - want[1]).abs().max() <= BOUND * max(1.0, want[1].abs().max())
    for a, b in ((k, kg), (v, vg)):                             # the appended rows
        for i, n in enumerate(lens):
            assert torch.equal(a[i, :, n], b[i, :, n])


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("lens", [[0, 1, 62, 63], [300, 2100], [20000]])
def test_records_keep_32_bits(cuda, dtype, group, lens):
    """Queries wide enough that a few keys decide: the record's columns and its LSE against 64 bits."""
    x = _inputs(cuda, dtype, lens, 2 * group, 2, group + sum(lens), spread=6)
    want, lse = _exact(*x, lens, D ** -0.5, 10000.0)
    got = _partial(*x, lens, D ** -0.5, 10000.0)
    _close(got[0], want)
    assert (got[1].double() - lse).abs().max() <= BOUND * max(1.0, lse.abs().max())


@pytest.mark.parametrize("dtype", ["bfloat16", "float16"])
@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("lens,at", [([63, 200], 0), ([63, 200], 40), ([700], 650)])
def test_infinite_keys_and_values(cuda, dtype, group, lens, at):
    """A key whose score is -inf has no weight; a value column that is infinite makes that column infinite and no other."""
    import torch
    x = _inputs(cuda, dtype, lens, 2 * group, 2, group + at)
    x[0][..., 5] = x[0][..., 5].abs() + 0.5
    x[1][:, :, at, 5] = -math.inf
    want, lse = _exact(*x, lens, D ** -0.5, None)
    got = _partial(*x, lens, D ** -0.5, None)
    _close(got[0], want)
    assert (got[1].double() - lse).abs().max() <= BOUND * max(1.0, lse.abs().max())
    x[1][:, :, at, 5] = 0.25
    want, _ = _exact(*x, lens, D ** -0.5, None)
    x[2][:, :, at, 7] = math.inf
    got = _partial(*x, lens, D ** -0.5, None)[0]
    assert bool((got[..., 7] == math.inf).all())
    others = [d for d in range(D) if d != 7]
    _close(got[..., others], want[..., others])


@pytest.mark.parametrize("group", [1, 2, 4, 8])
def test_large_fp16_queries(cuda, group):
    """Queries that their rotation takes beyond the largest fp16 value."""
    lens = [1, 100, 333]
    x = _inputs(cuda, "float16", lens, 2 * group, 2, group)
    x[0].fill_(60000.0)
    for t in (x[1], x[3]):
        t.mul_(2.0 ** -15)
    want, _ = _exact(*x, lens, 1.0, 10000.0)
    _close(_partial(*x, lens, 1.0, 10000.0)[0], want)


def test_repeated_cache_heads(cuda):
    """A cache whose heads share one row block (stride 0)."""
    import torch
    from vesper_b200 import capi
    cap = 200
    g = torch.Generator(device=cuda).manual_seed(1)
    q = torch.randn(2, 8, 1, D, generator=g, device=cuda).bfloat16()
    k, v = (torch.randn(2, 1, cap, D, generator=g, device=cuda).bfloat16() for _ in range(2))

    def run(kc, vc):
        part = torch.empty(2, 8, D + 2, device=cuda)
        capi.decode(q, None, kc, vc, scale=D ** -0.5, uniform_len=150, max_len=150, append_enabled=False, partial_out=part)
        return part
    got, want = run(k.expand(2, 2, cap, D), v.expand(2, 2, cap, D)), run(k.repeat(1, 2, 1, 1), v.repeat(1, 2, 1, 1))
    assert torch.equal(got, want)
