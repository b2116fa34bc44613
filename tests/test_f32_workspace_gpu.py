"""fp32 attention with less than the whole workspace: the same operators on the CUDA cores (head_dim 64 and 128 above 64 positions take them by no other way).

Bound: fp64 PyTorch, relative 2-norm; a sum of 513 fp32 FMAs in two chains of a block's 64 and one of nine blocks loses at most 74 * 2^-24 = 4.4e-6 of
its magnitudes, and a quarter of that (1.2e-6) is above the root mean square of such losses."""
import ctypes as C

import pytest

from test_f32_tensor_gpu import _off, _reference

pytestmark = pytest.mark.gpu
BOUND = 1.2e-6


def _forward(q, k, v, do, causal):
    import torch
    o, lse, *want = _reference(q, k, v, do, 0, causal)
    return o.float(), lse.float(), want


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("N,causal", [(65, True), (129, False), (200, True), (513, True)])
def test_backward_with_a_float_per_row(cuda, lib, D, N, causal):
    """B * H * N floats, what the header says is enough: no multiple of 64 here."""
    import torch
    from vesper_b200 import capi
    B, H = 1, 3
    g = torch.Generator(device=cuda).manual_seed(N + D)
    q, k, v, do = (torch.randn(B, H, N, D, generator=g, device=cuda) for _ in range(4))
    o, lse, want = _forward(q, k, v, do, causal)
    a = capi.AttnBwdArgs()
    a.struct_size, a.device, a.stream, a.dtype = C.sizeof(capi.AttnBwdArgs), 0, capi._stream_ptr(None), capi.dtype_code(q)
    a.B, a.H, a.N, a.D, a.causal, a.scale = B, H, N, D, int(causal), D ** -0.5
    got = [torch.empty_like(q) for _ in range(3)]
    rows = torch.empty(B * H * N + 64, device=cuda)
    rows[B * H * N:] = 7.0
    for name, t in zip(("d_out", "q", "k", "v", "out", "lse", "dq", "dk", "dv", "workspace"), (do, q, k, v, o, lse, *got, rows)):
        setattr(a, name, t.data_ptr())
    a.workspace_bytes = 4 * B * H * N - 1
    assert lib.vb200_attention_bwd(C.byref(a)) == -4
    a.workspace_bytes = 4 * B * H * N
    capi.check(lib.vb200_attention_bwd(C.byref(a)))
    torch.cuda.synchronize()
    assert (rows[B * H * N:] == 7.0).all()
    for x, w in zip(got, want):
        assert _off(x, w) <= BOUND


def test_a_caller_may_decline_the_terms(cuda, lib):
    """A smaller workspace that a call can do with is the one it uses: nothing is allocated in its place."""
    import torch
    from vesper_b200 import capi
    B, H, N, D = 2, 16, 1000, 128
    g = torch.Generator(device=cuda).manual_seed(1)
    q, k, v, do = (torch.randn(B, H, N, D, generator=g, device=cuda) for _ in range(4))
    o, lse = torch.empty_like(q), torch.empty(B, H, N, device=cuda)
    none, rows = torch.empty(0, dtype=torch.uint8, device=cuda), torch.empty(B * H * N, device=cuda)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    assert capi.prefill(q, k, v, o, lse, scale=D ** -0.5, workspace=none) is none
    assert lib.vb200_last_prefill_kernel() == b"prefill_f32_kernel"
    got = capi.attention_bwd(do, q, k, v, o, lse, scale=D ** -0.5, workspace=rows)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - before <= 3 * q.numel() * 4 + (8 << 20)          # (the gradients, in torch's rounded blocks)
    whole = capi.prefill(q, k, v, o.clone(), lse.clone(), scale=D ** -0.5)
    assert lib.vb200_last_prefill_kernel() == b"attention_f32_forward_kernel" and whole.numel() > 4 * q.numel()
    for x, w in zip((o, lse, *got), _reference(q, k, v, do, 0, True)):
        assert _off(x, w) <= 2 * BOUND
    # a workspace that the call cannot do with is replaced, as it always was
    kc, vc = (torch.zeros(B, H, N, D, device=cuda) for _ in range(2))
    assert capi.prefill(q, k, v, o, lse, scale=D ** -0.5, theta=1e4, k_cache=kc, v_cache=vc, workspace=none) is not none
