"""A wait inside a kernel that ran out is an error of the next call that waits for the device, not a silently wrong result."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _expire(cuda):
    """A peer's words that nothing writes: the kernel gives up after about a millisecond and sets the device status word."""
    import torch
    from vesper_b200 import capi
    bufs = [torch.zeros(capi.exchange_buffer_bytes(2, 16, 128), dtype=torch.uint8, device=cuda) for _ in range(2)]
    partial = torch.zeros(16, 130, device=cuda)
    capi.exchange_combine(partial, [b.data_ptr() for b in bufs], 0, torch.empty(16, 128, dtype=torch.bfloat16, device=cuda), timeout_cycles=2_000_000)
    torch.cuda.synchronize()


def test_forward_and_generation_report_it_once(cuda):
    from vesper_b200 import capi, model
    m = model.TransformerLM(64, 256, 1, 2, 1, 512, 32)
    rng = np.random.default_rng(0)
    for name, shape in model.param_shapes(64, 256, 1, 2, 1, 512).items():
        m.set_param(name, 0.02 * rng.standard_normal(shape))
    ids = rng.integers(0, 64, size=(2, 8)).astype(np.int32)
    m.init_cache(2)
    want = m.forward_with_cache(ids, 0)
    _expire(cuda)
    with pytest.raises(RuntimeError, match="gave up waiting"):
        m.forward_with_cache(ids, 0)
    assert np.array_equal(m.forward_with_cache(ids, 0), want)
    tokens, _ = m.generate_greedy(ids, 6)
    _expire(cuda)
    with pytest.raises(RuntimeError, match="gave up waiting"):
        m.generate_greedy(ids, 6)
    assert np.array_equal(m.generate_greedy(ids, 6)[0], tokens)
    capi.check_kernel_status(0)


def test_an_expired_wait_replaces_a_note_about_an_id(cuda):
    """An id outside the vocabulary leaves a note and a result; it must not keep an expired wait out of the status word."""
    import torch
    from vesper_b200 import capi
    capi.embedding(torch.tensor([9], dtype=torch.int32, device=cuda), torch.zeros(4, 128, dtype=torch.bfloat16, device=cuda), torch.empty(1, 128, device=cuda))
    _expire(cuda)
    with pytest.raises(capi.Vb200Error, match="bounded in-kernel wait"):
        capi.check_kernel_status(0)
    capi.check_kernel_status(0)


def test_the_word_in_host_memory(cuda, lib):
    """Set by the kernels themselves, seen without a copy and cleared by a check; the same on a first use while a graph is captured (a process of its own)."""
    import ctypes as C
    import subprocess
    import sys
    import torch
    from vesper_b200 import capi
    word = C.POINTER(C.c_int32)()
    capi.check(lib.vb200_kernel_status_on_host(0, C.byref(word)))
    assert word[0] == 0
    _expire(cuda)
    assert word[0] >> 24 == 3 and lib.vb200_kernel_status_of(word[0]) == -7
    with pytest.raises(capi.Vb200Error):
        capi.check_kernel_status(0)
    assert word[0] == 0
    r = subprocess.run([sys.executable, "-c", CAPTURED], capture_output=True, text=True, timeout=300, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and r.stdout.strip() == "-8 0", r.stdout + r.stderr


# the library's first launch is a captured one: ids outside the vocabulary, replayed
CAPTURED = """
import torch
from vesper_b200 import capi
lib = capi.load()
ids, table, out = torch.tensor([9], dtype=torch.int32, device="cuda"), torch.ones(4, 128, dtype=torch.bfloat16, device="cuda"), torch.ones(1, 128, device="cuda")
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    capi.embedding(ids, table, out)
graph.replay()
torch.cuda.synchronize()
assert (out == 0).all()
print(lib.vb200_check_kernel_status(0, None), lib.vb200_check_kernel_status(0, None))
"""
