"""fp32 attention from several streams: temporaries that one stream's kernels still read go to no other.  The results must have the bits of calls that ran alone."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _build():
    from vesper_b200.build import LIBDIR, build_host
    build_host()
    exe = os.path.join(ROOT, "tests", "cpp", "_build", "test_streams_b200")
    os.makedirs(os.path.dirname(exe), exist_ok=True)
    src = os.path.join(ROOT, "tests", "cpp", "test_streams_b200.cpp")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", os.path.join(ROOT, "vesper_b200", "host", "include"), "-I", os.path.join(ROOT, "include"), src, "-o", exe,
                           "-L", LIBDIR, "-lvesper_b200_host", "-lvesper_b200", f"-Wl,-rpath,{LIBDIR}"])
    return exe


def test_the_program_of_two_threads_builds(lib):
    assert os.access(_build(), os.X_OK)


@pytest.mark.gpu
def test_host_operator_from_two_threads(cuda, lib):
    r = subprocess.run([_build()], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
def test_operators_on_a_side_stream_own_what_they_allocate(cuda, lib):
    """Calls queued on a side stream behind a long kernel, their workspaces let go of at once: what the current stream allocates and overwrites meanwhile
    is not memory that those calls still read or write."""
    import torch
    from vesper_b200 import capi
    g = torch.Generator(device=cuda).manual_seed(3)
    q, k, v, do = (torch.randn(1, 8, 700, 64, generator=g, device=cuda) for _ in range(4))
    o, lse = torch.empty_like(q), torch.empty(1, 8, 700, device=cuda)

    def call(stream=None):
        capi.prefill(q, k, v, o, lse, scale=0.125, stream=stream)
        return capi.attention_bwd(do, q, k, v, o, lse, scale=0.125, stream=stream)

    want = [x.clone() for x in call()] + [o.clone(), lse.clone()]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)                  # about ten milliseconds
        got = call(side)
        for nbytes in (1 << 20, 7 << 20, 14 << 20, 28 << 20, 30 << 20):
            torch.empty(nbytes, dtype=torch.uint8, device=cuda).fill_(255)
        torch.cuda.synchronize()
        assert all(torch.equal(x, y) for x, y in zip([*got, o, lse], want))
