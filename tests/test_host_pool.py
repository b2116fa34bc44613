"""The host layer against a fake CUDA runtime (tests/cpp/fake_cuda.h): which buffers its pool hands to which stream and what it keeps, what it makes of a
status word that a kernel has set and of a full device."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("program,more", [("test_block_pool", []), ("test_pool_bounds", []), ("test_expired_wait", []), ("test_full_device", ["attention.cpp"])])
def test_against_a_fake_runtime(program, more):
    from vesper_b200.build import _nvcc
    exe = os.path.join(ROOT, "tests", "cpp", "_build", program)
    os.makedirs(os.path.dirname(exe), exist_ok=True)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", os.path.join(ROOT, "vesper_b200", "host", "include"), "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include"),
                           os.path.join(ROOT, "tests", "cpp", program + ".cpp")] + [os.path.join(ROOT, "vesper_b200", "host", "src", f) for f in ["tensor.cpp"] + more] + ["-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout + r.stderr
