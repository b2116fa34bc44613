"""The host layer's buffer pool against a fake CUDA runtime (tests/cpp/test_block_pool.cpp): a buffer that a stream still works on goes to no other stream."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_buffer_in_use_by_one_stream_goes_to_no_other():
    from vesper_b200.build import _nvcc
    exe = os.path.join(ROOT, "tests", "cpp", "_build", "test_block_pool")
    os.makedirs(os.path.dirname(exe), exist_ok=True)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-I", os.path.join(ROOT, "vesper_b200", "host", "include"), "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_nvcc()))), "include"),
                           os.path.join(ROOT, "tests", "cpp", "test_block_pool.cpp"), os.path.join(ROOT, "vesper_b200", "host", "src", "tensor.cpp"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout + r.stderr
