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
