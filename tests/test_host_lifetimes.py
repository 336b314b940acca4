"""The engine's host code on a stand-in for the CUDA runtime (tests/host_cuda):
copies queued on a stream read their host memory when the stream is waited for,
under AddressSanitizer, so memory that was freed in between is reported."""
import glob
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "host_cuda")


def build(tmp, name):
    """The test program `name` linked with the engine's objects and the fake runtime."""
    from lf_dem_gb300 import build as B
    if shutil.which("g++") is None:
        pytest.skip("no host C++ compiler")
    B.build()
    objs = sorted(glob.glob(os.path.join(B.BUILD, "*.o")))
    if len(objs) != len(B.sources()):
        B.build(force=True)
        objs = sorted(glob.glob(os.path.join(B.BUILD, "*.o")))
    cuda = os.path.dirname(os.path.dirname(B._nvcc()))
    exe = os.path.join(str(tmp), name)
    subprocess.run(["g++", "-std=c++17", "-g", "-fsanitize=address", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(cuda, "include"), os.path.join(SRC, name + ".cpp"),
                    os.path.join(SRC, "fake_cudart.cpp"), *objs, "-lpthread", "-o", exe],
                   check=True, capture_output=True, text=True)
    return exe


def run(exe, *args):
    env = dict(os.environ, ASAN_OPTIONS="detect_leaks=0:abort_on_error=0")
    return subprocess.run([exe, *args], capture_output=True, text=True, env=env, timeout=300)


@pytest.fixture(scope="module")
def lifetimes(tmp_path_factory):
    return build(tmp_path_factory.mktemp("host"), "lifetimes")


@pytest.mark.parametrize("path", ["analysis", "values", "superset"])
def test_copies_outlive_no_host_memory(lifetimes, path):
    p = run(lifetimes, path)
    assert p.returncode == 0 and p.stdout == f"done {path}\n", p.stdout + p.stderr[-3000:]


def test_failed_allocations_leave_nothing_to_launch(tmp_path):
    p = run(build(tmp_path, "failures"))
    assert p.returncode == 0 and p.stdout == "0\n", p.stdout + p.stderr[-3000:]
