"""Buckets that are handed to the GPU together, on the host: tests/cpp/joined_buckets.cc, the engine's own sources over a stand-in for the
CUDA runtime and the kernels, under ThreadSanitizer."""
import os
import shutil
import subprocess

import pytest

from test_cpu_sanitizers import CSRC, ROOT, SOURCES, _nccl_include


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    gxx = shutil.which("g++")
    cuda_inc = "/usr/local/cuda/include"
    if gxx is None or not os.path.exists(os.path.join(cuda_inc, "cuda_runtime_api.h")):
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("joined") / "joined_buckets")
    cpp = os.path.join(ROOT, "tests", "cpp")
    # of what both define, the program's own stand-ins come before those that abort (stubs.cc)
    cmd = [gxx, "-std=c++17", "-O1", "-g", "-fsanitize=thread", "-fno-omit-frame-pointer", "-I", CSRC, "-I", cuda_inc, "-I", _nccl_include(),
           os.path.join(cpp, "joined_buckets.cc"), os.path.join(cpp, "stubs.cc")] + [os.path.join(CSRC, s) for s in SOURCES] + [
               "-o", exe, "-Wl,--allow-multiple-definition", "-L/usr/local/cuda/lib64", "-lcudart", "-lpthread"]
    build = subprocess.run(cmd, capture_output=True, text=True)
    if build.returncode != 0 and "sanitize" in build.stderr and "cannot find" in build.stderr:
        pytest.skip("sanitizer runtime not installed")
    assert build.returncode == 0, build.stderr[-2000:]
    return exe


def _run(program, case):
    env = dict(os.environ, LD_LIBRARY_PATH="/usr/local/cuda/lib64:" + os.environ.get("LD_LIBRARY_PATH", ""), LOG_LEVEL="OFF")
    run = subprocess.run([program, case], capture_output=True, text=True, env=env, timeout=60)
    out = run.stdout + run.stderr
    assert run.returncode == 0 and "0 failures" in out and "ThreadSanitizer" not in out, out[-3000:]


def test_buckets_that_share_memory_are_executed_one_after_the_other(program):
    _run(program, "overlap")


def test_joined_buckets_are_locked_in_one_order(program):
    _run(program, "locks")


def test_staged_buckets_share_one_block_however_they_meet(program):
    _run(program, "staging")


def test_a_bucket_that_cannot_be_prepared_fails_alone(program):
    _run(program, "failing")


def test_the_watchdog_names_all_buckets_of_a_launch(program):
    _run(program, "watchdog")


def test_a_launch_has_sixteen_buckets_at_most_and_none_twice(program):
    _run(program, "most")
