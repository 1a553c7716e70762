"""Trace conditioning by several engines at once, a thread each, on traces
whose cubics take different amounts of shared memory: every call must launch,
with the samples it gives alone.  tests/condition_threads_check.cpp is
compiled against the engine library; native threads, since Python's take turns
where the calls meet."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_engines_in_threads_condition_their_own_traces(engine_lib, tmp_path):
    cxx, cuda = shutil.which("g++"), os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if cxx is None or not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    out, libdir = str(tmp_path / "condition_threads_check"), os.path.join(ROOT, "psdm_b200", "lib")
    r = subprocess.run([cxx, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I",
                        os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "condition_threads_check.cpp"),
                        "-o", out, "-L", libdir, "-lpsdm_rtm", "-L", os.path.join(cuda, "lib64"), "-lcudart",
                        "-lpthread", "-Wl,-rpath," + libdir], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    r = subprocess.run([out, "10000"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.split() == ["0", "0"], r.stdout + r.stderr
