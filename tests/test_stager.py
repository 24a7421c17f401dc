"""Staging of host arrays when memory runs out while its threads are started (tests/cpp/stager_check.cpp,
built for the host against the engine's library; no GPU): each failing allocation is reported or leaves
fewer threads, and the process goes on."""
import os
import subprocess

import pytest

from conftest import ROOT

LIBDIR = os.path.join(ROOT, "agama_b200", "_lib")
CUDA = "/usr/local/cuda"


def test_no_memory_for_a_thread(tmp_path):
    if not os.path.exists(os.path.join(LIBDIR, "libagama_b200.so")):
        pytest.skip("engine library not built")
    exe = str(tmp_path / "stager_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wno-unknown-pragmas", "-x", "c++",
                        "-I" + os.path.join(ROOT, "agama_b200", "csrc"), "-I" + os.path.join(ROOT, "include"),
                        "-I" + CUDA + "/include", os.path.join(ROOT, "tests", "cpp", "stager_check.cpp"), "-o", exe,
                        "-L" + LIBDIR, "-lagama_b200", "-L" + CUDA + "/lib64", "-lcudart", "-pthread",
                        "-Wl,-rpath," + LIBDIR], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    running = dict(map(int, line.split()) for line in out.stdout.splitlines())
    assert sorted(running) == list(range(1, 8))
    # once the first thread runs, the ones that follow are not needed
    first = min(k for k in running if running[k] == 1)
    assert all(running[k] == 1 for k in range(first, 8))
