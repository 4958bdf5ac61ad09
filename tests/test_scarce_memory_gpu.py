"""Calls that use more temporaries than they need, with each of them refused in
turn (out of memory, or not in the pool under capture): a native program with
the library's objects and a memory resource that refuses."""
import glob
import importlib.util
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "opencl-sdk_gb300")


def test_refused_temporaries(tmp_path):
    spec = importlib.util.spec_from_file_location("gbc_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    build.build()
    exe = tmp_path / "scarce_memory"
    subprocess.run([build.nvcc(), "-std=c++17", "-O2", "-I" + build.CSRC, os.path.join(ROOT, "tests", "native", "scarce_memory.cpp")]
                   + sorted(glob.glob(os.path.join(build.OUT_DIR, "*.o"))) + ["-cudart", "static", "-lpthread", "-ldl", "-lrt",
                                                                            "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
