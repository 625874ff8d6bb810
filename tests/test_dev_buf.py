"""Host bookkeeping of device buffers when an allocation is refused (no GPU)."""
import os
import subprocess

from conftest import ROOT


def test_refused_allocation_leaves_no_buffer(tmp_path):
    exe = tmp_path / "dev_buf_failures"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I",
                        os.path.join(ROOT, "libaccint-public_b200", "csrc"), "-I", "/usr/local/cuda/include",
                        os.path.join(ROOT, "tests", "cpp", "dev_buf_failures.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "0 failures" in r.stdout, r.stdout
