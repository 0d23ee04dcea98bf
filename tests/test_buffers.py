"""Replacing the renderer's path buffers (sprout_b200/csrc/buffers.hpp): what a failed allocation
leaves behind, driven by a C++ check program with an allocator that fails at each call in turn."""

import pathlib
import shutil
import subprocess

import pytest

HERE = pathlib.Path(__file__).resolve().parent
CSRC = HERE.parent / "sprout_b200" / "csrc"


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_failed_allocations_leave_no_buffer_behind(tmp_path):
    exe = tmp_path / "buffers_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", str(CSRC), str(HERE / "buffers_check.cpp"), "-o", str(exe)],
                   check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout + res.stderr
    assert res.stdout.count("ok ") == 4, res.stdout
