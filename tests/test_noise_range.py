"""The stress kernel's reads of the caller's noise arrays, on the CPU: its per-point
function compiled for the host over noise fields without ghosts, under the address
sanitizer."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_edge_noise_is_read_inside_its_fields(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "noise_range_check")
    cmd = [cxx, "-std=c++17", "-O1", "-g", "-fsanitize=address", "-I", os.path.join(ROOT, "tests", "cpp", "host_cuda"),
           "-I", os.path.join(ROOT, "fhdex_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "noise_range_check.cpp"),
           "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
