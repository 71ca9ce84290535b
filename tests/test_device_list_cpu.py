"""Lists in device memory whose replacement fails (tests/device_list_errors.cpp, built for the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_failed_replacement_keeps_the_list(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    exe = str(tmp_path / "list_errors")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", os.path.join(ROOT, "simuverse_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "device_list_errors.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert "ok" in r.stdout
