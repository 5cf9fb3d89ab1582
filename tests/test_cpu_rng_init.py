"""The generator initialisation's jump tables reach every pixel of every image a
camera may ask for (run on the host from the header that the kernel uses)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_jump_tables_reach_every_pixel(tmp_path):
    exe = tmp_path / "xorwow_init_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", str(exe), os.path.join(HERE, "native", "xorwow_init_check.cpp")],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout
