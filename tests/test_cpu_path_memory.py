"""The blocks of path state kept between calls (csrc/path_memory.h) with a fake
allocator on the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("path_memory") / "path_memory_check"
    build = ["g++", "-g", "-O1", "-std=c++17", "-pthread", "-o", str(exe), os.path.join(HERE, "native", "path_memory_check.cpp")]
    subprocess.run(build[:1] + ["-fsanitize=address"] + build[1:], check=True)
    return exe


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("what", ["exit", "in_turn", "at_once", "pressure"])
def test_kept_blocks(check, what):
    """exit: a scene released by a static object's destructor finds the blocks' records still there.
    in_turn: one block serves calls one after the other.  at_once: calls at the same time keep a block each.
    pressure: the idle blocks give way where memory is short."""
    out = subprocess.run([str(check), what], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr[:2000]
