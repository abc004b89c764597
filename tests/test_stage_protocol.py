"""The threads of a team that solves a stage agree on every branch, whatever order they run in between
two barriers (stage_protocol.cpp runs them in all of them)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def explorer(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("protocol") / "stage_protocol")
    subprocess.run([cxx, "-std=c++17", "-O1", os.path.join(HERE, "stage_protocol.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("model", ["sweeps", "items"])
def test_threads_agree_in_every_order(explorer, model):
    res = subprocess.run([explorer, model], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
