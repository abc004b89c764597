"""What a call shares between host threads is done also where the system starts none."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("threads,helpers", [("all", "3"), ("none", "0")])
def test_all_work_is_done(tmp_path, threads, helpers):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "host_threads")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", os.path.join(HERE, "host_threads.cpp"), "-o", exe], check=True)
    res = subprocess.run([exe, threads], capture_output=True, text=True, timeout=60)
    assert (res.returncode, res.stdout) == (0, helpers)
