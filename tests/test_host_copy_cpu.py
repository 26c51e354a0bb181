"""The threaded host copy of batch downloads (fr_hostcopy.h): every split of the bytes,
and allocation failures while its threads start."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_copy_is_whole_for_every_split_and_without_memory_for_threads(tmp_path):
    exe = str(tmp_path / "test_host_copy")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-I{ROOT}/forkerrenderer_gb300/csrc",
                    f"{ROOT}/tests/cpp/test_host_copy.cpp", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "differences 0" in r.stdout
