"""The SSAO kernels' test intervals (fr_ssao.cuh, ssao_ends) compiled for the host."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ssao_intervals_hold_the_exact_values(tmp_path):
    exe = str(tmp_path / "test_ssao_ends")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    f"-I{ROOT}/forkerrenderer_gb300/csrc", f"{ROOT}/tests/cpp/test_ssao_ends.cpp",
                    "-o", exe], check=True)
    for seed in ("1", "2"):
        r = subprocess.run([exe, "60000", seed], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        assert "outside 0;" in r.stdout
