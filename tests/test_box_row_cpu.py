"""The row of a pixel in a triangle's box (fr_exact.cuh, box_row), compiled for the host."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rows_of_every_box(tmp_path):
    exe = str(tmp_path / "test_box_row")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT}/forkerrenderer_gb300/csrc",
                    f"{ROOT}/tests/cpp/test_box_row.cpp", "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout + r.stderr
