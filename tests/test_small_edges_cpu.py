"""The setup kernel's small-triangle path (fr_exact.cuh) compiled for the host, against
the general barycentric form on every pixel of random clamped boxes."""

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_small_edge_functions_match_the_general_form(tmp_path):
    exe = str(tmp_path / "test_small_edges")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    f"-I{ROOT}/forkerrenderer_gb300/csrc", f"{ROOT}/tests/cpp/test_small_edges.cpp",
                    "-o", exe], check=True)
    for seed in ("1", "2"):
        r = subprocess.run([exe, "60000", seed], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        assert "mismatches 0" in r.stdout
