"""The common eigenbasis of dense couplings to twice the FP64 precision (host code)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_refined_basis(tmp_path):
    exe = str(tmp_path / "eigenbasis_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(HERE, "..", "libheom_gb300", "csrc"),
                    os.path.join(HERE, "eigenbasis_check.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, timeout=60).stdout.strip() == "OK"
