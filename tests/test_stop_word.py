"""The stop word of the CTA form: however late its copy arrives, it never lands in memory that has gone back to the pool
(host code, checked against a stand-in for the CUDA runtime)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "optimized-gpu-accelerator_b200", "csrc")


def test_copies_end_before_the_word_does(tmp_path):
    exe = tmp_path / "stop_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-I", os.path.join(HERE, "fake_cuda"), "-I", CSRC,
                    os.path.join(HERE, "stop_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
