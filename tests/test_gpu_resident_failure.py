"""The resident form's interval is reported as failed whenever a block has recorded a timeout, also one that block 0's
own barriers do not see (a block that gives up at the last of them has already been counted)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.join(HERE, "..")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = tmp_path_factory.mktemp("resident") / "resident_check"
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--fmad=false",
                    "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "optimized-gpu-accelerator_b200", "csrc"),
                    os.path.join(HERE, "resident_check.cu"), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("blocks", [1, 2])
@pytest.mark.parametrize("error", [0, 1])
def test_outcome(check, blocks, error):
    out = subprocess.run([check, str(blocks), str(error)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
    assert out.stdout.split() == ["failed", str(error)]
