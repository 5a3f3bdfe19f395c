"""The tilings of the U-Net's convolutions (csrc/conv_plan.h), checked on
the CPU: a host-only harness (tests/native/conv_plan.cu) asks for the tiling
of every convolution of the network over the widths a network may have."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "multiscale-and-multiphysics-integrated-simulator-for-tsunami_b200" / "csrc"


def test_every_convolution_has_a_tiling(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "conv_plan"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{CSRC}", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "conv_plan.cu")], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert " 0 failures" in r.stdout, r.stdout
