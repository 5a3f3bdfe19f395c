"""The copy depth of the MILU sweeps (sweep_cp_depth in csrc/sweep_cp.cuh),
checked on the CPU by a host-only harness (tests/native/sweep_depth.cu)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "multiscale-and-multiphysics-integrated-simulator-for-tsunami_b200" / "csrc"


def test_depth_follows_the_devices_sms(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "sweep_depth"
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{CSRC}", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "sweep_depth.cu")], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert " 0 failures" in r.stdout, r.stdout
