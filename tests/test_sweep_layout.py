"""The tile-overlapped layout of the solver's arrays and the shared-memory
slots of the sweeps (csrc/kernels.h, csrc/sweep_cp.cuh), checked on the CPU:
a host-only harness (tests/native/sweep_layout.cu) enumerates the entries of
every cell, coefficient and halo value for a set of grids and tile shapes."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "multiscale-and-multiphysics-integrated-simulator-for-tsunami_b200" / "csrc"


def test_every_cell_and_halo_value_has_its_own_entry(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "sweep_layout"
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{CSRC}", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "sweep_layout.cu")], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert " 0 failures" in r.stdout, r.stdout
