"""The buffers of the sums over the grid (sum_partials in csrc/kernels.h),
checked on the CPU: a host-only harness (tests/native/sum_partials.cu)
compares their size with what the kernels write, and the solver's handle
takes its buffer of five sums from it."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "multiscale-and-multiphysics-integrated-simulator-for-tsunami_b200" / "csrc"


def test_partials_fit_their_buffers(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "sum_partials"
    subprocess.run([nvcc, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{CSRC}", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "sum_partials.cu")], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert " 0 failures" in r.stdout, r.stdout


def test_the_handle_allocates_by_that_size():
    sizes = re.findall(r"AL\(h->rb5, (.*?)\);", (CSRC / "api.cu").read_text())
    assert sizes == ["5 * (size_t)sum_partials(h->q)"]
