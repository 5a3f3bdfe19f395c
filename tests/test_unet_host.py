"""The U-Net's entry points (csrc/unet.cu) when a launch or a runtime call
fails, checked on the CPU: tests/native/unet_host.cu compiles the host code
against a stand-in for the CUDA runtime and makes each call fail in turn."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "multiscale-and-multiphysics-integrated-simulator-for-tsunami_b200" / "csrc"


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if Path("/usr/local/cuda/bin/nvcc").exists() else None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path_factory.mktemp("unet_host") / "unet_host"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_100a,code=sm_100a", f"-I{CSRC}", "-Xcompiler",
                    "-pthread", "-o", str(exe), str(ROOT / "tests" / "native" / "unet_host.cu")], check=True,
                   capture_output=True)
    return exe


def run(exe, mode):
    r = subprocess.run([str(exe), mode], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert " 0 failures" in r.stdout, r.stdout


def test_failed_launches_are_reported(exe):
    run(exe, "launch")


def test_nothing_is_queued_after_a_call(exe):
    run(exe, "runtime")
