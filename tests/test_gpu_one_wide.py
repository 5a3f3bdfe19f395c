"""Preconditioner blocks one column wide with neighbours on both sides, and
blocks of more than 576 columns, whose A P is formed before the sweep: the
sizes where the sweeps' ring, its halo slots or the form itself change.

FP64 steps equal the oracle's bit for bit (tolerance 0).  The mixed solver
keeps the bounds of its comparison with the FP64 solver: max |dp| <= 1e-8
max |p|, max |du| <= 1e-9 m/s, max |dF| <= 1e-8, NF equal.
"""
import numpy as np
import pytest

from test_gpu_parity import run_pair
from test_gpu_slices import flume

pytestmark = pytest.mark.gpu

#           nx  ny  nz  ti  tj
SHAPES = [(30, 4, 9, 12, 1),     # 12 columns
          (210, 4, 9, 100, 1),   # 100, ragged last tile
          (210, 4, 9, 200, 1),   # 200: halo values in the readers' banks
          (310, 3, 8, 300, 1),   # 300: packed halo values
          (640, 3, 6, 630, 1),   # 630: no fused sweep
          (6, 70, 9, 1, 30),     # one wide along x
          (5, 130, 8, 1, 120),
          (7, 9, 12, 1, 1),      # both
          (140, 11, 9, 128, 5)]  # 640 columns, not one wide


@pytest.mark.parametrize("nx,ny,nz,ti,tj", SHAPES)
def test_fp64_bitwise(gpu_lib, pkg, orc, nx, ny, nz, ti, tj):
    run_pair(pkg, orc, pkg.cases.random_tank(nx + tj, nx=nx, ny=ny, nz=nz), 2, precond_ti=ti, precond_tj=tj)


@pytest.mark.parametrize("nx,ny,nz,ti,tj", SHAPES)
def test_mixed(gpu_lib, pkg, nx, ny, nz, ti, tj):
    c = flume(pkg, max(nx, 20), ny, nz + 12)
    t0, t1 = (pkg.Tank(c, solver=s, precond_ti=ti, precond_tj=tj, cgepsr=1e-12) for s in (0, 1))
    for t in (t0, t1):
        t.init_state(True)
        for _ in range(3):
            t.step(c.dt)
    s0, s1 = t0.get_state(), t1.get_state()
    assert t1.stats()["fallbacks"] == 0
    assert np.abs(s1["pp"] - s0["pp"]).max() <= 1e-8 * np.abs(s0["pp"]).max()
    assert max(np.abs(s1[n] - s0[n]).max() for n in ("uu", "vv", "ww")) <= 1e-9
    assert np.abs(s1["ff"] - s0["ff"]).max() <= 1e-8
    assert np.array_equal(s1["nf"], s0["nf"])
