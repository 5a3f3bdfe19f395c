"""Vertical slices (one row of columns, one or more tiles along x), which run
the sweeps with thread copies although their tiles are one column wide, and
batches whose members' tiles are one column wide with and without
neighbours.

FP64 steps equal the oracle's bit for bit (tolerance 0).  The mixed solver
keeps the bounds of its comparison with the FP64 solver: max |dp| <= 1e-8
max |p|, max |du| <= 1e-9 m/s, max |dF| <= 1e-8, NF equal.  A batch equals its
members alone bit for bit.
"""
import numpy as np
import pytest

from test_gpu_parity import run_pair

pytestmark = pytest.mark.gpu


def flume(pkg, nx, ny, nz):
    c = pkg.cases.porous_flume(nx=nx, ny=ny, nz=nz, dx=0.05, dz=0.4 * 1.25 / nz, depth=0.4,
                               block=(0.3 * nx * 0.05, 0.5 * nx * 0.05, 0.4), sponge_width=0.3, dt=2e-3)
    pkg.cases.linear_wave_initial(c, 0.04, 1.0, 0.4)
    return c


#        nx  nz  ti (0: the whole row)
SLICES = [(400, 40, 0), (256, 30, 0), (31, 17, 0), (40, 9, 16), (65, 25, 32), (49, 21, 12), (300, 12, 260),
          (800, 12, 0)]  # the widest block


@pytest.mark.parametrize("nx,nz,ti", SLICES)
def test_slice_bitwise(gpu_lib, pkg, orc, nx, nz, ti):
    run_pair(pkg, orc, flume(pkg, nx, 1, nz), 2, precond_ti=ti, precond_tj=1 if ti else 0)


@pytest.mark.parametrize("nx,nz,ti", SLICES)
def test_slice_mixed(gpu_lib, pkg, nx, nz, ti):
    c = flume(pkg, nx, 1, nz)
    t0, t1 = (pkg.Tank(c, solver=s, precond_ti=ti, precond_tj=1 if ti else 0, cgepsr=1e-12) for s in (0, 1))
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


@pytest.mark.parametrize("rows", [(1, 1, 1), (1, 3, 2)])
def test_batch_of_slices(gpu_lib, pkg, rows):
    mk = lambda: [flume(pkg, nx, ny, nz) for nx, ny, nz in zip((64, 40, 90), rows, (30, 22, 41))]
    kw = dict(solver=1, precond_ti=16, precond_tj=1, cgepsr=1e-10)
    together, alone = ([pkg.Tank(c, **kw) for c in mk()] for _ in range(2))
    for t in together + alone:
        t.init_state(True)
    batch = pkg.Batch(together)
    for _ in range(3):
        assert batch.step() == [0] * 3
        for t in alone:
            t.step()
    batch.close()
    for a, b in zip(together, alone):
        assert a.stats()["icgitr"] == b.stats()["icgitr"]
        sa, sb = a.get_state(), b.get_state()
        for k in ("uu", "vv", "ww", "pp", "ff", "nf"):
            assert sa[k].tobytes() == sb[k].tobytes(), k
