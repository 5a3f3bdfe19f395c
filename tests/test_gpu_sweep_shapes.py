"""The MILU sweeps, the vector passes over the tile-overlapped layout and the
cell and scan kernels of a step, at the sizes where their splits can go
wrong: tiles whose columns do not fill warps, one-wide last tiles, one-wide
tiles (the bulk-copy form), tiles of more than 256 and 576 columns (other
copy depths and halo layouts), fewer layers than a tile's ramp (no overlap),
planes that are no multiple of a block and depths that are no multiple of
the planes per scan.

FP64 steps equal the oracle's bit for bit (tolerance 0).  The mixed solver
keeps the bounds of its comparison with the FP64 solver: max |dp| <= 1e-8
max |p|, max |du| <= 1e-9 m/s, max |dF| <= 1e-8, NF equal, and the schedule
(sweep_occupancy) does not change a bit of it.
"""
import numpy as np
import pytest

from test_gpu_parity import assert_same, run_pair

pytestmark = pytest.mark.gpu

#        nx  ny  nz  ti  tj
SHAPES = [(37, 9, 21, 16, 8),    # T = 128, ragged in x and y
          (33, 17, 20, 16, 16),  # compiled-in shape; last tiles one wide both ways
          (40, 13, 18, 7, 5),    # T = 40: a padding column, warps not full
          (21, 9, 6, 8, 16),     # fewer layers than the ramp: tiles do not overlap
          (30, 20, 3, 16, 16),   # three layers, the fewest
          (50, 5, 11, 1, 4),     # one-wide tiles: bulk-copy form
          (19, 6, 9, 8, 1),
          (49, 25, 13, 24, 16),  # T = 384
          (70, 21, 11, 32, 20),  # T = 640
          (4, 3, 3, 4, 3)]       # one small tile


@pytest.mark.parametrize("occ", [0, 1, 2])
@pytest.mark.parametrize("nx,ny,nz,ti,tj", SHAPES)
def test_tile_shapes_bitwise(gpu_lib, pkg, orc, nx, ny, nz, ti, tj, occ):
    c = pkg.cases.random_tank(nx + ny, nx=nx, ny=ny, nz=nz, nobst=0 if nx < 8 or nz < 4 else 2,
                              nporous=0 if nx < 8 or nz < 4 else 2)
    run_pair(pkg, orc, c, 2, precond_ti=ti, precond_tj=tj, sweep_occupancy=occ)


@pytest.mark.parametrize("nx,ny,ti,tj", [(37, 9, 16, 8), (33, 17, 16, 16), (40, 13, 7, 5), (50, 5, 1, 4),
                                         (49, 25, 24, 16), (70, 21, 32, 20)])
def test_mixed_tile_shapes(gpu_lib, pkg, nx, ny, ti, tj):
    c = pkg.cases.porous_flume(nx=nx, ny=ny, nz=30, dx=0.05, dz=0.025, depth=0.4, block=(0.6, 0.9, 0.5),
                               sponge_width=0.3, dt=2e-3)
    pkg.cases.linear_wave_initial(c, 0.04, 1.0, 0.4)
    over = dict(precond_ti=ti, precond_tj=tj, cgepsr=1e-10)
    ts = [pkg.Tank(c, solver=s, sweep_occupancy=o, **over) for s, o in ((0, 0), (1, 1), (1, 2))]
    for t in ts:
        t.init_state(True)
        for _ in range(3):
            t.step(c.dt)
    s0, s1, s2 = (t.get_state() for t in ts)
    assert_same(s2, s1, "mixed, two blocks per SM")
    assert ts[1].stats()["fallbacks"] == 0
    assert np.abs(s1["pp"] - s0["pp"]).max() <= 1e-8 * np.abs(s0["pp"]).max()
    assert max(np.abs(s1[n] - s0[n]).max() for n in ("uu", "vv", "ww")) <= 1e-9
    assert np.abs(s1["ff"] - s0["ff"]).max() <= 1e-8
    assert np.array_equal(s1["nf"], s0["nf"])
