"""The mixed solver on grids of few layers cut into many small tiles: a tile
then has fewer wavefront slabs than a block of the slab sums, so the
backward sweeps leave more partials (one per tile) than a slab sum does.

Bounds of the comparison with the FP64 solver, as for other shapes: max |dp|
<= 1e-8 max |p|, max |du| <= 1e-9 m/s, max |dF| <= 1e-8, NF equal.  A batch
equals its members alone bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

#         nz ti tj  (slabs a tile: nz + ti + tj - 2)
SHAPES = [(3, 2, 2), (5, 2, 2), (3, 3, 3), (4, 1, 1)]


def tank_case(pkg, nz, nx=96, ny=60):
    return pkg.cases.dam_break(nx=nx, ny=ny, nz=nz, column=(nx // 2, nz - 1), dt=1e-3)


@pytest.mark.parametrize("nz,ti,tj", SHAPES)
def test_mixed_solver_on_few_layers(gpu_lib, pkg, nz, ti, tj):
    c = tank_case(pkg, nz)
    over = dict(precond_ti=ti, precond_tj=tj, cgepsr=1e-12)
    t0, t1 = (pkg.Tank(c, solver=s, **over) for s in (0, 1))
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


@pytest.mark.parametrize("nz,ti,tj", SHAPES)
def test_batch_on_few_layers(gpu_lib, pkg, nz, ti, tj):
    mk = lambda: [tank_case(pkg, nz), tank_case(pkg, nz, 70, 41), tank_case(pkg, nz + 20, 40, 30)]
    kw = dict(solver=1, precond_ti=ti, precond_tj=tj, cgepsr=1e-10)
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
