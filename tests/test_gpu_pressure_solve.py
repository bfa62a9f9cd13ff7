"""The pressure stage (right-hand side, tridiagonal solve of every column from
both ends, inverse transforms) against the oracle at level counts around the
solve's chunks of rows and its meeting row, on grids whose columns fill the
last warp and grids whose do not.

Bar 1e-11: FP64 round-off (1.1e-16) times the condition of the lowest mode's
column, about 4 / (dz k)^2 = 4 x 66^2 at the tallest grid here, times the few
roundings of a row."""
import numpy as np
import pytest

from gpu_util import make_pair, oracle_field, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(32, 24), (36, 36), (12, 6)])
@pytest.mark.parametrize("nz", [3, 4, 5, 16, 17, 18, 34, 65])
def test_pressure_matches_oracle(built_lib, nx, ny, nz):
    p, o, g = make_pair(nx=nx, ny=ny, Nz=nz, seed=5)
    rng = np.random.default_rng(7)
    d = np.zeros_like(o.divtz)
    d[1:, :, :nx] = rng.uniform(-1, 1, d[1:, :, :nx].shape)
    w = o.w.copy()
    w[p.nz, :, :nx] = rng.uniform(-0.1, 0.1, (ny, nx))   # an intermediate velocity through the lid
    o.divtz[:], o.w[:] = d, w
    g.set("divtz", d)
    g.set("w", w)
    o.press_stag_array()
    g.press_stag_array()
    for f in ("p", "dpdx", "dpdy", "dpdz"):
        e = rel_err(p, f, g.get(f), oracle_field(o, f))
        assert e < 1e-11, (f, e)
    g.close()


def test_every_instance_of_a_batch(built_lib):
    """The mean modes' warps and the columns' come in the instances' order."""
    from lesgo_gb300.solver import LesgoBatch, LesgoGPU
    kw = dict(nx=36, ny=24, Nz=13, dt=1e-4, dyn_init=2, cs_count=2)
    b = LesgoBatch(5, **kw)
    ids = [b.add(1e-4 * (i + 1), 60 + i) for i in range(5)]
    b.step(2)
    b.sync()
    for i, iid in enumerate(ids):
        s = LesgoGPU(zo=1e-4 * (i + 1), **kw)
        s.init_ic(60 + i)
        s.step(2)
        s.sync()
        assert np.array_equal(s.get("p"), b.get(iid, "p")), i
        s.close()
    b.close()
