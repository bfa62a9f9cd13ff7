"""The passes whose transforms are held in registers, at every length they
serve in x and y and for every boundary treatment, against the oracle and
against the run-time radix passes (LESGO_RFFT=0), which serve all other
lengths.

Bars: the mixed form's 2e-4 against the oracle, and against the run-time
radix passes the 5e-5 (velocity) and 1e-3 (pressure) of two FP32 transforms
that round differently (as the tensor-core form is held to)."""
import numpy as np
import pytest

from gpu_util import make_pair, oracle_field, rel_err

pytestmark = pytest.mark.gpu

# nx/2, 3 nx/4 and ny run through every length; Nz small, odd and even
GRIDS = [
    (32, 24, 12, {}), (36, 36, 13, {}), (48, 54, 10, dict(ubc_mom=2)), (64, 64, 9, {}), (72, 32, 9, dict(lbc_mom=0)),
    (96, 48, 17, {}), (108, 72, 11, dict(lbc_mom=1, ubc_mom=1, molec=True)), (128, 128, 8, {}), (144, 96, 7, {}),
    (192, 108, 6, {}), (216, 144, 5, {}), (256, 256, 4, {}), (64, 192, 8, {}), (96, 216, 8, {}),
]
IDS = ["%dx%dx%d" % g[:3] for g in GRIDS]


@pytest.mark.parametrize("grid", GRIDS, ids=IDS)
def test_steps_match_oracle_and_radix(built_lib, monkeypatch, grid):
    """Four fused steps, the dynamic update in the third: every forward,
    inverse, padded and test-filter pass of the step."""
    nx, ny, nz, kw = grid
    kw = dict(nx=nx, ny=ny, Nz=nz, dt=1e-4, dyn_init=3, cs_count=3, **kw)
    p, o, g = make_pair(precision="mixed", **kw)
    monkeypatch.setenv("LESGO_RFFT", "0")
    _, _, r = make_pair(precision="mixed", **kw)
    for _ in range(4):
        o.step()
    for h in (g, r):
        h.step(4)
        h.sync()
    for f in ("u", "v", "w", "p"):
        e = rel_err(p, f, g.get(f), oracle_field(o, f))
        assert e < 2e-4, (f, e)
        e = rel_err(p, f, g.get(f), r.get(f))
        assert e < (1e-3 if f == "p" else 5e-5), (f, e)
    g.close()
    r.close()


@pytest.mark.parametrize("grid", [GRIDS[1], GRIDS[3], GRIDS[8]], ids=[IDS[1], IDS[3], IDS[8]])
def test_batch_of_uneven_rows_matches_alone(built_lib, grid):
    """Blocks that span the rows of two instances, and a last block that is
    not full, give each instance's own result bit for bit."""
    from lesgo_gb300.solver import LesgoBatch, LesgoGPU
    nx, ny, nz, kw = grid
    kw = dict(nx=nx, ny=ny, Nz=nz, dt=1e-4, dyn_init=2, cs_count=2, precision="mixed", **kw)
    b = LesgoBatch(3, **kw)
    ids = [b.add(1e-4 * (i + 1), 40 + i) for i in range(3)]
    b.step(3)
    b.sync()
    for i, iid in enumerate(ids):
        s = LesgoGPU(zo=1e-4 * (i + 1), **kw)
        s.init_ic(40 + i)
        s.step(3)
        s.sync()
        for f in ("u", "v", "w", "p"):
            assert np.array_equal(s.get(f), b.get(iid, f)), (i, f)
        s.close()
    b.close()


@pytest.mark.parametrize("grid", GRIDS, ids=IDS)
def test_fp64_steps_match_oracle_and_radix(built_lib, monkeypatch, grid):
    """The same passes in FP64: the form's 1e-10 against the oracle, and 1e-11
    against the run-time radix passes (two FP64 transforms of at most 2^16
    points differ by a few 1e-16, which four steps of dt = 1e-4 do not
    amplify beyond the pressure's division by dt)."""
    nx, ny, nz, kw = grid
    kw = dict(nx=nx, ny=ny, Nz=nz, dt=1e-4, dyn_init=3, cs_count=3, **kw)
    p, o, g = make_pair(**kw)
    monkeypatch.setenv("LESGO_RFFT", "0")
    _, _, r = make_pair(**kw)
    for _ in range(4):
        o.step()
    for h in (g, r):
        h.step(4)
        h.sync()
    for f in ("u", "v", "w", "p"):
        e = rel_err(p, f, g.get(f), oracle_field(o, f))
        assert e < 1e-10, (f, e)
        e = rel_err(p, f, g.get(f), r.get(f))
        assert e < 1e-11, (f, e)
    g.close()
    r.close()


@pytest.mark.parametrize("grid", GRIDS, ids=IDS)
def test_double_word_steps_match_oracle_and_radix(built_lib, monkeypatch, grid):
    """The y passes that the double-word form has: 1e-10 against the oracle,
    and 1e-11 against the run-time radix passes (transforms whose operations
    round at 2^-46 or so, 1.4e-14, a few tens of them in a chain)."""
    nx, ny, nz, kw = grid
    kw = dict(nx=nx, ny=ny, Nz=nz, dt=1e-4, dyn_init=3, cs_count=3, **kw)
    p, o, g = make_pair(precision="fp64dw", **kw)
    monkeypatch.setenv("LESGO_RFFT", "0")
    _, _, r = make_pair(precision="fp64dw", **kw)
    for _ in range(4):
        o.step()
    for h in (g, r):
        h.step(4)
        h.sync()
    for f in ("u", "v", "w", "p"):
        e = rel_err(p, f, g.get(f), oracle_field(o, f))
        assert e < 1e-10, (f, e)
        e = rel_err(p, f, g.get(f), r.get(f))
        assert e < 1e-11, (f, e)
    g.close()
    r.close()
