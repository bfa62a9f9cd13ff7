"""Grids of which only one direction has register transforms: register x
passes with run-time radix y passes (nx listed, ny not) and the reverse.  The
fused step then forms the vorticity from the gradients, behind the column
pass, and the register inverse x passes read spectra that a run-time y pass
wrote (and the reverse).  Fused steps with two dynamic updates against the
oracle, under every pair of boundary treatments, and the moving no-slip wall
where the vorticity comes from the velocity's modes.

Bars: the forms' own against the oracle, 1e-10 for FP64 and double-word and
2e-4 for the mixed form.  Which passes ran is read from the step's profile:
`convec.ypass_vpad` is launched where both directions are register passes and
`convec.ypass_pad` elsewhere, so that a length that leaves a list fails here."""
import pytest

from gpu_util import make_pair, oracle_field, rel_err

pytestmark = pytest.mark.gpu

X_ONLY = [(108, 162, 12), (64, 16, 9)]
Y_ONLY = [(24, 32, 12), (16, 54, 7)]
BOUNDARIES = [dict(), dict(lbc_mom=0, ubc_mom=0), dict(lbc_mom=1, ubc_mom=1, molec=True), dict(lbc_mom=2, ubc_mom=2)]
BAR = {"fp64": 1e-10, "fp64dw": 1e-10, "mixed": 2e-4}


def check(precision, grid, kw, vpad):
    nx, ny, nz = grid
    p, o, g = make_pair(precision=precision, nx=nx, ny=ny, Nz=nz, dt=1e-4, dyn_init=2, cs_count=2, **kw)
    for _ in range(4):
        o.step()
    g.step(4)
    g.sync()
    for f in ("u", "v", "w", "p"):
        e = rel_err(p, f, g.get(f), oracle_field(o, f))
        assert e < BAR[precision], (f, e)
    g.profile(True)
    g.step(1)
    ran = g.profile_report()
    g.profile(False)
    assert ("convec.ypass_vpad" in ran) == vpad and ("convec.ypass_pad" in ran) != vpad, sorted(ran)
    g.close()


@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64dw"])
@pytest.mark.parametrize("grid", X_ONLY + Y_ONLY, ids=lambda g: "%dx%dx%d" % g)
def test_one_listed_direction(built_lib, precision, grid):
    check(precision, grid, {}, False)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("bc", BOUNDARIES[1:], ids=lambda b: ",".join("%s=%s" % i for i in b.items()))
@pytest.mark.parametrize("grid", [X_ONLY[1], Y_ONLY[0]], ids=lambda g: "%dx%dx%d" % g)
def test_boundaries(built_lib, precision, bc, grid):
    check(precision, grid, bc, False)


@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64dw"])
@pytest.mark.parametrize("grid", [(48, 36, 12), (64, 16, 9)], ids=lambda g: "%dx%dx%d" % g)
def test_moving_bottom_wall(built_lib, precision, grid):
    """The no-slip wall's velocity is taken off the mean mode of u."""
    check(precision, grid, dict(lbc_mom=1, molec=True, ubot=3.0), grid == (48, 36, 12) and precision != "fp64dw")


NX = [32, 36, 48, 64, 72, 96, 108, 128, 144, 192, 216, 256]
NY = [24, 32, 36, 48, 54, 64, 72, 96, 108, 128, 144, 192, 216, 256]


@pytest.mark.parametrize("nx,ny", [(NX[i % len(NX)], ny) for i, ny in enumerate(NY)])
def test_listed_lengths_take_the_register_passes(built_lib, nx, ny):
    """(Where they did not, a comparison with the run-time passes would be
    one of these with themselves.)"""
    from lesgo_gb300.solver import LesgoGPU
    g = LesgoGPU(nx=nx, ny=ny, Nz=4, precision="mixed")
    g.init_ic(1)
    g.profile(True)
    g.step(1)
    assert "convec.ypass_vpad" in g.profile_report()
    g.close()
