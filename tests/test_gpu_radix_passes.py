"""The run-time radix passes, which serve the lengths without register
transforms and most of the double-word form, held to what the register passes
are: with LESGO_RFFT=0 every pass of the FP64 and mixed forms is one of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def handle(**kw):
    from lesgo_gb300.solver import LesgoGPU
    return LesgoGPU(dyn_init=3, cs_count=3, **kw)


def tags(g):
    g.profile(True)
    g.step(1)
    t = g.profile_report()
    g.profile(False)
    return t


@pytest.mark.parametrize("precision", ["mixed", "fp64dw"])
def test_handles_of_different_grids_replay_together(built_lib, monkeypatch, precision):
    """Handles of different grids share the run-time kernels' instances, whose
    blocks need different amounts of dynamic shared memory (the one-pass
    convective rows: 65.7, 65.1 and 65.3 KB mixed, 109.5, 86.8 and 97.9 KB
    double-word).  Stepped in turn with graph replay, each equals its run
    alone bit for bit."""
    if precision == "mixed":
        monkeypatch.setenv("LESGO_RFFT", "0")
    grids = [(64, 64, 16), (128, 64, 16), (96, 48, 16)]
    hs = [handle(nx=g[0], ny=g[1], Nz=g[2], precision=precision) for g in grids]
    for i, h in enumerate(hs):
        h.init_ic(20 + i)
    for _ in range(7):
        for h in hs:
            h.step(1)
    for i, (g, h) in enumerate(zip(grids, hs)):
        a = handle(nx=g[0], ny=g[1], Nz=g[2], precision=precision)
        a.init_ic(20 + i)
        a.step(7)
        for f in ("u", "w", "p"):
            assert np.array_equal(a.get(f)[1:a.nz], h.get(f)[1:h.nz]), (g, f)
        t = tags(a)
        assert "convec.rows" in t and "convec.ypass_vpad" not in t
        a.close()
        h.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_y_pass_shortcuts_match_transforms(built_lib, monkeypatch, precision):
    """The run-time y pass's transform-free outputs against the same steps
    with every output transformed (LESGO_YSHORTCUT=0), over two dynamic
    updates.  Bars: the two routes' round-off after seven steps, 1e-13 of
    the largest value in FP64 and 2e-5 in FP32."""
    monkeypatch.setenv("LESGO_RFFT", "0")
    kw = dict(nx=64, ny=48, Nz=24, precision=precision)
    monkeypatch.setenv("LESGO_YSHORTCUT", "0")
    a = handle(**kw)
    monkeypatch.delenv("LESGO_YSHORTCUT")
    b = handle(**kw)
    for g in (a, b):
        g.init_ic(9)
        g.step(7)
        g.sync()
    tol = {"fp64": 1e-13, "mixed": 2e-5}[precision]
    for f in ("u", "v", "w", "p", "F_LM", "F_MM"):
        x, y = a.get(f)[1:a.nz, :, :64], b.get(f)[1:b.nz, :, :64]
        assert np.max(np.abs(x - y)) <= tol * np.max(np.abs(x)), f
    assert "convec.ypass_vpad" not in tags(b)
    a.close()
    b.close()


@pytest.mark.parametrize("shape", [(1024, 32768), (4096, 112640)], ids=lambda s: "%d,%d" % s)
@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64dw"])
def test_tile_shapes_do_not_change_results(built_lib, monkeypatch, precision, shape):
    """Steps at the smallest and the largest tiles equal those at the default
    ones bit for bit."""
    monkeypatch.setenv("LESGO_RFFT", "0")
    kw = dict(nx=48, ny=32, Nz=24, precision=precision)
    a = handle(**kw)
    monkeypatch.setenv("LESGO_XTARGET", str(shape[0]))
    monkeypatch.setenv("LESGO_YBUDGET", str(shape[1]))
    b = handle(**kw)
    for g in (a, b):
        g.init_ic(1)
        g.step(7)
    for f in ("u", "v", "w", "p", "RHSx", "Cs_opt2", "F_LM"):
        assert np.array_equal(a.get(f)[1:a.nz, :, :48], b.get(f)[1:b.nz, :, :48]), f
    a.close()
    b.close()


def test_autotune_keeps_state(built_lib, monkeypatch):
    """A tuned mixed-form run of run-time passes equals an untuned one."""
    monkeypatch.setenv("LESGO_RFFT", "0")
    kw = dict(nx=48, ny=32, Nz=24, precision="mixed")
    a, b = handle(**kw), handle(**kw)
    for g in (a, b):
        g.init_ic(1)
        g.step(3)
    cfg = a.autotune()
    assert cfg["xtarget"] in (1024, 2048, 4096) and cfg["ybudget"] in (32768, 49152, 65536, 112640)
    for g in (a, b):
        g.step(4)
    for f in ("u", "v", "w", "p", "RHSx", "Cs_opt2", "F_LM"):
        assert np.array_equal(a.get(f)[1:a.nz, :, :48], b.get(f)[1:b.nz, :, :48]), f
    a.close()
    b.close()


@pytest.mark.parametrize("precision,nx,ny,x,y", [("mixed", 48, 32, False, False), ("mixed", 64, 16, False, True),
                                                 ("mixed", 24, 32, True, False), ("fp64", 48, 32, True, False),
                                                 ("fp64dw", 48, 32, True, True)])
def test_autotune_leaves_shapes_that_nothing_reads(built_lib, monkeypatch, precision, nx, ny, x, y):
    """Only the tile shapes of passes that the step launches are tuned (x: the
    x or 3/2-grid row passes are run-time ones; y: some y pass is)."""
    monkeypatch.setenv("LESGO_XTARGET", "512")
    monkeypatch.setenv("LESGO_YBUDGET", "20000")
    g = handle(nx=nx, ny=ny, Nz=12, precision=precision)
    g.init_ic(1)
    cfg = g.autotune()
    assert (cfg["xtarget"] == 512) != x and (cfg["ybudget"] == 20000) != y, cfg
    g.close()
