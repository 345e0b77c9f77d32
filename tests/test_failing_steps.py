"""Steps that end in an error while all blocks of a membrane stage are at work:
the error is the one that the first failing element raises, the handle refuses
further work, and another handle on the device is not disturbed."""
import numpy as np
import pytest

from lbibcell_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lbib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lbibcell_b200 import build, runner
    build.build()
    return runner


def _tissue(nodes, extra=()):
    cells = configs.hex_tissue(320, 320, 46.0, 20.0, 2.0, nodes, 0, cols=5, rows=5)
    cells = cells[:len(cells) - len(extra)] + [(25 - k, v) for k, v in enumerate(extra)]
    return configs.Config(name="hex25", nx=320, ny=320, tau_fluid=1.0, iterations=40, report_step=20, cells=cells,
                          species=[configs.Species(configs.SPECIES_NAMES[0], 0.8)])


def _fail(lbib, paths, precision, spoil, code):
    sim = lbib.Simulation(paths, precision)
    if spoil is not None:
        spoil(sim)
    with pytest.raises(lbib.LbibError) as e:
        sim.step(45)
    assert e.value.code == code, e.value
    with pytest.raises(lbib.LbibError) as again:
        sim.step(1)
    assert again.value.code == code
    sim.close()


def _nan_fluid(sim):
    f = sim.lattice().f
    f[:] = np.nan
    sim.set_lattice(f=f)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", ["every crossing", "a ring too long", "a tile too full"])
def test_error_in_a_working_stage(lbib, tmp_path, case, precision):
    """every crossing: undefined positions at all of 17,500 connections, whose
    crossings refuse them; a ring too long: 2,100 nodes in the last of 25 cells,
    which the coarsening refuses; a tile too full: 1,100 (FP64: 800) nodes in
    one force tile, which the force lists or the spread refuse."""
    if case == "every crossing":
        cfg, spoil, code = _tissue(700), _nan_fluid, 40
    elif case == "a ring too long":
        cfg, spoil, code = _tissue(300, [configs.circle(160.3, 160.2, 20.0, 2100)]), None, 70
        cfg.cells = [c for c in cfg.cells if c[0] == 25 or np.hypot(*(c[1].mean(0) - 160.25)) > 41.0]
    else:
        cfg, spoil, code = _tissue(300, [configs.circle(280.4, 40.3, 5.0, 1100 if precision else 800)]), None, 70
        cfg.cells = [c for c in cfg.cells if c[0] == 25 or np.hypot(*(c[1].mean(0) - (280.4, 40.3))) > 28.0]
    paths = cfg.write(str(tmp_path / "failing"))
    other = lbib.Simulation(_tissue(250).write(str(tmp_path / "sound")), precision)
    same = lbib.Simulation(_tissue(250).write(str(tmp_path / "sound")), precision)
    for _ in range(6):
        other.step(5)
        _fail(lbib, paths, precision, spoil, code)
        same.step(5)
        a, b = other.lattice(), same.lattice()
        for k in ("f", "g", "vel", "force", "dom"):
            np.testing.assert_array_equal(getattr(a, k), getattr(b, k), err_msg=k)
        np.testing.assert_array_equal(other.membrane()[1], same.membrane()[1])


def _message(lbib, paths, precision, steps, spoil=None, before=0):
    """The error of a run of one call (steps > 0) or of single steps."""
    sim = lbib.Simulation(paths, precision)
    if spoil is not None:
        spoil(sim)
    if before:
        sim.step(before)
    with pytest.raises(lbib.LbibError) as e:
        if steps:
            sim.step(steps)
        else:
            for _ in range(70):
                sim.step(1)
    sim.close()
    return str(e.value)


def _flow(sim):
    """The whole fluid at 0.35 lattice units per step."""
    c = np.array([[0, 0], [1, 0], [0, 1], [-1, 0], [0, -1], [1, 1], [-1, 1], [-1, -1], [1, -1]], float)
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    u = np.array([0.35, 0.0])
    cu = c @ u
    feq = w * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * u @ u)
    lat = sim.lattice()
    sim.set_lattice(f=np.tile(feq[[0, 3, 4, 1, 2, 7, 8, 5, 6]], (lat.f.shape[0], 1)))


def _long_ring(force=0.0):
    """A ring of 3,000 nodes which the remeshing of iteration 1 doubles, past
    what the ring order takes.  Were the run to go on, iteration 10 would refuse
    to coarsen it, and strong forces would move nodes too fast before."""
    cfg = configs.Config(name="ring", nx=640, ny=640, tau_fluid=1.0, iterations=200, report_step=100,
                         cells=[(1, configs.circle(320.3, 320.2, 300.0, 3000))],
                         species=[configs.Species(configs.SPECIES_NAMES[0], 0.8)], current_iteration=1,
                         forces=[f"2\t{k}\t{force}\t0.0" for k in range(100, 120)])
    return cfg


def _long_ring_slow():
    return _long_ring(0.05)


def _long_ring_fast():
    return _long_ring(0.4)


def _many_changes():
    """225 cells carried by the flow: more nodes change their domain in a step
    than the re-initialisation takes (4096)."""
    cells = configs.hex_tissue(800, 800, 46.0, 20.0, 1.0, 260, 1, cols=15, rows=17)
    return configs.Config(name="many", nx=800, ny=800, tau_fluid=1.0, iterations=200, report_step=100, cells=cells,
                          species=[configs.Species(configs.SPECIES_NAMES[0], 0.8)])


def _crowded_tile():
    """Cells of radius 1.4 side by side, whose nodes the remeshing of iteration 0
    doubles: more than 768 stencils in one force tile at iteration 1."""
    cells = [(1 + 16 * j + i, configs.circle(8.3 + 3.0 * i, 8.2 + 3.0 * j, 1.4, 10, phase=0.1 * i + 0.2 * j))
             for j in range(16) for i in range(16)]
    return configs.Config(name="crowd", nx=64, ny=64, tau_fluid=1.0, iterations=200, report_step=100, cells=cells,
                          species=[], area=None)


@pytest.mark.parametrize("make, spoil, precision, expected", [
    (_long_ring_slow, None, 0, "device error 70 at stage 13, iteration 1"),
    (_long_ring_fast, None, 0, "device error 70 at stage 13, iteration 1"),
    (_many_changes, _flow, 0, "device error 70 at stage 7, iteration"),
    (_many_changes, _flow, 1, "device error 70 at stage 7, iteration"),
    (_crowded_tile, None, 0, "device error 70 at stage 2, iteration 1"),
], ids=["ring order beside", "ring order beside, strong forces", "re-initialisation beside fp64",
        "re-initialisation beside fp32", "spread of the next step"])
def test_error_is_the_same_however_the_steps_are_called(lbib, tmp_path, make, spoil, precision, expected):
    """Error, stage, iteration and index, in graphs of one and of ten steps and
    in single calls: an error beside the main sequence ends the run at its step,
    with its own stage, whatever later stages and the next step's forces raise.
    (Of several tiles that are too full the main sequence names the first one
    to raise the error, whichever that is.)"""
    paths = make().write(str(tmp_path))
    part = slice(None, None) if make is not _crowded_tile else slice(0, 1)
    single = _message(lbib, paths, precision, 0, spoil).split(" (index")[part]
    assert expected in single[0]
    for _ in range(4):
        for steps in (64, 70, 9):
            assert _message(lbib, paths, precision, steps, spoil).split(" (index")[part] == single
