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
