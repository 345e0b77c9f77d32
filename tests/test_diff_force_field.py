"""The force field of differentiated runs: what lbib_diff_end restores."""
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


def _simulation(lbib, tmp_path, precision):
    cfg = configs.toy(n=96, r=10.0, nodes=100, iterations=100, species=1)
    cfg.area = None
    return lbib.Simulation(cfg.write(str(tmp_path)), precision)


def _same(a, b):
    for k in ("f", "g", "vel", "force", "dom", "ctype"):
        np.testing.assert_array_equal(getattr(a, k), getattr(b, k), err_msg=k)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("motion", [False, True])
@pytest.mark.parametrize("before", ["an uploaded field", "steps", "nothing"])
def test_end_restores_the_lattice(lbib, tmp_path, before, motion, precision):
    """The lattice before lbib_diff_begin, its force field included, is the one
    after lbib_diff_end, and the lattice steps that follow are the same."""
    sims = [_simulation(lbib, tmp_path, precision) for _ in range(2)]
    rng = np.random.default_rng(5)
    field = rng.normal(0.0, 1e-4, (96 * 96, 2))
    for sim in sims:
        if before == "an uploaded field":
            sim.set_lattice(force=field)
        elif before == "steps":
            sim.step(12)
    sim, other = sims
    at_begin = sim.lattice()
    assert (np.abs(at_begin.force).max() > 0) == (before != "nothing")
    _same(at_begin, other.lattice())
    sim.diff_begin(8, 3)
    if motion:
        sim.diff_motion(True)
    M = sim.sizes()["M"]
    sim.diff_forward(rng.normal(0.0, 1e-2, (M, 2)))
    sim.diff_backward(np.ones((1, 96 * 96)))
    sim.diff_end()
    _same(sim.lattice(), at_begin)
    for s in sims:
        s.lattice_step(3)
    _same(sim.lattice(), other.lattice())
