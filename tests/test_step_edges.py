"""Full steps at the sizes where a stage kernel's partition can go wrong:
membranes of one node less and more than a warp, a block and a force tile's
list hold, lattice rows of one node more than a block and a 32-node segment
cover, one cell and several.  FP64 runs are exact against the oracle;
FP32-shifted runs stay within FP32 rounding of the FP64 run (about 20 steps
of 1e-7 each, positions in FP64)."""
import numpy as np
import pytest

from lbibcell_b200 import configs

pytestmark = pytest.mark.gpu

# nx, ny, cells (x, y, radius, nodes), species, steps
SIZES = {
    "8 nodes less one": (48, 48, [(24.3, 24.1, 3.0, 7)], 1, 12),
    "33 nodes": (33, 47, [(16.4, 23.2, 8.0, 33)], 1, 12),
    "row of 65": (65, 40, [(31.7, 20.2, 12.0, 151)], 2, 22),
    "row of 257": (257, 33, [(100.3, 16.6, 9.0, 128), (230.1, 16.3, 9.5, 129)], 3, 22),
    "dense tile list": (48, 50, [(24.2, 25.3, 5.0, 300)], 1, 12),
    "dense, coarsened": (64, 64, [(32.2, 31.3, 9.0, 700)], 2, 22),
    "256 nodes, coarsened": (48, 48, [(24.2, 24.3, 4.0, 256)], 1, 12),
    "one of two coarsened, 513 nodes": (72, 48, [(20.2, 24.3, 4.0, 453), (50.1, 23.2, 9.6, 60)], 1, 22),
    "column of 600": (40, 600, [(20.2, 40.0 + 130.0 * k, 9.0 + k, 110 + 19 * k) for k in range(5)], 1, 22),
}


@pytest.fixture(scope="module")
def lbib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lbibcell_b200 import build, runner
    build.build()
    return runner


def _cfg(size):
    nx, ny, cells, species, steps = SIZES[size]
    cfg = configs.toy(n=48, iterations=steps, report_step=steps, species=species)
    cfg.nx, cfg.ny = nx, ny
    cfg.cells = [(k + 1, configs.circle(x, y, r, n, phase=0.1 + k)) for k, (x, y, r, n) in enumerate(cells)]
    return cfg, steps


@pytest.mark.parametrize("size", sorted(SIZES))
def test_fp64_steps_equal_the_oracle(lbib, oracle_mod, tmp_path, size):
    cfg, steps = _cfg(size)
    paths = cfg.write(str(tmp_path))
    sim, o = lbib.Simulation(paths, lbib.FP64), oracle_mod.Oracle(paths)
    sim.step(steps)
    o.step(steps)
    a, st = sim.lattice(), o.state()
    for name in ("f", "g", "vel", "force", "dom", "ctype"):
        assert np.array_equal(getattr(a, name), getattr(st, name)), name
    ids, node = sim.membrane()
    assert np.array_equal(ids, st.ids) and np.array_equal(node, st.node)
    assert np.array_equal(sim.connections(), st.conn)


@pytest.mark.parametrize("size", sorted(SIZES))
def test_fp32_steps_close_to_fp64(lbib, tmp_path, size):
    cfg, steps = _cfg(size)
    paths = cfg.write(str(tmp_path))
    x, y = lbib.Simulation(paths, lbib.FP32_SHIFTED), lbib.Simulation(paths, lbib.FP64)
    x.step(steps)
    y.step(steps)
    a, b = x.lattice(), y.lattice()
    for name in ("f", "g", "vel", "force"):
        u, v = getattr(a, name), getattr(b, name)
        assert np.abs(u - v).max() <= 1e-5 * np.abs(v).max(), name
    assert np.array_equal(a.dom, b.dom)
    (ia, na), (ib, nb) = x.membrane(), y.membrane()
    assert np.array_equal(ia, ib) and np.abs(na[:, :2] - nb[:, :2]).max() <= 1e-6
