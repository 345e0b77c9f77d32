"""The read-out of the state: arrays larger than one chunk (1 MB), cut at
places inside a node's values and inside a part, equal what was uploaded, and
equal the same arrays read one at a time."""
import ctypes

import numpy as np
import pytest

from lbibcell_b200 import configs

pytestmark = pytest.mark.gpu

W = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)[[0, 3, 4, 1, 2, 7, 8, 5, 6]]


@pytest.fixture(scope="module")
def lbib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lbibcell_b200 import build, runner
    build.build()
    return runner


def _p(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("nx, ny, species", [(48, 48, 1), (123, 77, 2), (301, 517, 3), (64, 1025, 1)])
def test_read_out_equals_upload(lbib, tmp_path, nx, ny, species, precision):
    cfg = configs.toy(n=48, species=species)
    cfg.nx, cfg.ny = nx, ny
    cfg.cells = [(1, configs.circle(24.2, 24.3, 9.0, 100)), (2, configs.circle(nx - 18.1, ny - 18.4, 9.0, 120))]
    if nx < 60 and ny < 60:
        cfg.cells = cfg.cells[:1]
    sim = lbib.Simulation(cfg.write(str(tmp_path)), precision)
    rng = np.random.default_rng(nx)
    L = nx * ny
    f, g, force = W + 1e-2 * rng.normal(size=(L, 9)), rng.normal(size=(species, L, 5)), rng.normal(size=(L, 2))
    sim.set_lattice(f, g, force)
    if precision:
        f = (f - W).astype(np.float32).astype(np.float64) + W
        g, force = (a.astype(np.float32).astype(np.float64) for a in (g, force))
    a = sim.lattice()
    for name, want in (("f", f), ("g", g), ("force", force)):
        assert np.array_equal(getattr(a, name), want), name
    assert np.array_equal(sim.concentrations(), a.g.sum(axis=2))
    # one array per call
    vel, dom, ctype = np.full((L, 2), np.nan), np.full(L, 9, np.uint32), np.full(L, 9, np.uint32)
    for slot, array in ((3, vel), (5, dom), (6, ctype)):
        args = [None] * 6
        args[slot - 1] = _p(array)
        assert sim._L.lbib_download_lattice(sim._h, *args) == 0
    assert np.array_equal(a.vel, vel) and np.array_equal(a.dom, dom) and np.array_equal(a.ctype, ctype)
    assert set(np.unique(dom)) == set(range(1 + len(cfg.cells)))


def test_read_out_of_a_large_membrane(lbib, tmp_path):
    """25 cells of 700 nodes: ids, states and connections over several chunks,
    before and after the first steps' topology changes."""
    cells = configs.hex_tissue(320, 320, 46.0, 20.0, 2.0, 700, 0, cols=5, rows=5)
    cfg = configs.Config(name="hex25", nx=320, ny=320, tau_fluid=1.0, iterations=40, report_step=20, cells=cells,
                         species=[configs.Species(configs.SPECIES_NAMES[0], 0.8)])
    sim = lbib.Simulation(cfg.write(str(tmp_path)), 0)
    ids, state = sim.membrane()
    assert np.array_equal(ids, np.arange(1, 1 + 25 * 700))
    assert np.array_equal(state[:, :2], np.concatenate([v for _, v in cells])) and not state[:, 2:].any()
    conn = sim.connections()
    assert conn.shape == (25 * 700, 3) and np.array_equal(conn[:, 0], ids)
    assert np.array_equal(conn[:, 2], np.repeat(np.arange(1, 26), 700))
    sim.step(21)
    ids, state = sim.membrane()
    assert (np.diff(ids.astype(np.int64)) > 0).all() and np.isfinite(state).all() and state[:, 4:].any()
    conn = sim.connections()
    assert set(conn[:, 0]) == set(ids) == set(conn[:, 1])
