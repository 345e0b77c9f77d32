"""The four-nodes-per-thread stream-collide kernel (LBIB_COLLIDE_X4=1) inside
graphs of ten steps, where it follows a join of several streams: the states of
long calls equal the one-node-per-thread kernel's to the last bit.  Rows of 256
nodes exactly and of 512, with cells that remesh, coarsen and hold each other by
junctions, so that the joined streams have work."""
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


def _tissue(nx, ny, cols, rows, species, nodes):
    cells = configs.hex_tissue(nx, ny, 44.0, 20.0, 2.0, nodes, 1, cols=cols, rows=rows)
    sp = [configs.Species(configs.SPECIES_NAMES[k], (0.8, 1.2, 1.0)[k], decay=1e-4 * k, source={1: 1e-3, 4: 2e-3})
          for k in range(species)]
    return configs.Config(name="strip", nx=nx, ny=ny, tau_fluid=1.0, iterations=400, report_step=100, cells=cells,
                          species=sp, tension=(0.05, 10), bio=["LbibCellJunction\tradius\t1.0\tk\t0.02\tl0\t2.0"])


@pytest.mark.parametrize("nx,ny,cols,rows,species,nodes", [(256, 181, 4, 3, 0, 240), (256, 200, 4, 3, 1, 700),
                                                            (512, 256, 10, 5, 2, 220), (512, 137, 10, 2, 3, 600)])
def test_four_nodes_per_thread_equal_one_in_long_calls(lbib, tmp_path, monkeypatch, nx, ny, cols, rows, species, nodes):
    paths = _tissue(nx, ny, cols, rows, species, nodes).write(str(tmp_path))
    states = []
    for x4 in ("0", "1"):
        monkeypatch.setenv("LBIB_COLLIDE_X4", x4)
        sim = lbib.Simulation(paths, lbib.FP32_SHIFTED)
        out = []
        for n in (64, 87, 41):
            sim.step(n)
            lat = sim.lattice()
            out += [lat.f, lat.g, lat.vel, lat.force, lat.dom, sim.membrane()[1], sim.connections()]
        states.append(out)
        sim.close()
    for a, b in zip(*states):
        np.testing.assert_array_equal(a, b)
