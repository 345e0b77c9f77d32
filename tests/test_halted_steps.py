"""Steps queued behind one that halts for a host event (a membrane node, a
connection or a new node that the host has to perturb) change nothing: a call of
many steps gives, to the last bit, what single steps give, whatever was queued
behind the halt (renewals of the force list, cell junctions, the resets of the
boundary nodes that the next step uses), and, where the oracle has the solvers,
the oracle's result.  The events fall on iterations that are not multiples of 10, inside a
batch that crosses several, and, once the handle has steps enough, inside a
graph of ten steps."""
import math

import numpy as np
import pytest

from lbibcell_b200 import configs

pytestmark = pytest.mark.gpu

A = configs.SPECIES_NAMES[0]


@pytest.fixture(scope="module")
def lbib():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from lbibcell_b200 import build, runner
    build.build()
    return runner


def _state(sim):
    lat = sim.lattice()
    ids, node = sim.membrane()
    dom, area = sim.areas_array()
    out = {k: getattr(lat, k) for k in ("f", "g", "vel", "force", "dom", "ctype")}
    out.update(ids=ids, node=node, conn=sim.connections(), area_dom=np.array(dom), area=np.array(area))
    out.update({"forces_" + k: v for k, v in sim.forces().items()})
    return out


def _equal(a, b):
    for name in a:
        np.testing.assert_array_equal(a[name], b[name], err_msg=name)


def _single_steps(sim, n):
    """n calls of one step; the iterations at which host events happened."""
    at, before = [], sim.sizes()["host_events"]
    for _ in range(n):
        it = sim.sizes()["iteration"]
        sim.step(1)
        now = sim.sizes()["host_events"]
        at += [it] * (now - before)
        before = now
    return at


def _remesh_at_4(**kw):
    """Starts at iteration 4, whose remeshing makes new nodes on the line
    y = 32 (120 nodes at odd multiples of pi/120 around a lattice node): the
    host perturbs them.  The loaded forces act far from those nodes."""
    cfg = configs.toy(n=64, r=12.0, nodes=120, iterations=200, report_step=50, species=1)
    cfg.cells = [(1, configs.circle(32.0, 32.0, 12.0, 120, phase=math.pi / 120))]
    cfg.current_iteration = 4
    for key, value in kw.items():
        setattr(cfg, key, value)
    return cfg


LOADED = ["2\t31\t0.01\t0.02", "0\t29\t33\t0.05\t0.4", "2\t90\t-0.02\t0.01"]
REMESH = {
    # the list is loaded and lasts to the clearing at iteration 10
    "loaded forces": dict(forces=LOADED, tension=(0.05, 10)),
    "loaded forces alone": dict(forces=LOADED, tension=None),
    # the renewal at iteration 7 edits a list that holds other forces
    "renewal of a mixed list": dict(forces=LOADED, tension=(0.05, 7)),
    "tension every third": dict(tension=(0.05, 3)),
    # the boundary nodes that iteration 4 leaves are used by iteration 5
    "no-flux": dict(boundary=[("BoundarySolverNoFluxD2Q5", A)], tension=(0.05, 10)),
    "bounce-back": dict(species=[configs.Species("DiracD2Q5", 1.0)], area=None, tension=(0.05, 10)),
}


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("case", sorted(REMESH))
def test_remeshing_event_in_a_batch(lbib, oracle_mod, tmp_path, case, precision):
    cfg = _remesh_at_4(**REMESH[case])
    paths = cfg.write(str(tmp_path))
    x, y = lbib.Simulation(paths, precision), lbib.Simulation(paths, precision)
    x.step(31)
    assert _single_steps(y, 31) == [4]
    assert x.sizes()["host_events"] == 1
    a, b = _state(x), _state(y)
    _equal(a, b)
    if precision == lbib.FP64 and case not in ("no-flux", "bounce-back"):
        o = oracle_mod.Oracle(paths)
        o.step(31)
        st = o.state()
        _equal({k: a[k] for k in ("f", "g", "vel", "force", "dom", "ctype", "ids", "node", "conn")},
               {k: getattr(st, k) for k in ("f", "g", "vel", "force", "dom", "ctype", "ids", "node", "conn")})


def _quad(shift):
    """Two pairs of cells within junction distance, moved by `shift` in x."""
    cfg = configs.junction_quad(tension=(0.3, 10))
    cfg.area = (1.3, 0.02, 0.004)
    cfg.cells = [(d, v + [shift, 0.0]) for d, v in cfg.cells]
    return cfg


def _single(shift):
    cfg = configs.toy(n=64, r=12.0, nodes=200, iterations=200, report_step=50, species=2)
    cfg.cells = [(1, configs.circle(32.2 + shift, 31.7, 12.0, 200, phase=0.3))]
    cfg.tension = (0.3, 5)
    return cfg


@pytest.mark.parametrize("make, iteration, n, precision", [
    (_quad, 15, 60, 0), (_quad, 15, 60, 1), (_quad, 57, 90, 0), (_quad, 57, 90, 1), (_single, 23, 60, 0)],
    ids=["junctions at 15 fp64", "junctions at 15 fp32", "junctions at 57 fp64", "junctions at 57 fp32",
         "one cell at 23 fp64"])
def test_moved_node_event_in_a_graph_of_ten_steps(lbib, oracle_mod, tmp_path, make, iteration, n, precision):
    """The geometry is shifted until the step of that iteration moves a
    node to within 1e-9 of a lattice line, where the reference perturbs it."""
    rng = np.random.default_rng(iteration)
    shift, target = 0.0, None
    # (in FP32-shifted runs the last digits are rounding: a matter of attempts)
    for attempt in range(12 if precision == lbib.FP64 else 80):
        paths = make(shift).write(str(tmp_path / str(attempt)))
        sim = lbib.Simulation(paths, precision)
        at = _single_steps(sim, iteration + 1)
        if at == [iteration]:
            break
        ids, node = sim.membrane()
        if target is None:  # the node nearest to a line in the undisturbed run
            target = ids[np.argmin(np.abs(node[:, 0] - np.round(node[:, 0])))]
        x = node[np.flatnonzero(ids == target)[0], 0]
        shift -= x - round(x) + (0.0 if precision == lbib.FP64 else rng.uniform(-1e-8, 1e-8))
        sim.close()
    assert at == [iteration], f"no event at iteration {iteration}: {at}"
    assert _single_steps(sim, n - iteration - 1) == []
    whole = lbib.Simulation(paths, precision)
    whole.step(n)
    assert whole.sizes()["host_events"] == 1
    a = _state(whole)
    _equal(a, _state(sim))
    if precision == lbib.FP64 and make is _single:
        o = oracle_mod.Oracle(paths)
        o.step(n)
        st = o.state()
        _equal({k: a[k] for k in ("f", "g", "vel", "force", "dom", "ctype", "ids", "node", "conn")},
               {k: getattr(st, k) for k in ("f", "g", "vel", "force", "dom", "ctype", "ids", "node", "conn")})


@pytest.mark.parametrize("precision", [0, 1])
def test_new_node_event_at_a_coarsening_step(lbib, oracle_mod, tmp_path, precision):
    """A growing cell is remeshed in iterations 7 to 13.  The geometry is
    shifted until a node made at iteration 10, a coarsening step, lies on a
    lattice line: the step halts with the pass applied and not committed, and
    with a ring order that the passes before have outdated."""
    rng = np.random.default_rng(10)
    shift = 0.0
    for attempt in range(12 if precision == lbib.FP64 else 80):
        cfg = configs.toy(n=64, r=12.0, nodes=155, iterations=200, report_step=50, species=1)
        cfg.cells = [(1, configs.circle(32.2 + shift, 31.7, 12.0, 155, phase=0.3))]
        cfg.tension, cfg.area = (0.1, 10), (3.0, 0.2, 0.05)
        paths = cfg.write(str(tmp_path / str(attempt)))
        sim = lbib.Simulation(paths, precision)
        at = _single_steps(sim, 10)
        before = sim.membrane()[0]
        at += _single_steps(sim, 1)
        if at == [10]:
            break
        ids, node = sim.membrane()
        assert len(before) > 155 and len(ids) > len(before)
        x = node[np.isin(ids, np.setdiff1d(ids, before)), 0]
        off = x - np.round(x)
        shift -= off[np.argmin(np.abs(off))] + (0.0 if precision == lbib.FP64 else rng.uniform(-1e-8, 1e-8))
        sim.close()
    assert at == [10], f"no event at iteration 10: {at}"
    assert _single_steps(sim, 44 - 11) == []
    whole = lbib.Simulation(paths, precision)
    whole.step(44)
    assert whole.sizes()["host_events"] == 1
    a = _state(whole)
    _equal(a, _state(sim))
    if precision == lbib.FP64:
        o = oracle_mod.Oracle(paths)
        o.step(44)
        st = o.state()
        _equal({k: a[k] for k in ("f", "g", "vel", "force", "dom", "ctype", "ids", "node", "conn")},
               {k: getattr(st, k) for k in ("f", "g", "vel", "force", "dom", "ctype", "ids", "node", "conn")})
