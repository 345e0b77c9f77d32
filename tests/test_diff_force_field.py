"""The force field of differentiated runs: what lbib_diff_end restores, and the
tiles that a run with moving nodes reads, against central differences of the
same forward (tolerance as in test_adjoint_motion.py: 1e-4 relative plus 1e-7 of
the gradient's scale)."""
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


def _flow(sim, u):
    """The whole fluid at velocity u."""
    c = np.array([[0, 0], [1, 0], [0, 1], [-1, 0], [0, -1], [1, 1], [-1, 1], [-1, -1], [1, -1]], float)
    w = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    cu = c @ u
    feq = w * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * u @ u)
    sim.set_lattice(f=np.tile(feq[[0, 3, 4, 1, 2, 7, 8, 5, 6]], (96 * 96, 1)))


class _Run:
    def __init__(self, lbib, tmp_path, where, precision=0):
        self.sim = _simulation(lbib, tmp_path, precision)
        if where == "into empty tiles":
            self.sim.step(1)
            _flow(self.sim, np.array([0.2, 0.1]))
        rng = np.random.default_rng(3)
        M = self.sim.sizes()["M"]
        self.F = rng.normal(0.0, 5e-3, (M, 2))
        self.w = rng.normal(size=(1, 96 * 96))
        self.v = rng.normal(size=(M, 2))
        self.tau = np.array([0.9, 1.1])
        self.rates = rng.uniform(0.5e-3, 2e-3, (1, self.sim.domain_count()))
        self.sim.diff_begin(24, 5)
        self.sim.diff_motion(True, self.v)

    def loss(self, F):
        self.sim.diff_forward(F, self.tau, self.rates)
        return float((self.sim.concentrations() * self.w).sum() + (self.sim.diff_positions() * self.v).sum())


@pytest.mark.parametrize("where", ["never stepped", "into empty tiles"])
def test_moving_nodes_read_the_force_wherever_they_are(lbib, tmp_path, where):
    """A handle that made no step and got no force field, whose tiles are all
    empty; nodes that the flow carries 5 lu, into tiles that were empty when
    the tiles were last listed."""
    P = _Run(lbib, tmp_path, where)
    start = P.sim.membrane()[1][:, :2]
    P.loss(P.F)
    end, field = P.sim.diff_positions(), P.sim.lattice().force
    assert np.abs(end - start).max() > (4.0 if where == "into empty tiles" else 1e-4)
    # the field of the last step is that of the forces as they are spread, whole
    np.testing.assert_allclose(field.sum(0), P.F.sum(0), rtol=0, atol=2e-2 * np.abs(P.F).sum())
    assert np.abs(field).max() > 1e-4
    g = P.sim.diff_backward(P.w)
    scale = np.abs(g["force"]).max()
    h = 1e-5
    for i, c in ((0, 0), (len(P.F) // 3, 1), (int(np.argmax(end[:, 0])), 0), (int(np.argmax(end[:, 1])), 1)):
        Fp, Fm = P.F.copy(), P.F.copy()
        Fp[i, c] += h
        Fm[i, c] -= h
        fd = (P.loss(Fp) - P.loss(Fm)) / (2 * h)
        assert abs(g["force"][i, c] - fd) <= 1e-4 * abs(fd) + 1e-7 * scale, (i, c, g["force"][i, c], fd)
    u = np.random.default_rng(7).normal(size=P.F.shape)
    fd = (P.loss(P.F + h * u) - P.loss(P.F - h * u)) / (2 * h)
    got = float((g["force"] * u).sum())
    assert abs(got - fd) <= 1e-4 * abs(fd) + 1e-7 * np.abs(g["force"] * u).sum()
    # the FP32-shifted forward: gradients within 1e-3 of these
    Q = _Run(lbib, tmp_path, where, 1)
    Q.loss(Q.F)
    q = Q.sim.diff_backward(Q.w)
    for key in ("force", "tau", "rates"):
        assert np.abs(q[key] - g[key]).max() <= 1e-3 * np.abs(g[key]).max(), key
