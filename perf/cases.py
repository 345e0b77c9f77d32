"""The calls whose speed matters to a user of lbibcell_b200.

A case is one pass of a program that uses the package through
lbibcell_b200.runner.Simulation; `kind` names the program:

  run      steps of the whole simulation (membrane forces, spreading, lattice,
           motion, domains, remeshing, bio solvers), then the read-out of a
           report: lattice, membrane, connections, cell areas;
  control  the same advanced one step per call, with the per-cell secretion
           rates of every species sent and the cell areas read back each step,
           as a controller on the host does;
  frozen   lattice steps with the geometry held (a morphogen field settling in
           a fixed tissue), then the lattice;
  adjoint  one gradient evaluation of a differentiated run: T forward steps,
           the concentrations at the end, the quadratic misfit to a target,
           the reverse pass;
  moving   the same with moving membrane nodes and a target for their final
           positions.

The tissues are cells on a hexagonal grid with seeded radii, phases and
secreting cells: radius 20 as in the package's 200^2 and 1024^2
configurations, smaller ones in small lattices.  Their tension is the
reference's tutorial_01 one (0.01, renewed every 10 steps), and an area
regulator holds (tissues) or slowly grows (single cells) each cell, so that a
simulation can be advanced for many passes.  About half of the cells start
with their membrane nodes more than 0.5 lu apart, so that the first steps
remesh and coarsen them.
"""
import math
import os
import tempfile

import numpy as np
import torch

from lbibcell_b200 import configs, runner

TAU_SPECIES = (0.8, 1.2, 1.0)
TAU_FLUID = 1.0
DECAY = 1e-4
RATE = 1e-3
TURING = (("tutorial_02_CDESolverD2Q5_L", 1.0), ("tutorial_02_CDESolverD2Q5_R", 1.2))


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # the smallest lattice of the tests, one cell, exact arithmetic: what a
        # step costs when there is almost no work in it
        {"name": "cell_48_fp64", "kind": "run", "nx": 48, "ny": 48, "cells": "one", "radius": 9.0, "species": 1,
         "precision": "fp64", "steps": 100},
        # a host program that steers one cell step by step
        {"name": "control_64_fp32", "kind": "control", "nx": 64, "ny": 64, "cells": "one", "radius": 12.0,
         "species": 1, "precision": "fp32", "steps": 50},
        # the tutorial's problem (200^2, one cell of radius 20, one species) to
        # its report step, in both precisions
        {"name": "cell_200_fp64", "kind": "run", "nx": 200, "ny": 200, "cells": "one", "radius": 20.0, "species": 1,
         "precision": "fp64", "steps": 500},
        {"name": "cell_200_fp32", "kind": "run", "nx": 200, "ny": 200, "cells": "one", "radius": 20.0, "species": 1,
         "precision": "fp32", "steps": 500},
        # a Turing pattern (tutorial_02's coupled species) in a small tissue of
        # odd size, exact arithmetic
        {"name": "turing_251x187_fp64", "kind": "run", "nx": 251, "ny": 187, "cells": "many", "radius": 20.0,
         "species": 2, "reaction": "turing", "precision": "fp64", "steps": 200},
        # a tissue of odd size with three species
        {"name": "tissue_337x521_fp32", "kind": "run", "nx": 337, "ny": 521, "cells": "many", "radius": 20.0,
         "species": 3, "precision": "fp32", "steps": 500},
        # the benchmark's lattice and 20 x 20 cells: the ordinary large run
        {"name": "tissue_1024_fp32", "kind": "run", "nx": 1024, "ny": 1024, "cells": "many", "radius": 20.0,
         "species": 2, "precision": "fp32", "steps": 500},
        {"name": "tissue_1024_fp64", "kind": "run", "nx": 1024, "ny": 1024, "cells": "many", "radius": 20.0,
         "species": 2, "precision": "fp64", "steps": 300},
        # the same patch of cells in a wide medium: the largest lattice
        {"name": "tissue_2048_fp32", "kind": "run", "nx": 2048, "ny": 2048, "cells": "many", "radius": 20.0,
         "species": 2, "precision": "fp32", "steps": 300},
        # species settling in a fixed tissue, odd size
        {"name": "frozen_701x499_fp64", "kind": "frozen", "nx": 701, "ny": 499, "cells": "many", "radius": 20.0,
         "species": 3, "precision": "fp64", "steps": 1000},
        # gradients: the package's 512^2 workload (50 to 100 cells, one
        # species, a checkpoint every T / 20 steps), with moving nodes in 256^2
        {"name": "adjoint_512_fp64", "kind": "adjoint", "nx": 512, "ny": 512, "cells": "many", "radius": 15.0,
         "species": 1, "precision": "fp64", "steps": 600},
        {"name": "moving_256_fp32", "kind": "moving", "nx": 256, "ny": 256, "cells": "many", "radius": 15.0,
         "species": 1, "precision": "fp32", "steps": 100},
    ]


def draw(rng):
    """One more case of the same ranges: lattices of 48 to 1200 on a side (the
    sides up to 1 : 3), one cell or a patch of them, 1 to 3 species, both
    precisions, passes of 20 to 500 steps (differentiated runs: lattices to
    512, up to 400 steps)."""
    kind = rng.choice(("run", "run", "run", "run", "control", "frozen", "adjoint", "moving"))
    top = 512 if kind in ("adjoint", "moving") else 1200
    low = 96 if kind in ("adjoint", "moving") else 48
    side = math.exp(rng.uniform(math.log(low), math.log(top)))
    aspect = math.exp(rng.uniform(-0.5, 0.5) * math.log(3.0))
    nx = max(48, min(top, int(side * aspect)))
    ny = max(48, min(top, int(side / aspect)))
    most = {"run": 500, "control": 100, "frozen": 400, "adjoint": 400, "moving": 100}[kind]
    steps = int(math.exp(rng.uniform(math.log(20), math.log(most))))
    case = {"kind": kind, "nx": nx, "ny": ny, "cells": rng.choice(("many", "many", "many", "one")),
            "radius": round(min(rng.uniform(9.0, 20.0), (min(nx, ny) - 24) / 2.4), 2),
            "species": rng.choice((1, 1, 2, 2, 3)), "precision": rng.choice(("fp64", "fp32")), "steps": steps}
    if kind == "run" and rng.random() < 0.15:
        case.update(reaction="turing", species=2)
    return case


# ---------------------------------------------------------------------------
# inputs

def tissue(case, seed):
    """[(domain, vertices)]: one cell, or a patch of cells of the case's radius
    (within a tenth) in the middle of the lattice, up to 20 x 20 (the
    benchmark's) of as many as fit with 20 lu to the edges (the mass outlet
    draws a tissue toward x = 0 and y = 0), 5 lu and more between them,
    membrane nodes 0.5 lu apart."""
    rng = np.random.default_rng([int(seed), case["nx"], case["ny"]])
    nx, ny, r0 = case["nx"], case["ny"], case["radius"]
    rmax = 1.1 * r0
    spacing = 2.0 * rmax + 5.0
    dy = spacing * math.sqrt(3.0) / 2.0
    room_x, room_y = nx - 2.0 * (rmax + 20.0), ny - 2.0 * (rmax + 20.0)
    cols = min(20, 1 + max(0, int(room_x / spacing)))
    if cols == 1:
        dy = spacing
    rows = min(20, 1 + max(0, int(room_y / dy)))
    if case["cells"] == "one":
        cols = rows = 1
    w = (cols - 1) * spacing
    x0, y0 = (nx - w) / 2.0, (ny - (rows - 1) * dy) / 2.0
    cells = []
    for row in range(rows):
        odd = row % 2 == 1 and cols > 1
        for col in range(cols - 1 if odd else cols):
            x = x0 + col * spacing + (spacing / 2.0 if odd else 0.0) + rng.uniform(-0.4, 0.4)
            y = y0 + row * dy + rng.uniform(-0.4, 0.4)
            r = r0 * rng.uniform(0.9, 1.1)
            n = max(16, int(round(2.0 * math.pi * r0 / 0.5)))
            cells.append((len(cells) + 1, configs.circle(x, y, r, n, phase=rng.uniform(0.0, 2.0 * math.pi))))
    return cells


def source_table(case, n_cells, seed):
    """Secretion rates [species][domain]: about a tenth of the cells (in
    differentiated runs all of them) at rates of their own."""
    rng = np.random.default_rng([int(seed), 7])
    table = np.zeros((case["species"], n_cells + 1))
    rates = RATE * rng.uniform(0.5, 1.5, (case["species"], n_cells))
    if case["kind"] not in ("adjoint", "moving"):
        rates *= np.arange(n_cells) % 10 == rng.integers(0, min(10, n_cells))
    table[:, 1:] = rates
    return table


def simulation(case, seed):
    cells = tissue(case, seed)
    table = source_table(case, len(cells), seed)
    turing = case.get("reaction") == "turing"
    diff = case["kind"] in ("adjoint", "moving")
    if turing:
        species = [configs.Species(name, tau) for name, tau in TURING]
    else:
        species = [configs.Species(configs.SPECIES_NAMES[k], TAU_SPECIES[k], decay=DECAY,
                                   source={d: float(table[k, d]) for d in range(1, len(cells) + 1) if table[k, d]})
                   for k in range(case["species"])]
    many = len(cells) > 1
    cfg = configs.Config(
        name="case", nx=case["nx"], ny=case["ny"], tau_fluid=TAU_FLUID, iterations=10 ** 6, report_step=1000,
        cells=cells, species=species, tension=(0.01, 10),
        area=None if diff else (1.0 if many else 1.1, 0.0005, 0.004),
        bio=["LbibCellJunction\tradius\t1.0\tk\t0.02\tl0\t2.0"] if many and not diff else [])
    with tempfile.TemporaryDirectory() as directory:
        sim = runner.Simulation(cfg.write(os.path.join(directory, "case")),
                                runner.FP64 if case["precision"] == "fp64" else runner.FP32_SHIFTED)
    return sim, cells, table


def lattice_state(case, seed):
    """A lattice as a run leaves it: density within 1e-3 of 1, velocities of
    1e-3, smooth positive concentrations, and a membrane-like force field.
    In the package's layout: f[L][9], g[S][L][5], force[L][2]."""
    rng = np.random.default_rng([int(seed), 11])
    nx, ny, S = case["nx"], case["ny"], case["species"]
    y, x = np.mgrid[0:ny, 0:nx].astype(float)

    def smooth():
        out = np.zeros((ny, nx))
        for _ in range(3):
            kx, ky = rng.integers(1, 4, 2)
            out += rng.normal() * np.cos(2 * math.pi * (kx * x / nx + ky * y / ny) + rng.uniform(0, 2 * math.pi))
        return out / 3.0

    weight = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)
    rho, ux, uy = 1.0 + 1e-3 * smooth(), 1e-3 * smooth(), 1e-3 * smooth()
    f = np.empty((ny * nx, 9))
    for d in range(9):
        cu = CX[NATURAL9[d]] * ux + CY[NATURAL9[d]] * uy
        f[:, d] = (weight[NATURAL9[d]] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy))).ravel()
    g = np.empty((S, ny * nx, 5))
    for k in range(S):
        c = (0.5 + 0.1 * smooth()).ravel()
        for d in range(5):
            g[k, :, d] = c * (1 / 3 if d == 0 else 1 / 6)
    force = np.stack([1e-5 * smooth().ravel(), 1e-5 * smooth().ravel()], axis=1)
    return f, g, force


def prepare(case, seed):
    sim, cells, table = simulation(case, seed)
    # the report's membrane arrays: room for a membrane that remeshing doubles
    state = {"case": case, "sim": sim, "room": 64 + 3 * sum(len(v) for _, v in cells)}
    if case["kind"] == "control":
        # the tables of the next steps, in pinned host memory
        rng = np.random.default_rng([int(seed), 13])
        n = sim.domain_count()
        tables = torch.zeros((case["steps"], case["species"], n), dtype=torch.float64).pin_memory()
        for t in range(case["steps"]):
            tables[t, :, :table.shape[1]] = torch.from_numpy(table * rng.uniform(0.5, 1.5, table.shape))[:, :n]
        state["tables"] = tables
        state["rates"] = [tables[t].numpy() for t in range(case["steps"])]
        room = sim.sizes()["cells"] + 64
        state["area_domain"] = torch.zeros(room, dtype=torch.int32).pin_memory().numpy().view(np.uint32)
        state["area"] = torch.zeros(room, dtype=torch.float64).pin_memory().numpy()
    elif case["kind"] == "frozen":
        f, g, force = lattice_state(case, seed)
        sim.set_lattice(f, g, force)
    elif case["kind"] in ("adjoint", "moving"):
        sim.set_lattice(*lattice_state(case, seed))
        T = case["steps"]
        sim.diff_begin(T, max(1, T // 20))
        state.update(gradient_inputs(case, cells, table, seed))
        if case["kind"] == "moving":
            sim.diff_motion(True)
    return state


def gradient_inputs(case, cells, table, seed):
    """The parameters of a differentiated run and the targets of its misfit."""
    rng = np.random.default_rng([int(seed), 17])
    S, L = case["species"], case["nx"] * case["ny"]
    nodes = np.concatenate([v for _, v in cells])
    tau = np.array([TAU_FLUID] + list(TAU_SPECIES[:S])) * rng.uniform(0.95, 1.05, 1 + S)
    return {"force": rng.normal(0.0, 1e-3, nodes.shape), "tau": tau, "rates": table,
            "c_target": 0.5 + 0.05 * rng.normal(size=(S, L)), "x_target": nodes + rng.normal(0.0, 0.1, nodes.shape)}


# ---------------------------------------------------------------------------
# one pass

def report(state):
    sim, room = state["sim"], state["room"]
    lattice = sim.lattice()
    domain, area = sim.areas_array()
    out = {"f": lattice.f, "g": lattice.g, "vel": lattice.vel, "force": lattice.force, "dom": lattice.dom,
           "ctype": lattice.ctype, "area_domain": domain.copy(), "area": area.copy()}
    # of one length whatever the remeshing did: the rows past the last are 0
    for name, rows in zip(("ids", "nodes", "connections"), (*sim.membrane(), sim.connections())):
        out[name] = np.zeros((room,) + rows.shape[1:], rows.dtype)
        out[name][:len(rows)] = rows
    return out


def run(state):
    case, sim = state["case"], state["sim"]
    kind = case["kind"]
    if kind == "run":
        sim.step(case["steps"])
        return report(state)
    if kind == "control":
        for rates in state["rates"]:
            sim.set_species_sources(rates)
            sim.step(1)
            sim.areas_into(state["area_domain"], state["area"])
        return report(state)
    if kind == "frozen":
        sim.lattice_step(case["steps"])
        lattice = sim.lattice()
        return {"f": lattice.f, "g": lattice.g, "vel": lattice.vel, "force": lattice.force, "dom": lattice.dom,
                "ctype": lattice.ctype}
    sim.diff_forward(state["force"], state["tau"], state["rates"])
    out = {"c": sim.concentrations()}
    if kind == "moving":
        out["x"] = sim.diff_positions()
        sim.diff_motion(True, 2.0 * (out["x"] - state["x_target"]))
    gradient = sim.diff_backward(2.0 * (out["c"] - state["c_target"]))
    out.update({"d_" + key: value for key, value in gradient.items()})
    if kind == "moving":
        out["d_x"] = sim.diff_positions(grad=True)[1]
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """Every step reads and writes the lattice once (nine fluid and five
    values per species and node), a reverse step reads the state and its
    adjoint and writes the adjoint (FP32); the read-out writes the FP64 report.
    About 250 flops per fluid update and 60 per species update, three times
    that in reverse."""
    S, L, T = case["species"], case["nx"] * case["ny"], case["steps"]
    size = 8 if case["precision"] == "fp64" else 4
    values = 9 + 5 * S
    forward = 2 * values * size * L * T
    flops = (250 + 60 * S) * L * T
    if case["kind"] in ("adjoint", "moving"):
        return {"bytes": forward + (values * size + 2 * values * 4) * L * T + 8 * 3 * S * L, "flops": 4 * flops}
    return {"bytes": forward + 8 * (values + 5) * L, "flops": flops}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits, for the kinds with a fixed topology

# direction order T, E, N, W, S, NE, NW, SW, SE; the stored slot of a
# direction is its inverse's
CX = (0, 1, 0, -1, 0, 1, -1, -1, 1)
CY = (0, 0, 1, 0, -1, 1, 1, -1, -1)
NATURAL9 = (0, 3, 4, 1, 2, 7, 8, 5, 6)
NATURAL5 = (0, 3, 4, 1, 2)
WEIGHT = (4 / 9, 1 / 9, 1 / 9, 1 / 9, 1 / 9, 1 / 36, 1 / 36, 1 / 36, 1 / 36)


def domain_ids(case, cells):
    """Per lattice node the domain of the cell whose polygon it lies in, else 0."""
    dom = np.zeros((case["ny"], case["nx"]), np.int64)
    for d, v in cells:
        x0, y0 = np.floor(v.min(0)).astype(int)
        x1, y1 = np.ceil(v.max(0)).astype(int) + 1
        y, x = np.mgrid[y0:y1, x0:x1].astype(float)
        a, b = v, np.roll(v, -1, 0)
        inside = np.ones(x.shape, bool)
        for (ax, ay), (bx, by) in zip(a, b):  # counter-clockwise and convex
            inside &= (bx - ax) * (y - ay) - (by - ay) * (x - ax) > 0
        dom[y0:y1, x0:x1][inside] = d
    return torch.from_numpy(dom)


def fast_cos(x):
    """The parabola approximation of the cosine that the Dirac weights use."""
    t = x + math.pi / 2
    t = torch.where(t > math.pi, t - 2 * math.pi, t)
    c = 1.27323954 * t - 0.405284735 * t * t.abs()
    return 0.225 * (c * c.abs() - c) + c


def stencil(X, nx):
    """Flat lattice indices and weights of the 4 x 4 nodes around each position."""
    with torch.no_grad():
        base = torch.ceil(X - 2.0)
    at = base[:, :, None] + torch.arange(4, device=X.device)
    w = 1.0 + fast_cos(math.pi / 2 * (at - X[:, :, None]))
    index = at[:, 1, None, :] * nx + at[:, 0, :, None]
    return index.long().reshape(len(X), 16), (w[:, 0, :, None] * w[:, 1, None, :] / 16.0).reshape(len(X), 16)


def plain_step(f, g, force, source, tau, outlet_nodes):
    """One lattice step: f[9][ny][nx], g[S][5][ny][nx], force[2][ny][nx],
    source[S][ny][nx], tau[1 + S]; returns f, g and the velocity."""
    f = torch.stack([torch.roll(f[q], (CY[q], CX[q]), (0, 1)) for q in range(9)])
    cx, cy, w = (torch.tensor(v, dtype=f.dtype, device=f.device)[:, None, None] for v in (CX, CY, WEIGHT))
    rho = f.sum(0)
    ux, uy = (cx * f).sum(0) / rho, (cy * f).sum(0) / rho
    cu = cx * ux + cy * uy
    equilibrium = w * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy))
    f = f + (equilibrium - f) / tau[0] + 3 * w * rho * (cx * force[0] + cy * force[1])
    u = torch.stack([(cx * f).sum(0) / rho, (cy * f).sum(0) / rho])
    scale = torch.ones_like(rho)
    for place in outlet_nodes:  # the mass outlet: x = 0, then y = 0
        scale = torch.where(place, scale / (f * scale).sum(0), scale)
    out = []
    cu = cx[:5] * u[0] + cy[:5] * u[1]
    w5 = torch.tensor([1 / 3] + [1 / 6] * 4, dtype=f.dtype, device=f.device)[:, None, None]
    for k in range(len(g)):
        gk = torch.stack([torch.roll(g[k][q], (CY[q], CX[q]), (0, 1)) for q in range(5)])
        c = gk.sum(0)
        gk = gk + (w5 * c * (1 + 3 * cu) - gk) / tau[1 + k] + w5 * (source[k] - DECAY * c)
        out.append(gk * scale)
    return f * scale, out, u


def exact(case, seed):
    """Frozen and differentiated runs in plain torch.  A full run's outputs
    depend on every remeshing and domain decision on the way: no plain value."""
    if case["kind"] not in ("frozen", "adjoint", "moving"):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    cells = tissue(case, seed)
    table = torch.from_numpy(source_table(case, len(cells), seed)).to(dev)
    nx, ny, S, T = case["nx"], case["ny"], case["species"], case["steps"]
    L = nx * ny
    dom = domain_ids(case, cells).to(dev)
    f, g, force = lattice_state(case, seed)
    f = torch.from_numpy(f[:, NATURAL9].T.reshape(9, ny, nx)).to(dev)
    g = [torch.from_numpy(g[k][:, NATURAL5].T.reshape(5, ny, nx)).to(dev) for k in range(S)]
    column, row = torch.zeros((2, ny, nx), dtype=torch.bool, device=dev)
    column[:, 0] = True
    row[0, :] = True
    if case["kind"] == "frozen":
        tau = torch.tensor([TAU_FLUID] + list(TAU_SPECIES[:S]), dtype=torch.float64, device=dev)
        field = torch.from_numpy(force.T.reshape(2, ny, nx)).to(dev)
        for _ in range(T):
            f, g, u = plain_step(f, g, field, table[:, dom], tau, (column, row))
        return {"f": f[list(NATURAL9)].reshape(9, L).T.contiguous(),
                "g": torch.stack([gk[list(NATURAL5)].reshape(5, L).T for gk in g]),
                "vel": u.reshape(2, L).T.contiguous(), "force": torch.from_numpy(force), "dom": None, "ctype": None}

    moving = case["kind"] == "moving"
    p = gradient_inputs(case, cells, table.cpu().numpy(), seed)
    nodes = torch.from_numpy(np.concatenate([v for _, v in cells])).to(dev)
    leaf = {"force": p["force"], "tau": p["tau"], "rates": p["rates"]}
    leaf = {k: torch.from_numpy(v).to(dev).requires_grad_() for k, v in leaf.items()}
    X = nodes.clone().requires_grad_(moving)

    def field_of(X):
        index, weight = stencil(X, nx)
        add = weight[:, None, :] * leaf["force"][:, :, None]
        zero = torch.zeros(L, dtype=torch.float64, device=dev)
        field = [zero.index_add(0, index.ravel(), add[:, i].reshape(-1)) for i in range(2)]
        return torch.stack(field).reshape(2, ny, nx)

    def segment(n, f, X, field, source, *g):
        g = list(g)
        for _ in range(n):
            if moving:
                field = field_of(X)
            f, g, u = plain_step(f, g, field, source, leaf["tau"], (column, row))
            if moving:
                index, weight = stencil(X, nx)
                X = X + (u.reshape(2, L)[:, index] * weight).sum(2).T
        return (f, X, *g)

    from torch.utils.checkpoint import checkpoint
    field, source = field_of(X), leaf["rates"][:, dom]
    at, done = X, 0
    while done < T:
        n = min(25, T - done)
        f, at, *g = checkpoint(segment, n, f, at, field, source, *g, use_reentrant=False)
        done += n
    c = torch.stack([gk.sum(0).reshape(L) for gk in g])
    loss = ((c - torch.from_numpy(p["c_target"]).to(dev)) ** 2).sum()
    out = {"c": c}
    if moving:
        out["x"] = at
        loss = loss + ((at - torch.from_numpy(p["x_target"]).to(dev)) ** 2).sum()
    loss.backward()
    out.update({"d_" + k: v.grad for k, v in leaf.items()})
    if moving:
        out["d_x"] = X.grad
    return {k: v.detach() for k, v in out.items()}
