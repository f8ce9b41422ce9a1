"""Measured cases: what users have this framework do, through its public entry points.

A case is a dict of plain values: an entry point (``call``), a point distribution
(``points``, generators of ``paragram_b200.workloads``) and a size. ``prepare``
makes what a program holds before the call (points, weights, a previous diagram,
a trained model, buffers for results whose length the points decide), ``run`` is
one call, and its result is returned whole.
"""

from __future__ import annotations

import numpy as np
import torch

import paragram_b200 as pg
from paragram_b200 import learned, workloads

DEVICE = "cuda"


def listed():
    return [
        # A handful of points, e.g. one molecule or a small mesh seeded interactively: latency and launches.
        {"name": "voronoi_1k", "call": "voronoi", "points": "uniform", "n": 1000},
        # The ordinary unweighted diagram (the first benchmark configuration).
        {"name": "voronoi_uniform_100k", "call": "voronoi", "points": "uniform", "n": 100_000},
        # The power diagram configuration: uniform points, weights that empty a few cells.
        {"name": "power_uniform_1m", "call": "power", "points": "power_uniform", "n": 1_000_000},
        # The headline configuration: strongly varying density.
        {"name": "voronoi_clustered_5m", "call": "voronoi", "points": "clustered", "n": 5_000_000},
        # A scanned surface of ragged size: long thin cells, many of them bounded by the box.
        {"name": "voronoi_surface_29765", "call": "voronoi", "points": "surface", "n": 29_765},
        # Near-degenerate input (almost cospherical lattice neighbours), weighted.
        {"name": "power_lattice_128", "call": "power", "points": "lattice", "n": 128},
        # Many uneven clouds in one build, the same batch shape every time (captured once, replayed).
        {"name": "batch_surface_24", "call": "batch", "points": "surface", "n": 24, "smallest": 1000,
         "largest": 60_000},
        # A simulation step: points moved a little, rebuilt with the previous diagram as guesses.
        {"name": "moving_uniform_500k", "call": "moving", "points": "uniform", "n": 500_000},
        # Lloyd relaxation / semi-discrete transport: volumes and centroids with the diagram.
        {"name": "geometry_uniform_300k", "call": "geometry", "points": "uniform", "n": 300_000},
        # Finite-volume coefficients: the area of every facet.
        {"name": "faces_uniform_100k", "call": "faces", "points": "uniform", "n": 100_000},
        # The nearest-neighbour query on its own.
        {"name": "knn_clustered_1m", "call": "knn", "points": "clustered", "n": 1_000_000, "k": 8},
        # The diagram with the trained search radius.
        {"name": "learned_clustered_1m", "call": "learned", "points": "clustered", "n": 1_000_000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(["voronoi", "voronoi", "voronoi", "power", "power", "batch", "moving", "geometry", "faces", "knn",
                       "learned"])
    case = {"call": call}
    if call == "batch":
        case.update(points="surface", n=rng.randint(2, 32), smallest=_log_uniform(rng, 200, 2000),
                    largest=_log_uniform(rng, 2001, 60_000))
        return case
    if call == "power":
        case["points"] = rng.choice(["power_uniform", "power_uniform", "lattice"])
        case["n"] = rng.randint(10, 140) if case["points"] == "lattice" else _log_uniform(rng, 1000, 3_000_000)
        return case
    if call == "voronoi":
        case["points"] = rng.choice(["uniform", "clustered", "surface"])
        case["n"] = _log_uniform(rng, 1000, 100_000 if case["points"] == "surface" else 4_000_000)
        return case
    if call == "faces":
        case.update(points="uniform", n=_log_uniform(rng, 1000, 200_000))
        return case
    case["points"] = rng.choice(["uniform", "clustered"])
    case["n"] = _log_uniform(rng, 1000, {"moving": 1_000_000, "geometry": 1_000_000, "knn": 3_000_000,
                                         "learned": 2_000_000}[call])
    if call == "knn":
        case["k"] = rng.randint(1, 16)
    return case


def _sizes(case):
    """Sizes of a batch's clouds: a geometric ladder from the smallest to the largest."""
    k, lo, hi = case["n"], case["smallest"], case["largest"]
    return [int(round(lo * (hi / lo) ** (i / max(k - 1, 1)))) for i in range(k)]


def _count(case):
    if case["call"] == "batch":
        return sum(_sizes(case))
    return case["n"] ** 3 if case["points"] == "lattice" else case["n"]


def _points(case, seed):
    """Host points and weights (or None) of a case."""
    kind, n = case["points"], case["n"]
    if kind == "uniform":
        return workloads.uniform(n, seed=seed), None
    if kind == "clustered":
        return workloads.clustered(n, seed=seed), None
    if kind == "surface":
        return workloads.surface_cloud(n, np.random.Generator(np.random.PCG64(seed))), None
    if kind == "power_uniform":
        return workloads.power_uniform(n, seed=seed)
    if kind == "lattice":
        return workloads.jittered_lattice(n, seed=seed)
    raise ValueError(kind)


def _cuda(a):
    return torch.from_numpy(a).to(DEVICE)


#: Adjacency entries per point that a program sets aside: the diagrams here have 13 to 18.
_ROOM = 24


def prepare(case, seed):
    call = case["call"]
    state = {"call": call, "k": case.get("k", 8)}
    if call != "knn":
        state["adjacency"] = torch.full((_ROOM * _count(case) + 4096,), -1, dtype=torch.int32, device=DEVICE)
    if call == "faces":
        state["areas"] = torch.zeros(state["adjacency"].shape, dtype=torch.float32, device=DEVICE)
    if call == "batch":
        rng = np.random.Generator(np.random.PCG64(seed))
        sizes = _sizes(case)
        order = rng.permutation(len(sizes))
        state["clouds"] = [None] * len(sizes)
        for i in order:
            state["clouds"][int(i)] = _cuda(workloads.surface_cloud(sizes[int(i)], rng))
        return state
    pts, weights = _points(case, seed)
    state["points"] = _cuda(pts)
    if weights is not None:
        state["weights"] = _cuda(weights)
    if call == "moving":
        # the previous step's diagram; since then every point moved by about 1% of the spacing
        state["previous"] = pg.voronoi_diagram(state["points"])
        rng = np.random.Generator(np.random.PCG64(seed + 1_000_003))
        step = 0.01 * len(pts) ** (-1.0 / 3.0)
        state["points"] = _cuda((pts + step * rng.standard_normal(pts.shape)).astype(np.float32))
    if call == "learned":
        # trained on a cloud of another seed; a program trains once and keeps the model
        other, _ = _points({"points": case["points"], "n": 100_000}, seed + 2_000_003)
        data = learned.collect(_cuda(other))
        state["model"] = learned.train([data], epochs=4)
        state["model"].calibrate(data, quantile=0.98)
    return state


def _kept(state, d):
    """The diagram in the program's own buffer: its adjacency has a length that the points decide."""
    state["adjacency"][: d.adjacency.shape[0]].copy_(d.adjacency)
    return state["adjacency"], d.offsets, d.status


def run(state):
    call = state["call"]
    if call == "voronoi":
        return _kept(state, pg.voronoi_diagram(state["points"]))
    if call == "power":
        return _kept(state, pg.power_diagram(state["points"], state["weights"]))
    if call == "batch":
        ds = pg.build_batch(state["clouds"], graph=True)
        length = sum(d.adjacency.shape[0] for d in ds)
        torch.cat([d.adjacency for d in ds], out=state["adjacency"][:length])
        return state["adjacency"], torch.cat([d.offsets for d in ds]), torch.cat([d.status for d in ds])
    if call == "moving":
        prev = state["previous"]
        return _kept(state, pg.voronoi_diagram(state["points"], initial_guesses=prev.adjacency,
                                               initial_guesses_offsets=prev.offsets))
    if call == "geometry":
        d, centroids, volumes = pg.cell_geometry(state["points"])
        return _kept(state, d) + (centroids, volumes)
    if call == "faces":
        d, areas = pg.face_areas(state["points"])
        state["areas"][: areas.shape[0]].copy_(areas)
        return _kept(state, d) + (state["areas"],)
    if call == "knn":
        return pg.knn(state["points"], state["k"])
    if call == "learned":
        return _kept(state, learned.voronoi_diagram(state["points"], state["model"]))
    raise ValueError(call)


#: Mean number of facets of a cell, and the FP32 operations of clipping one cell by its own facets
#: alone: per facet its plane (20), a side test (8) of each of the cell's 2d - 4 vertices and the
#: vertices it creates (228).
_DEGREE = 15.0
_CELL_FLOPS = _DEGREE * (20 + 8 * (2 * _DEGREE - 4) + 228)


def work(case):
    n = _count(case)
    points = 12 * n + (4 * n if case["call"] == "power" else 0)
    if case["call"] == "knn":
        # k neighbours out; at least the distances to them
        return {"bytes": points + 4 * n * case["k"], "flops": 8.0 * n * case["k"]}
    diagram = 4 * n * _DEGREE + 4 * n + 4 * n
    flops = n * _CELL_FLOPS
    if case["call"] == "moving":
        points += 4 * n * _DEGREE + 4 * n
    if case["call"] == "geometry":
        diagram += 16 * n
        flops += n * (2 * _DEGREE - 4) * 3 * 40  # a signed tetrahedron per directed edge of every facet
    if case["call"] == "faces":
        diagram += 4 * n * _DEGREE
        flops += n * (2 * _DEGREE - 4) * 3 * 20
    if case["call"] == "learned":
        flops += n * 2 * (16 * 64 + 64 * 64 + 64 * 2)
    return {"bytes": points + diagram, "flops": flops}


def exact(case, seed):
    """Diagrams and neighbours are whole numbers. The volumes, centroids and areas of cells have no
    64-bit construction short of a second Voronoi builder, which takes far longer than a few seconds
    in numpy at these sizes."""
    return None
