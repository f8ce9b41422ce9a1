"""The cell-per-lane first pass (builds of at least kLaneMinCells cells, pg_lane.cu) against the oracle, at
the sizes and inputs where its rules end: the last warp's idle lanes, coincident
points, cells of more than 42 vertices, reaches that hold too many points, chunks,
ranges, and the survey that declines it (surfaces; few cells of varying density)."""

import ctypes

import numpy as np
import pytest
import torch

from _helpers import diff_cells

pytestmark = pytest.mark.gpu

MIN = 32768  # kLaneMinCells


@pytest.fixture(scope="module")
def dev():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch.device("cuda:0")


def _cloud(kind, n, seed=5):
    from paragram_b200 import workloads as W

    rng = np.random.default_rng(seed)
    w = None
    if kind == "uniform":
        p = W.uniform(n, seed)
    elif kind == "power":
        p, w = W.power_uniform(n, seed)
    elif kind == "heavy":  # weights that empty many cells and move others off their points
        p = W.uniform(n, seed)
        w = (rng.random(n) * 4.0 * n ** (-2.0 / 3.0)).astype(np.float32)
    elif kind == "lattice":
        m = round(n ** (1 / 3))
        p, w = W.jittered_lattice(m, seed)
    elif kind == "exact_lattice":
        m = round(n ** (1 / 3))
        g = np.arange(m, dtype=np.float32) / np.float32(64.0)
        p = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3).copy()
    elif kind == "surface":
        p = W.surface_cloud(n, np.random.Generator(np.random.PCG64(seed)))
    elif kind == "clustered":
        p = W.clustered(n, seed)
    elif kind == "dense_spots":  # a tenth of the points in 40 spots a thousandth of the spacing wide
        p = W.uniform(n, seed)
        k = n // 10
        p[:k] = p[k:k + 40][rng.integers(0, 40, k)] + (1e-5 * rng.standard_normal((k, 3))).astype(np.float32)
    elif kind == "coincident":  # every fourth point is a copy, some places hold twenty
        p = W.uniform(n, seed)
        p[::4] = p[1::4][: len(p[::4])]
        p[:200] = np.repeat(p[300:310], 20, axis=0)
    elif kind == "wheel":  # hubs with 60 points around each: cells beyond 42 vertices
        hubs = W.uniform(n // 61, seed)
        a = rng.random((len(hubs), 60)) * 2 * np.pi
        d = 0.3 * len(hubs) ** (-1.0 / 3.0)
        ring = hubs[:, None, :] + d * np.stack([np.cos(a), np.sin(a), 0.05 * rng.standard_normal(a.shape)], -1)
        p = np.concatenate([hubs, ring.reshape(-1, 3)]).astype(np.float32)
    return np.ascontiguousarray(p), w


def _gpu(p, w, dev, **kw):
    import paragram_b200.cuda as pc

    t = torch.from_numpy(p).to(dev)
    tw = None if w is None else torch.from_numpy(w).to(dev)
    (a, o, s), st = pc.build_with_stats(t, tw, **kw)
    return (a.cpu().numpy(), o.cpu().numpy(), s.cpu().numpy()), st


@pytest.mark.parametrize("kind,n", [("uniform", MIN - 1), ("uniform", MIN), ("uniform", MIN + 1), ("power", MIN + 31),
                                    ("heavy", 40_000), ("lattice", 35_937), ("exact_lattice", 35_937),
                                    ("surface", 36_001), ("dense_spots", 40_000), ("coincident", 36_000),
                                    ("wheel", 36_600), ("clustered", MIN + 5), ("clustered", 60_001)])
def test_lane_pass_equals_oracle(dev, oracle, kind, n):
    p, w = _cloud(kind, n)
    got, _ = _gpu(p, w, dev)
    assert diff_cells(got, oracle.diagram(p, w)).size == 0


@pytest.mark.parametrize("kind,n,taken", [("uniform", MIN - 1, False), ("uniform", MIN, True), ("heavy", 40_000, True),
                                          ("lattice", 35_937, True), ("clustered", MIN + 5, False),
                                          ("clustered", 55_999, False), ("clustered", 56_000, True),
                                          ("clustered", 60_001, True), ("surface", 36_001, False),
                                          ("surface", 100_000, False), ("surface", 400_000, True)])
def test_lane_pass_choice(dev, kind, n, taken):
    """Which builds the pass takes, that most of their cells stay in it, and the same diagram either way
    (blocks_per_sm = 3 keeps a build from the pass)."""
    import paragram_b200.cuda as pc

    p, w = _cloud(kind, n)
    got, _ = _gpu(p, w, dev)
    prof = pc.last_profile()
    assert prof["lane_cells"] == (n if taken else 0)
    assert prof["listed_cells"] < 0.6 * n if taken else prof["listed_cells"] == 0
    ref, _ = _gpu(p, w, dev, blocks_per_sm=3)
    assert pc.last_profile()["lane_cells"] == 0
    assert all(np.array_equal(x, y) for x, y in zip(got, ref))


@pytest.mark.parametrize("kind,n", [("clustered", 70_001), ("surface", 100_000), ("surface", 300_000)])
def test_exports_do_not_depend_on_timing_chunks_or_ranges(dev, kind, n):
    """Volumes, centroids and vertices bit by bit: of a second call, of a build in chunks, and of a build of a
    range of the curve (whose ends lie inside groups of 32 cells)."""
    import paragram_b200.cuda as pc
    from paragram_b200 import _lib

    p, _ = _cloud(kind, n)
    t = torch.from_numpy(p).to(dev)
    names = ("centroids", "volumes", "vertices", "vertex_bound", "vertex_planes", "vertex_count")
    bits = lambda x: x.contiguous().view(torch.int32)  # noqa: E731
    _, a = pc.build_with_stats(t, geometry=True, vertices=24, features=True)
    for kw in ({}, {}, dict(num_chunks=5)):
        _, b = pc.build_with_stats(t, geometry=True, vertices=24, **kw)
        assert all(torch.equal(bits(a[k]), bits(b[k])) for k in names), kw
    begin, end = 1003, 1003 + max(MIN, int(0.9 * n))
    lib = _lib.load()
    size = ctypes.c_size_t(0)
    assert lib.pg_workspace_size(n, ctypes.byref(size)) == 0
    ws = torch.empty(size.value, dtype=torch.uint8, device=dev)
    status = torch.empty(n, dtype=torch.int32, device=dev)
    geom = torch.full((n, 4), -1.0, dtype=torch.float32, device=dev)
    opt = _lib.PgOptions(8, -1, 0, 0, 0)
    opt.geometry_out = geom.data_ptr()
    assert lib.pg_build_range(n, t.data_ptr(), None, ctypes.byref(opt), ws.data_ptr(), size.value, begin, end,
                              status.data_ptr(), torch.cuda.current_stream(dev).cuda_stream) == 0
    inside = torch.zeros(n, dtype=torch.bool, device=dev)
    inside[a["order"][begin:end].long()] = True
    assert torch.equal(bits(geom[inside, :3]), bits(a["centroids"][inside]))
    assert torch.equal(bits(geom[inside, 3]), bits(a["volumes"][inside]))
    assert bool((geom[~inside] == -1.0).all())


def test_declined_build_keeps_its_guesses(dev):
    """Cells left to the warp-per-cell pass are clipped by the caller's guesses there too: the true neighbours
    as guesses save it nodes (the counters of a build that the lane pass takes hold its shared searches too)."""
    import paragram_b200.cuda as pc

    p, _ = _cloud("surface", 40_000)
    (adj, off, st), cold = _gpu(p, None, dev)
    g = dict(initial_guesses=torch.from_numpy(adj).to(dev), initial_guesses_offsets=torch.from_numpy(off).to(dev))
    got, warm = _gpu(p, None, dev, **g)
    assert pc.last_profile()["lane_cells"] == 0
    assert all(np.array_equal(x, y) for x, y in zip(got, (adj, off, st)))
    assert warm["nodes"] < 0.9 * cold["nodes"]


def test_lane_pass_equals_warp_pass_and_chunks(dev):
    """blocks_per_sm = 3 is a register budget of the warp-per-cell pass; chunks split the lane pass's launches."""
    p, w = _cloud("power", 50_001)
    ref, _ = _gpu(p, w, dev, blocks_per_sm=3)
    for chunks in (1, 3, 7):
        got, st = _gpu(p, w, dev, num_chunks=chunks)
        assert all(np.array_equal(x, y) for x, y in zip(got, ref)), chunks
        assert st["clips"] > 10 * len(p)


@pytest.mark.parametrize("kind", ["uniform", "heavy", "surface"])
def test_lane_pass_exports(dev, kind):
    """Volumes, centroids and vertices of the lane pass against the warp-per-cell pass: the same vertices
    (each within both passes' bounds) and integrals of them. Both integrate FP32 vertices within 2^-19 of
    their length; a volume then differs by at most about 3 * 2^-18 times (length / size of the cell)."""
    p, w = _cloud(kind, 40_000)
    g0, a = _gpu(p, w, dev, geometry=True, vertices=64, blocks_per_sm=3)
    g1, b = _gpu(p, w, dev, geometry=True, vertices=64)
    assert all(np.array_equal(x, y) for x, y in zip(g0, g1))
    assert torch.equal(a["vertex_count"], b["vertex_count"])
    va, vb = a["volumes"].double(), b["volumes"].double()
    full = va > 0
    assert torch.equal(full, vb > 0)
    rel = ((va - vb).abs() / va)[full]
    assert float(rel.median()) < 1e-5 and float((va - vb).norm() / va.norm()) < 2e-5
    ca, cb = a["centroids"].double()[full], b["centroids"].double()[full]
    assert float((ca - cb).norm() / ca.norm()) < 2e-5
    assert torch.equal(torch.isnan(a["centroids"]), torch.isnan(b["centroids"]))
    # vertex by vertex: matched by their three planes
    k = min(64, int(a["vertex_count"].max()))
    pa, pb = a["vertex_planes"][:, :k].sort(2).values, b["vertex_planes"][:, :k].sort(2).values
    n = len(p)
    used = (torch.arange(k, device=dev)[None] < a["vertex_count"][:, None]) & (a["vertex_count"][:, None] <= 64)
    key = lambda q: ((q[..., 0] + 8) * (n + 16) + q[..., 1] + 8) * (n + 16) + q[..., 2] + 8  # noqa: E731
    big = torch.iinfo(torch.int64).max
    ka, ia = torch.where(used, key(pa.long()), big).sort(1)
    kb, ib = torch.where(used, key(pb.long()), big).sort(1)
    assert torch.equal(ka, kb)
    xa = torch.gather(a["vertices"][:, :k], 1, ia[..., None].expand(-1, -1, 3)).double()
    xb = torch.gather(b["vertices"][:, :k], 1, ib[..., None].expand(-1, -1, 3)).double()
    ba, bb = torch.gather(a["vertex_bound"][:, :k], 1, ia), torch.gather(b["vertex_bound"][:, :k], 1, ib)
    on = ka < big
    assert bool(((xa - xb).norm(dim=2)[on] <= (ba + bb)[on].double() * (1 + 1e-6)).all())


def test_lane_pass_keeps_all_bits_of_the_bounds(dev):
    """The vertex bounds of both passes come from the same formula over the same three planes (in another order:
    roundings either way): their ratio's median is 1. A bound rounded up to 8 or 9 bits would raise it by a
    third of 2^-8 to 2^-7; the line is drawn at 2^-10."""
    p, _ = _cloud("uniform", 40_000)
    _, a = _gpu(p, None, dev, vertices=42, blocks_per_sm=3)
    _, b = _gpu(p, None, dev, vertices=42)
    n, k = len(p), 42
    bounds = []
    for r in (a, b):
        count = r["vertex_count"]
        used = (torch.arange(k, device=dev)[None] < count[:, None]) & (count[:, None] <= k)
        q = r["vertex_planes"].long().sort(2).values
        key = ((q[..., 0] + 8) * (n + 16) + q[..., 1] + 8) * (n + 16) + q[..., 2] + 8
        key, at = torch.where(used, key, torch.iinfo(torch.int64).max).sort(1)
        bounds.append((key, torch.gather(r["vertex_bound"], 1, at).double(), used.sum()))
    (ka, ba, na), (kb, bb, nb) = bounds
    assert torch.equal(ka, kb) and int(na) == int(nb) > 20 * n
    ratio = (bb / ba)[ka < torch.iinfo(torch.int64).max]
    assert abs(float(ratio.median()) - 1.0) < 2.0 ** -10


def test_lane_pass_guesses_and_radius(dev):
    """Initial guesses (true neighbours, with repeats, the point itself and ids out of range; too many; none)
    and search radii (exact, far too small, none) leave the diagram as it is."""
    p, w = _cloud("power", 40_000)
    n = len(p)
    (adj, off, st), cold = _gpu(p, w, dev, diagnostics=True)
    rng = np.random.default_rng(3)
    rows = [adj[off[u]:off[u + 1]] for u in range(n)]
    for u in range(0, n, 7):
        rows[u] = np.concatenate([rows[u][::2], rows[u][:3], [u, -5, n + 9]]).astype(np.int32)
    for u in range(3, n, 50):
        rows[u] = rng.integers(0, n, 60).astype(np.int32)
    for u in range(5, n, 50):
        rows[u] = rows[u][:0]
    go = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    g = torch.from_numpy(np.concatenate(rows).astype(np.int32)).to(dev)
    guesses = dict(initial_guesses=g, initial_guesses_offsets=torch.from_numpy(go).to(dev))
    radius = cold["radius"]
    for kw in (guesses, dict(radius_hint=radius * 1.0001), dict(radius_hint=radius * 0.3),
               dict(radius_hint=radius * 1.0001, **guesses)):
        got, stats = _gpu(p, w, dev, **kw)
        assert all(np.array_equal(x, y) for x, y in zip(got, (adj, off, st))), list(kw)
        if "radius_hint" in kw:
            hits, misses = stats["hint_hits"], stats["hint_misses"]
            exact = kw["radius_hint"][0] > radius[0]
            assert hits + misses > 0.8 * n and (misses == 0 if exact else misses > 0.9 * (hits + misses))
