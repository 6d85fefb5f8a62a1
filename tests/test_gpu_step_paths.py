"""The step kernel's and the walk's variants against one another and the oracle.

* Walks over lists of any length, those around the 32 entries one pass of plane
  tests covers among them, with slivers, grazing rays, rays in a triangle's
  plane and rays that start outside the root cell: distance bits and triangle
  equal to the oracle's walk, which tests every listed triangle.
* A run's records do not depend on which step kernel its size selects (few
  primaries or many), on the empty leaves a fine mesh's walks pass along, or on
  which lane flies a secondary.
All comparisons are exact, but for sums of doubles added in another order.
"""
import numpy as np
import pytest

import nebula_b200 as nb

pytestmark = pytest.mark.gpu


def _oracle_geometry(g):
    from oracle import oracle as O
    od, tr = g.export()
    inf = g.info()
    t11 = np.concatenate([np.stack([tr["material_in"], tr["material_out"]], 1).astype(np.float32),
                          tr["r0"], tr["e1"], tr["e2"]], 1)
    return O.Geometry(od, t11, inf["center"], inf["halfsize"], inf["max_extent"]), tr


def _triangles(n, rng):
    """Triangles of mixed size and shape in a 100 nm cube: ordinary ones,
    slivers, coplanar pairs and axis-aligned ones."""
    a = rng.uniform(-50, 50, (n, 3))
    e1 = rng.standard_normal((n, 3)) * rng.choice([0.3, 5.0, 40.0], (n, 1))
    e2 = rng.standard_normal((n, 3)) * rng.choice([0.3, 5.0, 40.0], (n, 1))
    sliver = rng.random(n) < 0.2
    e2[sliver] = e1[sliver] * rng.uniform(0.5, 1.5, (sliver.sum(), 1)) + rng.standard_normal((sliver.sum(), 3)) * 1e-3
    flat = rng.random(n) < 0.2
    e1[flat, 2] = e2[flat, 2] = 0.0
    a[flat, 2] = np.round(a[flat, 2] / 25) * 25
    mats = rng.choice([0, 1, -123], (n, 2))
    return np.hstack([mats, a, a + e1, a + e2])


def _rays(tr, rng, n, half):
    """Rays of every kind through triangles in a cube of that half size."""
    pos = rng.uniform(-1.2 * half, 1.2 * half, (n, 3))
    d = rng.standard_normal((n, 3))
    # a third of the rays start near a triangle's plane and run almost along it
    k = rng.integers(0, len(tr), n)
    e1, e2, r0 = (tr[f][k].astype(np.float64) for f in ("e1", "e2", "r0"))
    nrm = np.cross(e1, e2)
    nrm /= np.maximum(np.linalg.norm(nrm, axis=1, keepdims=True), 1e-30)
    graze = np.arange(n) % 3 == 0
    w = rng.standard_normal((n, 2))
    along = w[:, :1] * e1 + w[:, 1:] * e2 + nrm * rng.choice([0, 1e-7, 1e-4, 1e-2], (n, 1))
    start = r0 + rng.uniform(-1, 2, (n, 1)) * e1 + rng.uniform(-1, 2, (n, 1)) * e2 + nrm * rng.choice([0, 1e-6, 1e-3], (n, 1))
    d[graze], pos[graze] = along[graze], start[graze]
    d[np.arange(n) % 7 == 1, 0] = 0.0
    outside = np.arange(n) % 11 == 5
    pos[outside] *= 30.0
    d[outside] = -pos[outside] + rng.standard_normal((outside.sum(), 3))
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-30)
    dist = np.where(rng.random(n) < 0.5, rng.exponential(5.0, n), 1e4)
    ignore_tri = np.where(rng.random(n) < 0.2, k, -1).astype(np.int32)
    ignore_mat = rng.choice([0, 1, -123], n).astype(np.int32)
    return pos.astype(np.float32), d.astype(np.float32), dist.astype(np.float32), ignore_tri, ignore_mat


def _equal_to_oracle(g, og, rays):
    gd, gt = g.ray_query(*rays)
    cd, ct = og.propagate(*rays)
    assert np.array_equal(gt, ct), int((gt != ct).sum())
    assert np.array_equal(gd.view(np.uint32), cd.view(np.uint32))
    return gt


@pytest.mark.parametrize("n_tri", [1, 31, 32, 33, 64, 65, 300])
def test_walk_equals_oracle_for_any_list_length(n_tri):
    rng = np.random.default_rng(n_tri)
    g = nb.Geometry.from_triangles(_triangles(n_tri, rng), max_depth=2, split_count=400)
    og, tr = _oracle_geometry(g)
    gt = _equal_to_oracle(g, og, _rays(tr, rng, 200_000, 50.0))
    assert n_tri < 31 or (gt >= 0).any()


def _leaf_lists(octree):
    """The triangle lists of an octree's leaves (child index < 0: minus the
    start of a list, which a negative entry ends)."""
    lists, nodes = [], [0]
    while nodes:
        at = nodes.pop()
        for child in octree[at:at + 8]:
            if child >= 0:
                nodes.append(int(child))
                continue
            end = start = -int(child)
            while octree[end] >= 0:
                end += 1
            lists.append(octree[start:end])
    return lists


@pytest.mark.parametrize("n_list", [1, 31, 32, 33, 63, 64, 65, 96, 97, 123, 124, 125])
def test_walk_equals_oracle_around_the_passes_of_a_list(n_list):
    """All triangles but four in one octant of the root: one leaf with a list of
    exactly this length.  (With the four that make the root cell, the last three
    lengths stand around a block of the kernel that makes the planes.)"""
    rng = np.random.default_rng(1000 + n_list)
    t = _triangles(n_list, rng)
    t[:, 2:] = np.clip(25.0 + 0.4 * t[:, 2:], 3.0, 47.0)
    corners = [(-50, -50, -50), (50, -40, -50), (-40, 50, -50), (-50, -40, 50)]
    box = [[0, 1, x, y, z, x * 0.99, y, z, x, y * 0.99, z] for x, y, z in corners]
    g = nb.Geometry.from_triangles(np.vstack([t, box]), max_depth=2, split_count=400)
    og, tr = _oracle_geometry(g)
    assert len(tr) == n_list + 4
    inside = tr["r0"].min(1) > 0
    leaf = [v for v in _leaf_lists(g.export()[0]) if np.array_equal(np.sort(v), np.flatnonzero(inside))]
    assert len(leaf) == 1 and len(leaf[0]) == n_list
    n = 100_000
    pos, d, dist, ignore_tri, ignore_mat = _rays(tr, rng, n, 50.0)
    # a fifth of the rays start inside the leaf and aim at one of its triangles
    aim = np.arange(n) % 5 == 2
    at = tr[rng.choice(leaf[0], n)]
    u = rng.dirichlet([1.0, 1.0, 1.0], n)
    target = at["r0"] + u[:, :1] * at["e1"] + u[:, 1:2] * at["e2"]
    pos[aim] = rng.uniform(3.0, 47.0, (n, 3))[aim]
    towards = (target - pos).astype(np.float64)
    d[aim] = (towards / np.maximum(np.linalg.norm(towards, axis=1, keepdims=True), 1e-30))[aim]
    dist[aim] = 1e4
    gt = _equal_to_oracle(g, og, (pos, d, dist, ignore_tri, ignore_mat))
    for first in range(0, n_list, 32):
        assert np.isin(gt, leaf[0][first:first + 32]).any(), first


def _sorted(rec):
    return np.sort(np.ascontiguousarray(rec).view(np.dtype((np.void, 36))).ravel())


def _records(g, mats, pri, **kw):
    sim = nb.Simulation(g, mats, seed=77, **kw)
    sim.push(pri)
    sim.run()
    rec, c = sim.flush_detected(), sim.counters()
    sim.close()
    assert c["primaries_started"] + c["spawned"] == c["detected"] + c["terminated"]
    return rec, c


@pytest.mark.parametrize("n", [1, 31, 33, 1000])
def test_few_and_many_primaries_give_the_same_records(inputs, n):
    from nebula_b200.synth import primaries
    g = nb.Geometry.from_tri_file(inputs["slab.tri"])
    m = nb.Material.load(inputs["si.nmat"])
    total = (1 << 19) + 1
    pri = primaries.point_beam(total, energy=150.0)
    pri["px"] = np.arange(total)
    few, _ = _records(g, [m], pri[:n], capacity=1 << 16)
    many, _ = _records(g, [m], pri, capacity=1 << 18)
    assert np.array_equal(_sorted(few), _sorted(many[many["px"] < n]))


@pytest.mark.parametrize("mesh, options", [
    ("slab", {}), ("fine", {}),
    ("slab", {"deposit": True}), ("fine", {"deposit": True}),
    ("slab", {"kieft": True}), ("fine", {"kieft": True}),
    ("fine", {"physics": {"interface_absorption": 1}}),
    ("slab", {"adjoint": True}), ("fine", {"adjoint": True}),
    ("slab", {"adjoint": True, "physics": {"interface_absorption": 1}}),
    ("fine", {"adjoint": True, "deposit": True}),
], ids=lambda v: v if isinstance(v, str) else "-".join(v) or "plain")
def test_a_large_run_is_its_two_halves(inputs, mesh, options):
    """2^18 + 2048 primaries take the step kernels for many electrons, the two
    halves those for few (the adjoint on a fine mesh, or with deposits or
    another physics selection, has one for both): the same records, images,
    spectrum and event counts, and the same deposits and gradients but for the
    order of their double-precision sums."""
    from nebula_b200.synth import primaries
    suffix = "_kieft.nmat" if options.get("kieft") else ".nmat"
    mats = [nb.Material.load(inputs[k + suffix]) for k in ("si", "pmma")]
    g = _rough_lines(88.0, 0.5) if mesh == "fine" else nb.Geometry.from_tri_file(inputs["slab.tri"])
    assert (g.info()["n_octree"] >= 1 << 19) == (mesh == "fine")
    nx, ny, per = 128, 129, 16
    pri = primaries.raster_scan(nx, ny, per, 0.5, 100.0, 40.0 if mesh == "fine" else 5.0, spot_sigma=1.0, seed=9, pixel_streams=False)
    half = len(pri) // 2
    assert half <= 1 << 18 < len(pri)
    kw = {"capacity": 1 << 17, "tally": (nx, ny), "physics": options.get("physics")}
    if options.get("kieft"):
        kw["physics"] = {"inelastic_model": 1}
    if options.get("deposit"):
        kw["deposit_grid"] = ((-50.0, -50.0, -20.0), (2.0, 2.0, 2.0), (50, 50, 25))
    kw["adjoint"] = bool(options.get("adjoint"))

    def run(part, first):
        sim = nb.Simulation(g, mats, seed=77, **kw)
        sim.set_primary_offset(first)
        sim.push(part)
        sim.run()
        c = sim.counters()
        se, bse, hist = sim.tallies()
        counts = [c[k] for k in ("flights", "boundary", "elastic", "inelastic", "spawned", "detected", "terminated")]
        sums = [sim.deposit_grid()] if options.get("deposit") else []
        if kw["adjoint"]:
            sums += list(sim.gradients())
        rec = sim.flush_detected()
        sim.close()
        return rec, [se.astype(np.int64), bse.astype(np.int64), hist.astype(np.int64), np.array(counts)], sums

    whole, parts = run(pri, 0), (run(pri[:half], 0), run(pri[half:], half))
    assert len(whole[0]) > 1000
    assert np.array_equal(_sorted(whole[0]), _sorted(np.concatenate([p[0] for p in parts])))
    for w, a, b in zip(whole[1], parts[0][1], parts[1][1]):
        assert np.array_equal(w, a + b)
    assert all(np.abs(w).max() > 0 for w in whole[2][:1])
    # sums of at most 10^6 doubles in any order: 10^6 * 2^-53 of the terms' sizes
    for w, a, b in zip(whole[2], parts[0][2], parts[1][2]):
        assert np.allclose(w, a + b, rtol=1e-9, atol=1e-9 * np.abs(w).max())
    if kw["adjoint"]:
        kw["adjoint"] = False
        assert np.array_equal(_sorted(whole[0]), _sorted(run(pri, 0)[0]))


def _rough_lines(length=100.0, spacing=0.25):
    from nebula_b200.synth import geometry
    rows = geometry.rough_grating(n_lines=4, line_length=length, vertex_spacing=spacing)
    return nb.Geometry.from_triangles(rows, max_depth=12, split_count=16)


def _batch_records(geometries, mats, jobs, **kw):
    batch = nb.Batch(geometries, mats, record_capacity=1 << 20, **{"capacity": 1 << 16, **kw})
    batch.set_jobs(jobs)
    batch.run()
    rec, job = batch.records()
    c = batch.counters()
    batch.close()
    return rec, job, c


def test_fine_mesh_equals_batch_and_other_budgets(inputs):
    """Walks on a fine mesh pass empty leaves along, in a plain run and in a
    batch; with other budgets they pass others."""
    from nebula_b200.synth import primaries
    mats = [nb.Material.load(inputs["si.nmat"]), nb.Material.load(inputs["pmma.nmat"])]
    g = _rough_lines()
    assert g.info()["n_octree"] >= 1 << 20
    pri = primaries.raster_scan(16, 16, 20, 0.5, 300.0, 40.0, spot_sigma=1.0, seed=3)
    one, c1 = _records(g, mats, pri)
    long, c2 = _records(g, mats, pri, walk_cells=1 << 10)
    rec, _, _ = _batch_records([g], mats, [(0, 77, pri)])
    assert c1["walk_resumes"] > 0 and c1["flights"] == c2["flights"]
    assert len(one) > 0
    assert np.array_equal(_sorted(one), _sorted(long))
    assert np.array_equal(_sorted(one), _sorted(rec))


@pytest.mark.parametrize("physics", [None, {"interface_absorption": 1}])
@pytest.mark.parametrize("block_size", [128, 512])
@pytest.mark.parametrize("coarse, fine_kernel", [(0, True), (31 * 512, True), (31 * 512 + 1, False)])
def test_batch_kernel_for_fine_meshes(inputs, physics, block_size, coarse, fine_kernel):
    """The batched kernel for fine meshes runs from 1/32 of the primaries on.
    Either gives the plain run's records; with it the walks on the mesh, which
    end last here, take as many iterations as the plain run's, without it half
    as many again (no empty leaf is passed)."""
    from nebula_b200.synth import primaries
    mats = [nb.Material.load(inputs["si.nmat"]), nb.Material.load(inputs["pmma.nmat"])]
    g = _rough_lines()
    pri = primaries.raster_scan(16, 16, 2, 0.5, 300.0, 40.0, spot_sigma=1.0, seed=3)
    plain, c = _records(g, mats, pri, physics=physics, iterations_per_graph=6)
    jobs = [(0, 77, pri)]
    if coarse:
        jobs.append((1, 77, primaries.point_beam(coarse, energy=100.0)))
    rec, job, b = _batch_records([g, nb.Geometry.from_tri_file(inputs["slab.tri"])], mats, jobs, physics=physics,
                                 block_size=block_size)
    assert len(plain) > 0
    assert np.array_equal(_sorted(plain), _sorted(rec[job == 0]))
    assert (b["iterations"] < 1.2 * c["iterations"]) == fine_kernel


@pytest.mark.parametrize("length, fine", [(85.0, False), (88.0, True)])
def test_meshes_are_fine_from_half_a_million_words(inputs, length, fine):
    """A plain run passes empty leaves on octrees of 2^19 words and more: it
    takes fewer iterations than a batch whose coarse jobs keep the coarse
    kernel (below, as many: up to the graph's 6 more, or 1 less, for other
    lanes take the secondaries)."""
    from nebula_b200.synth import primaries
    mats = [nb.Material.load(inputs["si.nmat"]), nb.Material.load(inputs["pmma.nmat"])]
    g = _rough_lines(length, 0.5)
    assert (g.info()["n_octree"] >= 1 << 19) == fine
    pri = primaries.raster_scan(16, 16, 2, 0.5, 300.0, 40.0, spot_sigma=1.0, seed=3)
    plain, c = _records(g, mats, pri, iterations_per_graph=6)
    rec, job, b = _batch_records([g, nb.Geometry.from_tri_file(inputs["slab.tri"])], mats,
                                 [(0, 77, pri), (1, 77, primaries.point_beam(32 * len(pri), energy=100.0))])
    assert len(plain) > 0
    assert np.array_equal(_sorted(plain), _sorted(rec[job == 0]))
    assert (c["iterations"] < b["iterations"] - 1) == fine


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65])
def test_secondaries_flown_in_ended_lanes(inputs, n):
    """Plain and batched runs pack their warps differently; so do pools of
    different size and the adjoint's replay."""
    from nebula_b200.synth import primaries
    g = nb.Geometry.from_tri_file(inputs["grating.tri"])
    mats = [nb.Material.load(inputs["si.nmat"]), nb.Material.load(inputs["pmma.nmat"])]
    pri = primaries.raster_scan(n, 1, 1, 0.5, 500.0, 40.0, seed=4)
    ref, c = _records(g, mats, pri)
    for kw in ({"capacity": 32}, {"adjoint": True, "tally": (n, 1)}, {"walk_cells": 7}, {"block_size": 32}):
        rec, c2 = _records(g, mats, pri, **kw)
        assert np.array_equal(_sorted(ref), _sorted(rec)), kw
        assert all(c[k] == c2[k] for k in ("flights", "boundary", "elastic", "inelastic", "spawned", "terminated")), kw
    batch = nb.Batch([g], mats, capacity=1 << 10, record_capacity=1 << 16)
    batch.set_jobs([(0, 77, pri)])
    batch.run()
    rec, _ = batch.records()
    batch.close()
    assert np.array_equal(_sorted(ref), _sorted(rec))


def test_reused_simulation_equals_fresh_ones(inputs):
    """Runs of one simulation with the same and with other counts, seeds and
    offsets (its launch graph is kept while they are the same)."""
    from nebula_b200.synth import primaries
    g = nb.Geometry.from_tri_file(inputs["slab.tri"])
    m = nb.Material.load(inputs["si.nmat"])
    sim = nb.Simulation(g, [m], capacity=1 << 12, seed=77)
    for seed, first, n, energy in ((77, 0, 200, 500.0), (77, 0, 200, 300.0), (78, 0, 200, 300.0), (78, 5, 200, 300.0),
                                   (78, 5, 201, 300.0), (78, 5, 5000, 300.0), (77, 0, 200, 500.0)):
        pri = primaries.point_beam(n, energy=energy)
        sim.reset()
        sim.set_seed(seed)
        sim.set_primary_offset(first)
        sim.push(pri)
        sim.run()
        fresh = nb.Simulation(g, [m], capacity=1 << 12, seed=seed)
        fresh.set_primary_offset(first)
        fresh.push(pri)
        fresh.run()
        assert np.array_equal(_sorted(sim.flush_detected()), _sorted(fresh.flush_detected()))
        fresh.close()
    sim.close()


@pytest.mark.parametrize("n", [699_050, 699_051, 2_330_168, 2_330_169, 2_500_001])
def test_large_pageable_push_equals_pinned(inputs, n):
    """Pushes of 80 MiB and more (2 330 169 records) go through staging threads,
    those of 24 MiB and more (699 051) from a simulation's third run on; from
    page-locked memory, or in small parts, they are copied directly."""
    import torch
    from nebula_b200.synth import primaries
    g = nb.Geometry.from_tri_file(inputs["slab.tri"])
    m = nb.Material.load(inputs["si.nmat"])
    pri = primaries.point_beam(n, energy=20.0)
    pri["px"] = np.arange(n)
    pri["pos"][:, 0] = np.random.default_rng(n).uniform(-300, 300, n)
    pinned = torch.empty(n * 36, dtype=torch.uint8, pin_memory=True).numpy().view(nb.PRI_DTYPE)
    pinned[:] = pri
    direct, _ = _records(g, [m], pinned, capacity=1 << 16)
    sim = nb.Simulation(g, [m], capacity=1 << 16, seed=77)
    for parts in (1, 1, 1, 9):
        for part in np.array_split(pri, parts):
            sim.push(part)
        sim.run()
        rec = sim.flush_detected()
        sim.reset()
        assert len(rec) > 0
        assert np.array_equal(_sorted(rec), _sorted(direct)), parts
    sim.close()


def test_first_pageable_push_waits_for_no_buffers(inputs):
    """A first push of 24 MB takes about as long as the next one (it makes the
    primaries' device buffer, 1.3 times).  Making the staging buffers for it
    would take three times as long."""
    import time
    g = nb.Geometry.from_tri_file(inputs["slab.tri"])
    m = nb.Material.load(inputs["si.nmat"])
    pri = np.zeros(24_000_000 // 36, nb.PRI_DTYPE)
    pri["E"] = 1.0
    times = []
    for _ in range(9):
        sim = nb.Simulation(g, [m], capacity=1 << 16)
        for _ in range(2):
            t = time.perf_counter()
            sim.push(pri)
            times.append(time.perf_counter() - t)
            sim.reset()
        sim.close()
    assert min(times[::2]) < 2 * min(times[1::2])


def test_queues_hold_the_population_bound(inputs):
    """Device memory of a simulation: queues for 6 times its capacity, the ring
    for 16 times (52 bytes an electron, 32 more for a continued walk), records
    for 4 times."""
    import torch
    g = nb.Geometry.from_tri_file(inputs["slab.tri"])
    m = nb.Material.load(inputs["si.nmat"])
    nb.Simulation(g, [m], capacity=1 << 10).close()      # loads the kernels
    free = torch.cuda.mem_get_info()[0]
    sim = nb.Simulation(g, [m], capacity=1 << 20)
    used = free - torch.cuda.mem_get_info()[0]
    sim.close()
    queues = 2 * (5 * 52 + 32)
    need = (1 << 20) * (6 * queues + 16 * 52 + 4 * 36)
    assert need <= used < need + (1 << 20) * queues
