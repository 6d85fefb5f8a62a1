"""The work a user of nebula_b200 has it do, as cases that can be timed and compared.

Every case goes through the package's public classes: a scan of primaries
pushed into a ``Simulation`` and run to its end, a ``Batch`` of jobs, a
``ScanProblem`` with its gradients, or a set of rays traced through a
``Geometry``.  The kinds:

* ``slab``      point beam on the Si slab; yields and the energy spectrum
* ``image``     raster scan of the line grating; SE / BSE images and spectrum
* ``records``   the same scan with every detected electron read back and put
                in order of energy, as a spectrum or a file writer does
* ``stream``    the same scan end to end: primaries streamed from page-locked
                memory, detected records streamed back while it runs
* ``rough``     raster scan of lines with edge roughness (a mesh of 1.2 M
                triangles, larger than the L2)
* ``dose``      energy deposited per voxel below the beam (exposure maps)
* ``kieft``     the grating with the Kieft-Bosch inelastic model
* ``adjoint``   forward run, replay and per-pixel gradients
* ``batch``     jobs of mixed geometry, energy and size in one launch
* ``rays``      nearest-triangle queries through the octree

Runs are deterministic for a seed except for the order in which records are
written and in which double-precision sums are added.
"""
import functools
import os
import tempfile

import numpy as np
import torch

import nebula_b200 as nb
from nebula_b200.synth import geometry, materials, nmat, primaries, workloads
from nebula_b200.torch_adjoint import ScanProblem

PHYSICAL = ("flights", "boundary", "elastic", "inelastic", "spawned", "detected", "terminated", "primaries_started")
DOSE_GRID = ((-50.0, -50.0, -100.0), (1.0, 1.0, 1.0), (100, 100, 100))


def listed():
    return [
        # a quick yield measurement: the driver's small job, where launches and
        # the tail of the last cascades are most of the time
        {"name": "slab_small", "kind": "slab", "n": 10_000, "energy": 1000.0},
        # few primaries with long cascades (backscatter at column voltage)
        {"name": "slab_15keV", "kind": "slab", "n": 4_001, "energy": 15_000.0},
        # a region of interest while an operator moves around: odd sizes, few
        # primaries per pixel
        {"name": "image_tile", "kind": "image", "nx": 37, "ny": 29, "per_pixel": 23, "energy": 500.0},
        # an ordinary image tile with its records
        {"name": "records_block", "kind": "records", "nx": 96, "ny": 96, "per_pixel": 100, "energy": 500.0},
        # the full line-space scan, host memory to host memory
        {"name": "stream_scan", "kind": "stream", "nx": 256, "ny": 256, "per_pixel": 100, "energy": 500.0},
        # roughness metrology: a block of the rough-line scan at low voltage
        {"name": "rough_block", "kind": "rough", "nx": 128, "ny": 128, "per_pixel": 100, "energy": 300.0},
        # a lithography dose map
        {"name": "dose_slab", "kind": "dose", "n": 50_000, "energy": 1000.0},
        # another physics selection than the default
        {"name": "kieft_image", "kind": "kieft", "nx": 64, "ny": 64, "per_pixel": 50, "energy": 500.0},
        # calibration of material parameters: yield and gradients per pixel
        {"name": "adjoint_scan", "kind": "adjoint", "nx": 64, "ny": 64, "per_pixel": 100, "energy": 500.0},
        # many small experiments in one go
        {"name": "batch_mixed", "kind": "batch", "jobs": 64, "scale": 0.1},
        # geometry checks and visibility queries from a host program
        {"name": "rays_grating", "kind": "rays", "n": 200_003},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(("slab", "image", "image", "records", "stream", "rough", "dose", "kieft", "adjoint", "batch", "rays"))
    if kind == "rays":
        return {"kind": kind, "n": log_int(1_000, 1_000_000)}
    if kind == "batch":
        return {"kind": kind, "jobs": rng.randint(3, 64), "scale": round(0.01 * 20 ** rng.random(), 4)}
    if kind in ("slab", "dose"):
        energy = float(log_int(200, 15_000 if kind == "slab" else 2_000))
        # at most about a tenth of the full scan's events
        return {"kind": kind, "n": log_int(1_000, min(200_000, int(3e8 / energy))), "energy": energy}
    energy = float(rng.randint(200, 1000))
    most = {"stream": 256, "image": 160, "records": 128, "rough": 160, "kieft": 96, "adjoint": 64}[kind]
    return {"kind": kind, "nx": log_int(16, most), "ny": log_int(16, most), "per_pixel": log_int(10, 100), "energy": energy}


@functools.lru_cache(maxsize=None)
def _material_file(name, e_max, model):
    """The scatter tables of a material as file contents (a user has the file)."""
    spec = materials.silicon(e_max) if name == "si" else materials.pmma(e_max)
    handle, path = tempfile.mkstemp(suffix=".nmat")
    os.close(handle)
    nmat.write(path, materials.build_raw_material(spec, inelastic=model))
    with open(path, "rb") as f:
        data = f.read()
    os.unlink(path)
    return data


def _material(name, e_max=10e3, model="full_penn"):
    handle, path = tempfile.mkstemp(suffix=".nmat")
    with os.fdopen(handle, "wb") as f:
        f.write(_material_file(name, e_max, model))
    try:
        return nb.Material.load(path)
    finally:
        os.unlink(path)


def _quads(mat_in, mat_out, p0, p1, p2, p3):
    """Two triangles per quad for arrays of corners."""
    n = max(np.shape(p)[0] for p in (p0, p1, p2, p3))
    head = np.broadcast_to(np.array([mat_in, mat_out], np.float64), (n, 2))
    return [np.hstack([head, p0, p1, p2]), np.hstack([head, p0, p2, p3])]


@functools.lru_cache(maxsize=None)
def _rough_mesh(n_lines=16, pitch=32.0, top_cd=16.0, run=2.1, height=30.0, size=1000.0, length=500.0, spacing=0.25,
                sigma=1.5, corr=20.0, rows=8):
    """Lines with exponentially correlated edge roughness on the slab: the
    rough-line mesh at its full density (1.2 M triangles)."""
    rng = np.random.default_rng(1234)
    h, m = size / 2, int(round(length / spacing))
    y = np.linspace(-length / 2, length / 2, m + 1)
    out, fixed = [], []
    geometry.box(fixed, (-h, -h, -size), (h, h, 0.0), 0, geometry.VACUUM, skip_top=True)
    for y0, y1 in ((-h, -length / 2), (length / 2, h)):
        fixed += [[0, geometry.VACUUM, -h, y0, 0, h, y0, 0, h, y1, 0], [0, geometry.VACUUM, -h, y0, 0, h, y1, 0, -h, y1, 0]]
    geometry.detector_plane(fixed, 50.0, h, h)
    out.append(np.asarray(fixed, np.float64))

    def at(x, z, lo):
        ys = y[:-1] if lo else y[1:]
        xs = np.broadcast_to(x, (m + 1,))[:-1] if lo else np.broadcast_to(x, (m + 1,))[1:]
        return np.stack([xs, ys, np.full(m, z)], 1)

    centres = (np.arange(n_lines) - (n_lines - 1) / 2) * pitch
    foot = [np.full(m + 1, -h)]
    for c in centres:
        side = []
        for s in (-1.0, 1.0):
            f = geometry.gaussian_random_field_1d(m + 1, spacing, sigma, corr, rng)
            side.append((c + s * (top_cd / 2 + run) + f, c + s * top_cd / 2 + f))
        foot += [side[0][0], side[1][0]]
        z = np.linspace(0.0, height, rows + 1)
        for (bottom, top), left in zip(side, (True, False)):
            for za, zb in zip(z[:-1], z[1:]):
                xa, xb = (bottom + (top - bottom) * v / height for v in (za, zb))
                corners = (at(xa, za, True), at(xb, zb, True), at(xb, zb, False), at(xa, za, False))
                out += _quads(1, geometry.VACUUM, *(corners if left else (corners[0], corners[3], corners[2], corners[1])))
        tl, tr = side[0][1], side[1][1]
        out += _quads(1, geometry.VACUUM, at(tl, height, True), at(tr, height, True), at(tr, height, False), at(tl, height, False))
        for k, sign in ((0, -1), (m, 1)):
            (bl, tl), (br, tr) = ((e[0][k], e[1][k]) for e in side)
            p = [[bl, y[k], 0.0], [br, y[k], 0.0], [tr, y[k], height], [tl, y[k], height]]
            p = [np.array([v]) for v in (p if sign < 0 else [p[0], p[3], p[2], p[1]])]
            out += _quads(1, geometry.VACUUM, *p)
    foot.append(np.full(m + 1, h))
    for k in range(len(foot) - 1):
        mo = 1 if k % 2 else geometry.VACUUM
        out += _quads(0, mo, at(foot[k], 0.0, True), at(foot[k + 1], 0.0, True), at(foot[k + 1], 0.0, False), at(foot[k], 0.0, False))
    return nb.triangles_from_vertices(np.vstack(out))


def _scan(case, seed):
    return primaries.raster_scan(case["nx"], case["ny"], case["per_pixel"], 0.5, case["energy"], workloads.GRATING_Z0,
                                 spot_sigma=1.0, seed=seed, pixel_streams=False)


def _pinned(n):
    return torch.empty(n * 36, dtype=torch.uint8, pin_memory=True).numpy().view(nb.PRI_DTYPE)


def prepare(case, seed):
    kind = case["kind"]
    run_seed = 0x5EED0000 + seed
    state = {"kind": kind}
    if kind == "rays":
        rng = np.random.default_rng([seed, 1])
        n = case["n"]
        state["geometry"] = nb.Geometry.from_triangles(workloads.grating_geometry())
        state["pos"] = np.stack([rng.uniform(-200, 200, n), rng.uniform(-200, 200, n), rng.uniform(-60, 45, n)], 1).astype(np.float32)
        d = rng.standard_normal((n, 3))
        state["dir"] = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
        # free paths in matter and lines of sight in vacuum
        state["dist"] = np.where(rng.random(n) < 0.7, rng.exponential(10.0, n), 2000.0).astype(np.float32)
        return state
    if kind == "batch":
        geoms, _, jobs, _ = workloads.batch(seed=seed, n_jobs=case["jobs"], scale=case["scale"])
        state["sim"] = nb.Batch([nb.Geometry.from_triangles(g) for g in geoms], [_material("si", 30e3), _material("pmma", 30e3)],
                                capacity=1 << 21, refill_threshold=0.5, block_size=512, queue_factor=8)
        state["jobs"], state["primaries"] = jobs, np.concatenate([p for _, _, p in jobs])
        return state
    if kind in ("slab", "dose"):
        energy = case["energy"]
        geo = nb.Geometry.from_triangles(geometry.slab())
        mats = [_material("si", 10e3 if energy <= 10e3 else 30e3)]
        state["primaries"] = primaries.point_beam(case["n"], energy=energy)
        more = {"deposit_grid": DOSE_GRID} if kind == "dose" else {}
        state["sim"] = nb.Simulation(geo, mats, seed=run_seed, hist_emax=energy, **more)
        return state
    model = "kieft" if kind == "kieft" else "full_penn"
    mats = [_material("si", model=model), _material("pmma", model=model)]
    state["primaries"] = _scan(case, seed)
    n = len(state["primaries"])
    tally = (case["nx"], case["ny"])
    if kind == "rough":
        geo = nb.Geometry.from_triangles(_rough_mesh(), max_depth=12, split_count=16)
    else:
        geo = nb.Geometry.from_triangles(workloads.grating_geometry())
    if kind == "adjoint":
        state["problem"] = ScanProblem(geo, mats, state["primaries"], tally, seed=run_seed, capacity=1 << 20)
        state["theta"] = state["problem"].theta0().numpy()
        return state
    capacity = 1 << 22 if n > 3_000_000 else 1 << 20
    physics = {"inelastic_model": 1} if kind == "kieft" else None
    state["sim"] = nb.Simulation(geo, mats, capacity=capacity, seed=run_seed, tally=tally, hist_emax=case["energy"],
                                 physics=physics)
    if kind == "stream":
        pinned = _pinned(n)
        pinned[:] = state["primaries"]
        state["primaries"], state["sink"] = pinned, _pinned(2 * n + (1 << 16))
    elif kind == "records":
        state["out"] = _pinned(2 * n + (1 << 16))
    return state


def _by_energy(records, room):
    """Records as words on the GPU in order of energy, then of x, at the start
    of a table with ``room`` rows."""
    words = torch.from_numpy(records.view(np.int32).reshape(-1, 9)).cuda()
    key = (words[:, 6].long() << 32) | (words[:, 0].long() & 0xFFFFFFFF)
    table = torch.zeros((room, 9), dtype=torch.int32, device="cuda")
    table[:len(words)] = words[torch.sort(key).indices]
    return table


def run(state):
    kind = state["kind"]
    if kind == "rays":
        dist, tri = state["geometry"].ray_query(state["pos"], state["dir"], state["dist"])
        return {"distance": dist, "triangle": tri}
    if kind == "batch":
        sim = state["sim"]
        sim.set_jobs(state["jobs"], state["primaries"])
        sim.run()
        se, bse = sim.job_yields()
        return {"se": se, "bse": bse, "counts": _counts(sim)}
    if kind == "adjoint":
        p = state["problem"]
        return {"yield": p.forward(state["theta"]), "jacobian": p.jacobian(state["theta"])}
    sim = state["sim"]
    sim.reset()
    if kind == "stream":
        sim.set_record_sink(state["sink"])
        sim.push_streamed(state["primaries"])
    else:
        sim.push(state["primaries"])
    sim.run()
    se, bse, hist = sim.tallies()
    out = {"se": se, "bse": bse, "hist": hist, "counts": _counts(sim)}
    if kind == "dose":
        out["dose"] = sim.deposit_grid()
    elif kind == "stream":
        # every record is in the sink here, in no particular order; the images
        # and the spectrum hold each of them once
        out["records"] = len(sim.sink_records())
    elif kind == "records":
        out["records"] = _by_energy(sim.flush_detected(state["out"]), len(state["out"]))
    return out


def _counts(sim):
    c = sim.counters()
    return np.array([c[k] for k in PHYSICAL], np.int64)


def work(case):
    """Bytes: primaries in, tallies, records and gradients out, the mesh and
    the tables once.  Operations: about 0.43 scatter events per eV of beam
    energy (215 per primary at 500 eV), each some 500 floating-point
    operations: free path, triangle tests, scattering angles and loss."""
    kind = case["kind"]
    if kind == "rays":
        return {"bytes": case["n"] * (36 + 8) + 1e6, "flops": case["n"] * 400}
    if kind == "batch":
        jobs = workloads.batch_jobs(n_jobs=case["jobs"])
        count = [max(1.0, j["n_primaries"] * case["scale"]) for j in jobs]
        events = sum(0.43 * c * j["energy"] for c, j in zip(count, jobs))
        return {"bytes": sum(count) * 36 + 1e7, "flops": events * 500}
    if kind in ("slab", "dose"):
        voxels = 8 * DOSE_GRID[2][0] * DOSE_GRID[2][1] * DOSE_GRID[2][2] if kind == "dose" else 0
        return {"bytes": case["n"] * 36 + voxels + 2e6, "flops": 0.43 * case["n"] * case["energy"] * 500}
    pixels = case["nx"] * case["ny"]
    n = pixels * case["per_pixel"]
    mesh = 1.6e8 if kind == "rough" else 3e6
    out = {"records": 1.3 * n * 36, "stream": 1.3 * n * 36, "adjoint": pixels * 6 * 8}.get(kind, 0)
    passes = 2 if kind == "adjoint" else 1
    return {"bytes": passes * n * 36 + out + pixels * 8 + mesh, "flops": passes * 0.43 * n * case["energy"] * 500}


def exact(case, seed):
    """The rays' distances in double precision, by testing every triangle.
    Transport runs have no such value: an electron's history is defined by
    comparisons of single-precision numbers with its random numbers, and
    their outputs are counts (and double-precision sums over those)."""
    if case["kind"] != "rays":
        return None
    state = prepare(case, seed)
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if device == "cpu" and case["n"] > 20_000:
        return None

    def dev(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(device, torch.float64)

    tri = state["geometry"].export()[1]
    r0, e1, e2 = dev(tri["r0"]), dev(tri["e1"]), dev(tri["e2"])
    normal = torch.linalg.cross(e1, e2)
    m_in, m_out = (torch.from_numpy(tri[k].astype(np.int32)).to(device) for k in ("material_in", "material_out"))
    best = []
    for i in range(0, case["n"], 2048):
        pos, d, most = (dev(state[k][i:i + 2048]) for k in ("pos", "dir", "dist"))
        det = -(d @ normal.T)
        s = pos[:, None, :] - r0
        t = (s * normal).sum(-1) / det
        q = torch.linalg.cross(s, d[:, None, :].expand_as(s))
        u, v = (q * e2).sum(-1) / det, -(q * e1).sum(-1) / det
        hit = (det.abs() > 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0) & (t < most[:, None])
        hit &= torch.where(det > 0, m_in, m_out) != geometry.VACUUM
        best.append(torch.minimum(torch.where(hit, t, torch.inf).amin(1), most))
    return {"distance": torch.cat(best).cpu().numpy(), "triangle": None}
