"""Performance cases: the work a program has this framework do, through its
public entry points, on synthetic vessels.

Whole jobs (mesh in, labels and counts out), batches of uneven jobs, the grid
calls of the interactive and the dataset path, fragment meshes, rays and the
device-buffer flood.  `listed()` gives fixed cases, `draw()` more of the same
ranges; `prepare` / `run` / `work` / `exact` work on any of them.
"""
import ctypes as C
import math

import numpy as np
import torch

import voxelfragmentml_gb300 as V
from voxelfragmentml_gb300 import vessel as Vs, workloads as W


def listed():
    return [
        # one small model, pageable output buffers: the latency of a single call
        dict(name="job_64", kind="job", x=60, y=57, z=64, angular=64, profile=48, fragments=6,
             distance=V.MANHATTAN, amplitude=0.0, erode=0, pinned=0),
        # one ordinary model with boundary noise and one erosion
        dict(name="job_256_eroded", kind="job", x=240, y=240, z=256, angular=256, profile=192,
             fragments=16, distance=V.EUCLIDEAN, amplitude=2.0, erode=1, pinned=1),
        # one large model
        dict(name="job_512", kind="job", x=476, y=476, z=512, angular=512, profile=384,
             fragments=64, distance=V.CHEBYSHEV, amplitude=2.0, erode=0, pinned=1),
        # a micro-batch of uneven models, meshes up and labels down in the call
        dict(name="batch_48", kind="batch", jobs=48, mix=11, resident=0),
        # a large batch whose meshes stay on the GPU, every stage re-run on them
        dict(name="resident_128", kind="batch", jobs=128, mix=12, resident=1),
        # the dataset path on one grid, default fracture parameters: fill, fracture with
        # extra seeds, erosion, counts, run-length export
        dict(name="model_200_extra", kind="model", x=200, y=197, z=208, angular=160, profile=120,
             fragments=8, extra=16, distance=V.CHEBYSHEV, erode=1, amplitude=0.0),
        # an impact on a model in the viewer: entry voxels, seeds around the impact, flood
        dict(name="impact_160", kind="impact", x=150, y=150, z=160, fragments=8, near=32,
             distance=V.EUCLIDEAN),
        # Voronoi fracture by straight distance, wide boundaries
        dict(name="voronoi_192", kind="voronoi", x=180, y=179, z=192, fragments=64,
             distance=V.EUCLIDEAN, boundary=2),
        # the raw surface (no smoothing) of a small model's fragments, with point clouds
        dict(name="mesh_96_raw", kind="mesh", x=90, y=91, z=96, fragments=8, smooth=0, marked=0,
             points=1024),
        # smoothed fragment meshes of a large model
        dict(name="mesh_512", kind="mesh", x=476, y=476, z=512, fragments=64, smooth=1, marked=1,
             points=0),
        # entry voxels of a picking / visibility pass
        dict(name="rays_1m", kind="rays", x=240, y=239, z=256, rays=1 << 20),
        # the flood alone, on the caller's device buffers
        dict(name="flood_128", kind="flood", x=120, y=121, z=127, fragments=8,
             distance=V.MANHATTAN),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, lo, hi):
    """A model's grid: the height spread over the range, the sides near it, any parity."""
    z = int(round(_log(rng, lo, hi)))
    side = [max(16, int(round(z * rng.uniform(0.8, 1.0)))) for _ in range(2)]
    return dict(x=side[0], y=side[1], z=z)


def _samples(rng, z):
    a = max(16, int(round(z * rng.uniform(0.5, 1.1))))
    return dict(angular=a, profile=max(8, int(round(0.75 * a))))


def draw(rng):
    kind = rng.choice(("job", "job", "job", "batch", "batch", "model", "impact", "voronoi", "mesh",
                       "mesh", "rays", "flood"))
    metric = rng.choice((V.EUCLIDEAN, V.MANHATTAN, V.CHEBYSHEV))
    if kind == "job":
        d = _dims(rng, 40, 440)
        return dict(kind=kind, **d, **_samples(rng, d["z"]), fragments=rng.randint(2, 64),
                    distance=metric, amplitude=rng.choice((0.0, round(rng.uniform(0.5, 3.0), 2))),
                    erode=rng.choice((0, 0, 1)), pinned=rng.choice((0, 1, 1)))
    if kind == "batch":
        return dict(kind=kind, jobs=int(round(_log(rng, 4, 112))), mix=rng.randrange(1000),
                    resident=rng.choice((0, 1)))
    if kind == "model":
        d = _dims(rng, 48, 260)
        return dict(kind=kind, **d, **_samples(rng, d["z"]), fragments=rng.randint(3, 24),
                    extra=rng.choice((0, 8, 16, 40)), distance=metric, erode=rng.choice((0, 1)),
                    amplitude=rng.choice((0.0, 1.5)))
    if kind == "impact":
        return dict(kind=kind, **_dims(rng, 48, 320), fragments=rng.randint(2, 32),
                    near=rng.choice((8, 32, 64)), distance=metric)
    if kind == "voronoi":
        return dict(kind=kind, **_dims(rng, 48, 256), fragments=rng.randint(2, 128), distance=metric,
                    boundary=rng.choice((1, 2, 3)))
    if kind == "mesh":
        smooth = rng.choice((0, 1, 1))
        return dict(kind=kind, **_dims(rng, 40, 400), fragments=rng.randint(2, 64), smooth=smooth,
                    marked=smooth, points=rng.choice((0, 1024)))
    if kind == "rays":
        return dict(kind=kind, **_dims(rng, 64, 400), rays=int(round(_log(rng, 256, 1 << 20))))
    return dict(kind="flood", **_dims(rng, 40, 160), fragments=rng.randint(2, 48), distance=metric)


# ---- inputs -----------------------------------------------------------------------
def _job_spec(case, seed):
    v, f = Vs.vessel_mesh(case["angular"], case["profile"], seed)
    p = V.Params.default(algorithm=V.FLOOD, distance=case["distance"], num_seeds=case["fragments"],
                         seed=seed * 7919 + 1, seed_location=V.BOTH,
                         noise_amplitude=case["amplitude"], noise_period=16, boundary_size=1)
    if case["erode"]:
        p.erode, p.erosion_type, p.erosion_size, p.erosion_iterations = 1, V.SQUARE, 3, 1
    pinned = bool(case["pinned"])
    if pinned:
        pv, pf = V.pinned_array(v.shape, np.float32), V.pinned_array(f.shape, np.uint32)
        pv[...], pf[...] = v, f
        v, f = pv, pf
    return V.JobSpec(v, f, p, dims=(case["x"], case["y"], case["z"]), aabb=Vs.mesh_aabb(v),
                     ncounts=256, pinned=pinned)


def _batch_specs(case, seed):
    """The jobs of a mixed batch; their labels lie one after another in one pinned buffer."""
    jobs = W.mixed(case["jobs"], case["mix"])
    sizes = [-(-int(np.prod(j["dims"])) // 64) * 64 for j in jobs]
    labels = V.pinned_array((sum(sizes),), np.uint16)
    labels[...] = 0
    counts = np.zeros((len(jobs), 256), np.uint32)
    specs, at = [], 0
    for i, (j, n) in enumerate(zip(jobs, sizes)):
        j["mesh_seed"], j["seed"] = seed * 1009 + i, seed * 31 + 7 * i + 1
        s = W.to_spec(j, V, want_labels=False, pinned=True)
        s.labels = labels[at:at + int(np.prod(s.dims))].reshape(s.dims)
        s.counts = counts[i]
        specs.append(s)
        at += n
    return specs, labels, counts


def _vessel_occupancy(dims, seed):
    """A thin-walled pot on the GPU: bool [X][Y][Z], the shape class of the vessel meshes."""
    g = np.random.Generator(np.random.PCG64(seed))
    c = g.uniform(-0.02, 0.02, 3)
    X, Y, Z = dims
    ax = [(torch.arange(n, device="cuda", dtype=torch.float32) + 0.5) / n for n in dims]
    z = ax[2]
    r = 0.3 + 0.15 * torch.sin(3.0 * z) + float(c[0]) + float(c[1]) * z + float(c[2]) * z * z
    rho = torch.hypot((ax[0] - 0.5)[:, None], (ax[1] - 0.5)[None, :])[:, :, None]
    wall = max(0.03, 1.6 / min(dims))
    return (rho <= r) & ((rho >= r - wall) | (z <= wall))


def _fragment_labels(dims, fragments, marked, seed):
    """uint16 labels 2.. of the occupied voxels by the nearest of random surface points, the
    voxels next to another fragment marked by bit 15 when asked."""
    occ = _vessel_occupancy(dims, seed)
    at = torch.nonzero(occ.reshape(-1)).reshape(-1)
    pick = np.random.Generator(np.random.PCG64(seed + 1)).integers(0, int(at.numel()), fragments)
    lin = at[torch.from_numpy(pick).cuda()].cpu().numpy()
    X, Y, Z = dims
    del at
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) for n in dims]
    best = torch.full(dims, 3e38, device="cuda")
    lab = torch.zeros(dims, dtype=torch.int16, device="cuda")
    for i, s in enumerate(lin):
        p = (int(s) // (Y * Z), int(s) // Z % Y, int(s) % Z)
        d = ((ax[0] - p[0]) ** 2)[:, None, None] + ((ax[1] - p[1]) ** 2)[None, :, None] + \
            ((ax[2] - p[2]) ** 2)[None, None, :]
        closer = d < best
        best = torch.where(closer, d, best)
        lab.masked_fill_(closer, 2 + i)
        del d, closer
    del best
    lab = torch.where(occ, lab, torch.zeros_like(lab))
    if marked:
        edge = torch.zeros(dims, dtype=torch.bool, device="cuda")
        for a in range(3):
            lo, hi = lab.narrow(a, 0, dims[a] - 1), lab.narrow(a, 1, dims[a] - 1)
            other = (lo != hi) & (lo > 1) & (hi > 1)
            edge.narrow(a, 0, dims[a] - 1).logical_or_(other)
            edge.narrow(a, 1, dims[a] - 1).logical_or_(other)
        lab = torch.where(edge, lab | -32768, lab)
    return lab


def _grid(case, host):
    dims = (case["x"], case["y"], case["z"])
    g = V.RegularGrid(dims, (-0.5, -0.5, 0.0), (0.5, 0.5, 1.0))
    up = V.pinned_array(dims, np.uint16)
    up[...] = host.cpu().numpy().view(np.uint16)
    g.upload(up)
    return g


def _surface(case):
    """Voxels of the grid's box surface: a model's wall has a few times as many."""
    return 2 * (case["x"] * case["y"] + case["y"] * case["z"] + case["x"] * case["z"])


def _kept(shape, dtype):
    """A page-locked buffer a program keeps from call to call, larger than a result can be."""
    a = V.pinned_array(shape, dtype)
    a[...] = 0
    return a


def prepare(case, seed):
    kind, dims = case["kind"], tuple(case.get(a, 0) for a in "xyz")
    s = dict(case=case)
    if kind == "job":
        s["spec"] = _job_spec(case, seed)
    elif kind == "batch":
        s["specs"], s["labels"], s["counts"] = _batch_specs(case, seed)
        if case["resident"]:
            s["resident"] = V.ResidentBatch(s["specs"], V.Context(0))
    elif kind == "model":
        v, f = Vs.vessel_mesh(case["angular"], case["profile"], seed)
        s["verts"], s["faces"] = v, f
        s["grid"] = V.RegularGrid(dims, *Vs.mesh_aabb(v))
        s["params"] = V.Params.default(num_seeds=case["fragments"], num_extra_seeds=case["extra"],
                                       distance=case["distance"], erode=case["erode"],
                                       noise_amplitude=case["amplitude"], seed=seed + 17)
        s["rle"] = np.zeros(4096 + 2 * dims[0] * dims[1] * dims[2], np.uint8)
    elif kind in ("impact", "voronoi"):
        s["grid"] = _grid(case, _vessel_occupancy(dims, seed).to(torch.int16))
        s["seed"] = seed + 5
        r = np.random.Generator(np.random.PCG64(seed + 2)).normal(size=(64, 3)).astype(np.float32)
        s["rays"] = np.concatenate([0.1 * r + 1.4, -r * 0.05 - 1.0], 1).astype(np.float32)
        s["fracturer"] = V.FloodFracturer() if kind == "impact" else V.NaiveFracturer()
        s["fracturer"].setDistanceFunction(case["distance"])
        s["labels"] = _kept(dims, np.uint16)
        s["used"] = np.zeros((case["fragments"] + case.get("near", 0), 4), np.uint32)
    elif kind == "mesh":
        s["grid"] = _grid(case, _fragment_labels(dims, case["fragments"], case["marked"], seed))
        s["params"] = V.MCParams.default(max(dims)) if case["smooth"] else V.MCParams(0, 0.9, 0, 0.2)
        s["seed"] = seed + 80
        F, NV = case["fragments"], 6 * _surface(case)
        s["arrays"] = (np.zeros(F, np.uint16), _kept((F + 1,), np.uint64), _kept((F + 1,), np.uint64),
                       _kept((NV, 4), np.float32), _kept((2 * NV, 4), np.uint32))
        s["points"] = np.zeros((F * case["points"], 4), np.float32)
    elif kind == "rays":
        s["grid"] = _grid(case, _vessel_occupancy(dims, seed).to(torch.int16))
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["rays"]
        o = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device="cuda"), dim=1) * 2.0
        to = torch.rand(n, 3, generator=g, device="cuda") - torch.tensor([0.5, 0.5, 0.0], device="cuda")
        s["rays"] = torch.cat([o, to - o], 1).cpu().numpy()
    else:  # flood
        occ = _vessel_occupancy(dims, seed)
        at = torch.nonzero(occ)
        pick = np.random.Generator(np.random.PCG64(seed + 1)).choice(int(at.shape[0]), case["fragments"],
                                                                     replace=False)
        xyz = at[torch.from_numpy(pick).cuda()].to(torch.int32)
        lab = torch.arange(2, 2 + case["fragments"], dtype=torch.int32, device="cuda")[:, None]
        s["seeds"] = torch.cat([xyz, lab], 1).contiguous()
        s["occ"] = occ.to(torch.int16).contiguous()
        s["labels"] = torch.empty_like(s["occ"])
    return s


# ---- one pass ---------------------------------------------------------------------
def _results(res):
    return np.array([[r.status, r.nseeds, r.voxels, r.occupied, r.fragments] for r in res], np.int64)


def _signed(a):
    return a.view(np.int16 if a.dtype == np.uint16 else np.int32)


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "job":
        res = V.batch_run([s["spec"]])
        return dict(labels=_signed(s["spec"].labels), counts=_signed(s["spec"].counts),
                    results=_results(res))
    if kind == "batch":
        res = s["resident"].execute(download=True) if case["resident"] else V.batch_run(s["specs"])
        return dict(labels=_signed(s["labels"]), counts=_signed(s["counts"]), results=_results(res))
    if kind == "model":
        g = s["grid"]
        g.fill(s["verts"], s["faces"])
        seeds = V.fracture_model(g, s["params"])
        counts, occupied = g.countValues(256)
        rle = np.frombuffer(g.exportRLE(), np.uint8)
        s["rle"][:len(rle)] = rle
        return dict(seeds=_signed(seeds), counts=_signed(counts), occupied=int(occupied),
                    rle=s["rle"], rle_bytes=len(rle))
    if kind in ("impact", "voronoi"):
        g = s["grid"]
        out = {}
        seeds = V.Seeder.uniform(g, case["fragments"], s["seed"], V.BOTH)
        if kind == "impact":
            out["entry"] = _signed(g.rayEntryVoxels(s["rays"]))
            seeds = V.Seeder.nearSeeds(g, seeds, 1, case["near"], 5, s["seed"])
        s["fracturer"].build(g, seeds)
        g.detectBoundaries(case.get("boundary", 1))
        V._check(V.lib().vf_grid_download(g.h, V._p(s["labels"])))
        s["used"][:len(seeds)] = seeds
        out.update(seeds=_signed(s["used"]), labels=_signed(s["labels"]))
        return out
    if kind == "mesh":
        g = s["grid"]
        sizes = g.triangulate(s["params"])
        vals, vo, fo, v, f = s["arrays"]
        if sizes[1] > len(v) or sizes[2] > len(f):
            raise ValueError("the kept mesh buffers are too small: %s" % (sizes,))
        V._check(V.lib().vf_grid_meshes(g.h, *(V._p(a) for a in s["arrays"])))
        out = dict(sizes=np.array(sizes, np.int64), values=_signed(vals), vert_offsets=vo.view(np.int64),
                   face_offsets=fo.view(np.int64), verts=v, faces=_signed(f))
        if case["points"]:
            pts = g.samplePointClouds(case["points"], s["seed"])
            at = 0
            for p in pts:
                s["points"][at:at + len(p)] = p
                at += len(p)
            out["points"] = s["points"]
        return out
    if kind == "rays":
        return _signed(s["grid"].rayEntryVoxels(s["rays"]))
    st = V.lib().vf_flood_noalloc(C.c_void_p(s["occ"].data_ptr()), C.c_void_p(s["labels"].data_ptr()),
                                  case["x"], case["y"], case["z"], C.c_void_p(s["seeds"].data_ptr()),
                                  case["fragments"], case["distance"], None)
    V._check(st)
    return s["labels"]


# ---- what a pass cannot do without ------------------------------------------------
def work(case):
    kind = case["kind"]
    vox = case.get("x", 0) * case.get("y", 0) * case.get("z", 0)
    mesh = 0
    if "angular" in case:
        mesh = 12 * (2 * case["angular"] * case["profile"] + 2) + 48 * case["angular"] * case["profile"]
    if kind == "job":
        return dict(bytes=mesh + 2 * vox + 1024, flops=0)
    if kind == "batch":
        jobs = W.mixed(case["jobs"], case["mix"])
        vox = sum(int(np.prod(j["dims"])) for j in jobs)
        return dict(bytes=18 * sum(j["triangles"] for j in jobs) + 2 * vox + 1024 * len(jobs), flops=0)
    if kind == "model":  # the labels are written and read by the export
        return dict(bytes=mesh + 4 * vox, flops=0)
    if kind in ("impact", "voronoi"):  # occupancy in, labels out
        return dict(bytes=4 * vox, flops=0)
    if kind == "mesh":
        # labels in; about two vertices and four faces of 16 bytes out per box surface voxel
        return dict(bytes=2 * vox + 48 * 2 * _surface(case), flops=0)
    if kind == "rays":  # occupancy bits, rays in, voxels out
        return dict(bytes=vox // 8 + 36 * case["rays"], flops=0)
    return dict(bytes=4 * vox, flops=0)


# ---- 64-bit values ----------------------------------------------------------------
def exact(case, seed):
    """Vertices of the unsmoothed fragment meshes: the midpoints between a fragment's voxels and
    their face neighbours of another value, by voxel then direction -x,+x,-y,+y,-z,+z, through
    the grid's affine map.  Smoothed positions and points have no independent value here; every
    other output is whole numbers."""
    if case["kind"] != "mesh" or case["smooth"]:
        return None
    dims = (case["x"], case["y"], case["z"])
    if dims[0] * dims[1] * dims[2] > 3 << 22:
        return None
    lab = _fragment_labels(dims, case["fragments"], case["marked"], seed).cpu().numpy()
    pad = np.pad(lab, 1, constant_values=1)
    mn, mx = np.array([-0.5, -0.5, 0.0]), np.array([0.5, 0.5, 1.0])
    scale = (mx - mn) / np.array(dims)
    verts = []
    for value in np.unique(lab[lab > 1]):
        own = np.argwhere(lab == value)
        faces = []
        for a in range(3):
            for up in (0, 1):
                q = own + 1
                q[:, a] += 1 if up else -1
                faces.append(pad[q[:, 0], q[:, 1], q[:, 2]] != value)
        at, d = np.nonzero(np.stack(faces, 1))
        p = own[at] + 1.0
        p[np.arange(len(d)), d // 2] += np.where(d % 2, 0.5, -0.5)
        verts.append(np.concatenate([p * scale + (mn - scale), np.zeros((len(d), 1))], 1))
    out = np.zeros((6 * _surface(case), 4))
    verts = np.concatenate(verts)
    out[:len(verts)] = verts
    return dict(verts=out)
