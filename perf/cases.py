"""Performance cases: what a program built on this package has it do.

Every case is a dict of plain values.  Its "kind" names the public entry point:

  host_map   Mesh.map: one surface-density map into a host array, the call of a
             script or a notebook (the array goes up, the map comes back)
  map        Mesh.map_device: one map into device memory on the caller's stream
  batch      Batch.launch: the maps of many cutouts in one persistent launch,
             replayed from a CUDA graph
  grid       Mesh.grid_device: the 3-D grid of the column walk
  whole      compute_density, the drop-in C entry point: host particles and host
             tetrahedra in, densities and map out; mesh build and copies included
  density    dtfe_density_noalloc: per-vertex densities on device arrays
  serve      Server.submit and Server.wait: a burst of map requests over
             resident cutouts, axes, sides and samples mixed

Particles come from sdtfe_b200.workloads (the recipes of the benchmark),
centred on the origin, and are triangulated by Qhull as the package's users do.
Qhull takes about 30 us a particle on one core, so a recipe's particles of one
size are triangulated once per process; a seed then picks one of the 48 symmetries of the
cube (a Delaunay mesh stays one), the particle mass and the Monte Carlo samples.

exact() is the same quantity in 64 bits in plain torch: densities by
scatter-add, the tets' linear fields by 3x3 solves, and every ray walked from
tet to tet through the planes of the faces.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import sdtfe_b200 as sd
from sdtfe_b200 import workloads

F64, MIXED = sd.DTFE_FP64, sd.DTFE_MIXED


def listed():
    return [
        # The smallest call: a few thousand particles, a thumbnail map into a
        # host array.  Launches, copies and synchronisation are what it costs.
        dict(name="thumbnail", kind="host_map", recipe="clustered", n=4096, precision=MIXED, side=64, samples=4,
             axis=0, box=1.0, depth=1.0, delta=0.0),
        # The benchmark's small plain map: uniform FP64 positions, FP64 walk.
        dict(name="plain_f64", kind="map", recipe="uniform", n=32768, precision=F64, side=256, samples=4, axis=0,
             box=1.0, depth=1.0, delta=0.0),
        # The same positions (no floats, so the walk's guards read FP64
        # records) walked in mixed precision, at a finer map.
        dict(name="plain_mixed", kind="map", recipe="uniform", n=32768, precision=MIXED, side=512, samples=4, axis=0,
             box=1.0, depth=1.0, delta=0.0),
        # The headline workload's recipe at an eighth of its particles: the
        # clustered box in full, 16 samples per pixel, mixed precision.
        dict(name="clustered_mixed", kind="map", recipe="clustered", n=131072, precision=MIXED, side=1024, samples=16,
             axis=0, box=1.0, depth=1.0, delta=0.0),
        # Its FP64 counterpart: the walk that every accuracy statement is made against.
        dict(name="clustered_f64", kind="map", recipe="clustered", n=131072, precision=F64, side=512, samples=16,
             axis=0, box=1.0, depth=1.0, delta=0.0),
        # A window on a halo's core along x: odd side, a slab shorter than the
        # mesh, samples drawn from a box wider than the pixel.
        dict(name="halo_window", kind="map", recipe="halo", n=65536, precision=MIXED, side=333, samples=7, axis=1,
             box=0.73, depth=1.1, delta=0.004),
        # Cutouts of uneven size in one launch, mixed and FP64.
        dict(name="batch_mixed", kind="batch", recipe="halo", n=40000, maps=16, precision=MIXED, side=512, samples=8),
        dict(name="batch_f64", kind="batch", recipe="halo", n=20000, maps=8, precision=F64, side=256, samples=8),
        # 3-D grids: the large field's recipe at one sample per cell, and a
        # small supersampled FP64 grid.
        dict(name="grid_mixed", kind="grid", recipe="lattice", n=83000, precision=MIXED, side=256, ss=1, box=1.0),
        dict(name="grid_f64", kind="grid", recipe="clustered", n=32768, precision=F64, side=120, ss=2, box=1.0),
        # The reference user's one call, everything on the host before and after.
        dict(name="whole_call", kind="whole", recipe="clustered", n=131072, side=512, samples=4, box=1.0, depth=1.0),
        # A burst of requests to the serving loop.
        dict(name="serve", kind="serve", recipe="clustered", n=20000, meshes=6, requests=24, precision=MIXED,
             side=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host_map", "map", "map", "map", "batch", "grid", "whole", "density", "serve"])
    recipe = rng.choice(["uniform", "clustered", "halo", "lattice"])
    precision = rng.choice([F64, MIXED, MIXED])
    full = 2.0 if recipe == "halo" else 1.0
    if kind == "density":
        return dict(kind=kind, recipe=recipe, n=_log(rng, 2000, 131072))
    if kind == "batch":
        return dict(kind=kind, recipe="halo", n=_log(rng, 5000, 40000), maps=rng.randint(2, 16), precision=precision,
                    side=_log(rng, 64, 400), samples=rng.randint(1, 12))
    if kind == "serve":
        return dict(kind=kind, recipe="clustered", n=_log(rng, 5000, 20000), meshes=rng.randint(2, 6),
                    requests=rng.randint(4, 24), precision=precision, side=_log(rng, 96, 400))
    if kind == "grid":
        return dict(kind=kind, recipe=recipe, n=_log(rng, 2000, 65536), precision=precision, side=_log(rng, 24, 160),
                    ss=rng.randint(1, 3), box=full * rng.uniform(0.3, 1.0))
    if kind == "whole":
        return dict(kind=kind, recipe=recipe, n=_log(rng, 2000, 131072), side=_log(rng, 32, 400),
                    samples=rng.randint(1, 8), box=full * rng.uniform(0.5, 1.0), depth=full)
    small = kind == "host_map"
    box = full * rng.choice([1.0, rng.uniform(0.1, 1.0)])
    side = _log(rng, 17, 200) if small else _log(rng, 48, 700)
    # up to a few hundred samples on small maps: rays stay within the largest case's
    most = max(1, min(64, (200_000 if small else 4_000_000) // side ** 2))
    return dict(kind=kind, recipe=recipe, n=_log(rng, 2000, 16384 if small else 131072), precision=precision,
                side=side, samples=_log(rng, 1, most), axis=rng.randint(0, 2), box=box,
                depth=rng.choice([full, full * rng.uniform(0.2, 0.9)]),
                delta=rng.choice([0.0, 0.0, box / side * rng.uniform(1.1, 3.0)]))


# --- inputs -----------------------------------------------------------------


@functools.lru_cache(maxsize=64)
def _triangulated(recipe, n, k):
    """Particles of one recipe, centred, and their Qhull tetrahedra (rows of tetra_data)."""
    if recipe == "uniform":
        pos = np.zeros((n, 4))
        pos[:, :3] = np.random.default_rng(1 + k).random((n, 3)) - 0.5
    elif recipe == "clustered":
        pos = workloads.clustered_box(n, seed=2 + k)[0]
        pos[:, :3] = (pos[:, :3] - 0.5).astype(np.float32)
    elif recipe == "halo":
        pos = workloads.halo_cutout(n, seed=3 + k)
    else:  # the large field: a lattice side whose recipe gives about n particles
        side = max(4, round((n / 1.3) ** (1 / 3)))
        pos = workloads.perturbed_lattice(side, n_clusters=max(1, 2000 * side ** 3 // 192 ** 3), seed=5 + k)
        pos[:, :3] = (pos[:, :3] - 0.5).astype(np.float32)
    return pos, sd.triangulate(pos)


def _mesh_input(recipe, n, seed, k=0):
    """(particle_data, tetra_data, p_mass): the recipe under the seed's symmetry of the cube."""
    pos, rows = _triangulated(recipe, n, k)
    rng = np.random.default_rng([seed, k])
    out = np.zeros_like(pos)
    out[:, :3] = pos[:, rng.permutation(3)] * rng.choice([-1.0, 1.0], 3)
    mass = float(np.float32(rng.uniform(0.5, 2.0)))
    # the layout step again: a reflection turns every tetrahedron's orientation around
    return out, sd.tetra_from_cells(out, rows[:, :4], rows[:, 4:]), mass


def _map_params(case, seed, **over):
    c = {"depth": 0.0, "delta": 0.0, "axis": 0, **case, **over}
    return sd.map_params(c["side"], c["box"], c["depth"], (0.0, 0.0, 0.0), c["samples"], c["delta"], seed=seed + 1,
                         axis=c["axis"], precision=c["precision"])


def _batch_maps(case, seed):
    """(mesh number, symmetry seed, side) of a batch: four cutout sizes, each under
    several symmetries, and sides of the case's, a half and a quarter of it."""
    rng = np.random.default_rng(77)
    return [(i % 4, seed + 1000 * (i // 4), max(16, case["side"] >> int(rng.integers(0, 3))))
            for i in range(case["maps"])]


def _batch_n(case, k):
    return max(2000, int(case["n"] * 0.6 ** k))


def _serve_requests(case):
    rng = np.random.default_rng(78)
    return [dict(mesh=int(rng.integers(case["meshes"])), axis=int(rng.integers(3)),
                 side=max(16, case["side"] >> int(rng.integers(0, 3))), samples=int(rng.integers(4, 17)), box=1.0,
                 depth=1.0, precision=case["precision"]) for _ in range(case["requests"])]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, seed=seed)
    dev = torch.device("cuda")
    if kind == "batch":
        meshes, jobs, outs = {}, [], []
        for k, sym, side in _batch_maps(case, seed):
            if (k, sym) not in meshes:
                meshes[k, sym] = sd.Mesh(*_mesh_input(case["recipe"], _batch_n(case, k), sym, k))
            out = torch.zeros(side, side, dtype=torch.float64, device=dev)
            p = _map_params(case, seed + len(jobs), side=side, box=2.0, depth=2.0)
            jobs.append((meshes[k, sym], p, out.data_ptr()))
            outs.append(out)
        s.update(batch=sd.Batch(jobs, sd.BATCH_GRAPH | sd.BATCH_ZERO_MAPS), out=outs, stream=torch.cuda.Stream())
        return s
    if kind == "serve":
        server = sd.Server(device_budget=8 << 30)
        meshes = [sd.Mesh(*_mesh_input(case["recipe"], _batch_n(case, k % 3), seed + k, k % 3), flags=sd.MESH_LAZY)
                  for k in range(case["meshes"])]
        ids = [server.add_mesh(m) for m in meshes]
        reqs = _serve_requests(case)
        s.update(server=server, reqs=[(ids[r["mesh"]], _map_params(r, seed + i)) for i, r in enumerate(reqs)],
                 out=[np.zeros((r["side"], r["side"])) for r in reqs])
        return s
    pos, tetra, mass = _mesh_input(case["recipe"], case["n"], seed)
    if kind == "whole":
        s.update(pos=pos, tetra=tetra, mass=mass, out=np.zeros((case["side"], case["side"])))
        return s
    if kind == "density":
        s.update(pos=torch.from_numpy(pos).to(dev), tetra=torch.from_numpy(tetra).to(dev), mass=mass,
                 out=torch.zeros(len(pos), dtype=torch.float64, device=dev), stream=torch.cuda.Stream())
        return s
    s["mesh"] = sd.Mesh(pos, tetra, mass)
    if kind == "grid":
        s.update(out=torch.zeros((case["side"],) * 3, dtype=torch.float64, device=dev), stream=torch.cuda.Stream())
        return s
    s["params"] = _map_params(case, seed)
    if kind == "map":
        s.update(out=torch.zeros(case["side"], case["side"], dtype=torch.float64, device=dev), stream=torch.cuda.Stream())
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "host_map":
        return s["mesh"].map(s["params"])[0]
    if kind == "batch":
        s["batch"].launch(s["stream"].cuda_stream)
        return s["out"]
    if kind == "serve":
        rids = [s["server"].submit(m, p, o) for (m, p), o in zip(s["reqs"], s["out"])]
        return [s["server"].wait(r)[0] for r in rids]
    if kind == "whole":
        s["out"].fill(0.0)
        L = sd.lib()
        L.dtfe_set_seed(s["seed"] + 1)
        L.compute_density(s["pos"], len(s["pos"]), s["tetra"], len(s["tetra"]), case["side"], case["box"],
                          case["depth"], s["out"].reshape(-1), s["mass"], 0.0, 0.0, 0.0, case["samples"], 0.0)
        return {"density": s["pos"][:, 3].copy(), "map": s["out"]}
    if kind == "density":
        status = sd.lib().dtfe_density_noalloc(
            _ptr(s["pos"]), len(s["pos"]), _ptr(s["tetra"]), len(s["tetra"]), ctypes.c_float(s["mass"]),
            _ptr(s["out"]), ctypes.c_void_p(s["stream"].cuda_stream))
        if status:
            raise RuntimeError("dtfe_density_noalloc: status %d" % status)
        return s["out"]
    # maps and grids are added to what the array holds: a new one starts at zero
    with torch.cuda.stream(s["stream"]):
        s["out"].zero_()
    if kind == "grid":
        s["mesh"].grid_device(case["side"], case["box"], (0.0, 0.0, 0.0), case["ss"], s["seed"] + 1,
                              s["out"].data_ptr(), case["precision"], s["stream"].cuda_stream)
    else:
        s["mesh"].map_device(s["params"], s["out"].data_ptr(), s["stream"].cuda_stream)
    return s["out"]


def _ptr(x):
    return ctypes.c_void_p(x.data_ptr())


# --- the work that no implementation can do without ---------------------------

TETS = 6.7  # tetrahedra per particle of a Delaunay mesh
STEP = 45   # flops per tet that a ray crosses: three edge products, one crossing, one field value


def _crossings(n):
    """Tets that one ray through the whole mesh crosses, about."""
    return 3.5 * n ** (1 / 3)


def work(case):
    kind = case["kind"]
    n = case["n"]
    mesh = n * (32 + 32 * TETS)
    if kind in ("host_map", "map", "whole"):
        part = min(1.0, case["box"] / (2.0 if case["recipe"] == "halo" else 1.0)) ** 2  # the mesh under the map
        rays = case["side"] ** 2 * case["samples"]
        b = 8.0 * case["side"] ** 2 + mesh * (1.0 if kind == "whole" else part) + (8 * n if kind == "whole" else 0)
        return dict(bytes=b, flops=rays * _crossings(n) * STEP + (mesh if kind == "whole" else 0))
    if kind == "density":
        return dict(bytes=mesh + 8 * n, flops=20 * TETS * n)
    if kind == "grid":
        rays = (case["side"] * case["ss"]) ** 2
        return dict(bytes=8.0 * case["side"] ** 3 + mesh,
                    flops=rays * (_crossings(n) * STEP + 5 * case["side"] * case["ss"]))
    total = dict(bytes=0.0, flops=0.0)
    if kind == "batch":
        each = [(_batch_n(case, k), side, case["samples"]) for k, _, side in _batch_maps(case, 0)]
    else:
        each = [(_batch_n(case, r["mesh"] % 3), r["side"], r["samples"]) for r in _serve_requests(case)]
    for m, side, samples in each:
        total["bytes"] += m * (32 + 32 * TETS) + 8.0 * side ** 2
        total["flops"] += side ** 2 * samples * _crossings(m) * STEP
    return total


# --- the same in 64 bits ------------------------------------------------------

M64 = 0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB


def _i64(u):
    u &= (1 << 64) - 1
    return u - (1 << 64) if u >> 63 else u


def _shr(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def _mix(z):
    z = z + _i64(M64[0])
    z = (z ^ _shr(z, 30)) * _i64(M64[1])
    z = (z ^ _shr(z, 27)) * _i64(M64[2])
    return z ^ _shr(z, 31)


def _u01(seed, pixel, sample, axis):
    """The sample offsets that a map is defined by: SplitMix64 of (seed, pixel, sample, axis)."""
    h = _mix((pixel + 1) * _i64(0x632BE59BD9B4E019) + _i64(seed))
    return _shr(_mix(h ^ (sample * 2 + axis)), 11).double() * 2.0 ** -53


def _exact_density(pos, tet, mass):
    v = pos[tet, :3]
    e = v[:, :3] - v[:, 3:]
    vol = torch.linalg.cross(e[:, 1], e[:, 2]).mul(e[:, 0]).sum(1).abs() / 6
    total = torch.zeros(len(pos), dtype=torch.float64, device=pos.device)
    total.index_add_(0, tet.reshape(-1), vol.repeat_interleave(4))
    return float(np.float32(mass) * np.float32(4)) / total


class _Field:
    """The mesh's linear field along the projection axis: per tet its faces' planes
    z = c - a (x - px) - b (y - py), which way they face, and its gradient."""

    def __init__(self, pos, rows, mass, axis):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        pos = torch.from_numpy(pos).to(dev)
        tet = torch.from_numpy(np.ascontiguousarray(rows[:, :4])).long().to(dev)
        self.nb = torch.from_numpy(np.ascontiguousarray(rows[:, 4:])).long().to(dev)
        rho = _exact_density(pos, tet, mass)
        xyz = pos[:, [axis, (axis + 1) % 3, (axis + 2) % 3]]
        v = xyz[tet]
        edge = v[:, 1:] - v[:, :1]
        rise = (rho[tet[:, 1:]] - rho[tet[:, :1]]).unsqueeze(2)
        d0, d1, d2 = edge[:, 0], edge[:, 1], edge[:, 2]
        c0, c1, c2 = torch.linalg.cross(d1, d2), torch.linalg.cross(d2, d0), torch.linalg.cross(d0, d1)
        grad = (c0 * rise[:, 0] + c1 * rise[:, 1] + c2 * rise[:, 2]) / (d0 * c0).sum(1, keepdim=True)
        self.value = torch.cat([v[:, 0], rho[tet[:, :1]], grad], 1)
        plane, up = [], []
        for f in range(4):
            p, q, r = (v[:, k] for k in range(4) if k != f)
            nrm = torch.linalg.cross(q - p, r - p)
            nrm = nrm * -torch.sign((nrm * (v[:, f] - p)).sum(1, keepdim=True))
            plane.append(torch.cat([p, nrm[:, :2] / nrm[:, 2:]], 1))
            up.append(torch.sign(nrm[:, 2]))
        self.plane, self.up = torch.stack(plane, 1), torch.stack(up, 1)
        low = (self.nb == -1) & (self.up < 0)
        t, f = low.nonzero(as_tuple=True)
        others = torch.tensor([[k for k in range(4) if k != j] for j in range(4)], device=dev)[f]
        self.tri, self.tri_tet = v[t[:, None], others][:, :, :2], t

    def first(self, x, y):
        """The tet through whose lower boundary face the line (x, y) comes in (-1: none)."""
        t = torch.full_like(x, -1, dtype=torch.long)
        for (a, b, c), k in zip(self.tri.tolist(), self.tri_tet.tolist()):
            s = [(q[0] - p[0]) * (y - p[1]) - (q[1] - p[1]) * (x - p[0]) for p, q in ((a, b), (b, c), (c, a))]
            t[((s[0] >= 0) & (s[1] >= 0) & (s[2] >= 0)) | ((s[0] <= 0) & (s[1] <= 0) & (s[2] <= 0))] = k
        return t

    def walk(self, x, y, chord):
        """chord(rays, tet, x, y, z_in, z_out) for every tet that each line crosses; which lines met the mesh."""
        tet = self.first(x, y)
        ray = (tet >= 0).nonzero()[:, 0]
        hit = tet >= 0
        tet, x, y, z_in = tet[ray], x[ray], y[ray], None
        while len(ray):
            p, up = self.plane[tet], self.up[tet]
            z = p[:, :, 2] - p[:, :, 3] * (x[:, None] - p[:, :, 0]) - p[:, :, 4] * (y[:, None] - p[:, :, 1])
            if z_in is None:
                z_in = torch.where(up < 0, z, -torch.inf).amax(1)
            z_out, face = torch.where(up > 0, z, torch.inf).min(1)
            chord(ray, tet, x, y, z_in, z_out)
            tet = self.nb[tet, face]
            on = tet >= 0
            if not bool(on.all()):
                ray, tet, x, y, z_out = ray[on], tet[on], x[on], y[on], z_out[on]
            z_in = z_out
        return hit

    def at(self, tet, x, y, z):
        v = self.value[tet]
        return v[:, 3] + v[:, 4] * (x - v[:, 0]) + v[:, 5] * (y - v[:, 1]) + v[:, 6] * (z - v[:, 2])


def _exact_map(pos, rows, mass, side, samples, box, depth, seed, axis=0, delta=0.0):
    fld = _Field(pos, rows, mass, axis)
    dev = fld.nb.device
    dxy = box / side
    scale = max(delta, dxy)
    off = -box / 2 - (scale - dxy) / 2
    out = torch.zeros(side * side, dtype=torch.float64, device=dev)
    step = max(1, (1 << 22) // samples)
    for p0 in range(0, side * side, step):
        pix = torch.arange(p0, min(p0 + step, side * side), device=dev).repeat_interleave(samples)
        smp = torch.arange(samples, device=dev).repeat(len(pix) // samples)
        x = (pix % side).double() * dxy + off + _u01(seed, pix, smp, 0) * scale
        y = torch.div(pix, side, rounding_mode="floor").double() * dxy + off + _u01(seed, pix, smp, 1) * scale
        total = torch.zeros_like(x)

        def chord(ray, tet, x, y, z_in, z_out):
            mid = (z_in + z_out) / 2
            inside = (mid > -depth / 2) & (mid < depth / 2)
            total[ray] += torch.where(inside, fld.at(tet, x, y, mid) * (z_out - z_in), 0.0)

        hit = fld.walk(x, y, chord)
        n = hit.view(-1, samples).sum(1)
        out[p0:p0 + step] = torch.where(n > 0, total.view(-1, samples).sum(1) / n.clamp(min=1), 0.0)
    return out.view(side, side)


def _exact_grid(pos, rows, mass, side, ss, box):
    fld = _Field(pos, rows, mass, 0)
    dev = fld.nb.device
    fine = box / side / ss
    cols = torch.arange(side * ss, device=dev)
    x = (-box / 2 + (cols.double() + 0.5) * fine).repeat_interleave(side * ss)
    y = (-box / 2 + (cols.double() + 0.5) * fine).repeat(side * ss)
    cell = (cols // ss).repeat_interleave(side * ss) * side + (cols // ss).repeat(side * ss)
    out = torch.zeros(side ** 3, dtype=torch.float64, device=dev)
    nodes = side * ss

    def chord(ray, tet, x, y, z_in, z_out):
        lo = ((z_in + box / 2) / fine - 0.5).ceil().clamp(0, nodes).long()
        hi = ((z_out + box / 2) / fine - 0.5).ceil().clamp(0, nodes).long()
        while True:
            on = (lo < hi).nonzero()[:, 0]
            if not len(on):
                return
            ray, tet, x, y, lo, hi = (v[on] for v in (ray, tet, x, y, lo, hi))
            z = -box / 2 + (lo.double() + 0.5) * fine
            out.index_add_(0, cell[ray] * side + lo // ss, fld.at(tet, x, y, z) / ss ** 3)
            lo = lo + 1

    fld.walk(x, y, chord)
    return out.view((side,) * 3)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_exact_map(*_mesh_input(case["recipe"], _batch_n(case, k), sym, k), side, case["samples"], 2.0, 2.0,
                           seed + i + 1) for i, (k, sym, side) in enumerate(_batch_maps(case, seed))]
    if kind == "serve":
        return [_exact_map(*_mesh_input(case["recipe"], _batch_n(case, r["mesh"] % 3), seed + r["mesh"], r["mesh"] % 3),
                           r["side"], r["samples"], 1.0, 1.0, seed + i + 1, r["axis"])
                for i, r in enumerate(_serve_requests(case))]
    pos, rows, mass = _mesh_input(case["recipe"], case["n"], seed)
    if kind == "grid":
        return _exact_grid(pos, rows, mass, case["side"], case["ss"], case["box"])
    if kind in ("density", "whole"):
        rho = _exact_density(torch.from_numpy(pos), torch.from_numpy(rows[:, :4].copy()).long(), mass)
        if kind == "density":
            return rho
        return {"density": rho, "map": _exact_map(pos, rows, mass, case["side"], case["samples"], case["box"],
                                                  case["depth"], seed + 1)}
    return _exact_map(pos, rows, mass, case["side"], case["samples"], case["box"], case["depth"], seed + 1,
                      case["axis"], case["delta"])
