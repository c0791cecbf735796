"""Performance cases of the framework, through its public entry points.

What a program built on it spends its time in, over the range of sizes that
such programs use:

* transport runs (``Context``: upload a scene once, then zero the tallies, run
  a source, read the tallies): dose in a voxelized phantom from an X-ray or an
  embedded voxelized source, CT projections, dose in a meshed phantom, and
  several projections as the jobs of one launch;
* phantom volumes: a CT image converted to material labels, a phantom drawn
  from analytic shapes;
* the scatter surrogate: line integrals of a scan, the network's forward pass,
  its gradients and its training step.

Inputs are synthetic, made from the seed: random phantoms, images and weights,
and the random streams of the transport.
"""

import ctypes as C
import functools
import math
import os
import tempfile

import numpy as np
import torch

from ggems_b200 import abi, scatter, workloads
from ggems_b200._native import Context, Volume, check, lib

F = np.float32
DEG = math.pi / 180.0
SLOTS = abi.GG_MAXIMUM_PARTICLES
# axis matrices of the source, the phantom and the detector frames
SOURCE_AXIS = ((0.0, 0.0, -1.0), (0.0, 1.0, 0.0), (1.0, 0.0, 0.0))
DETECTOR_AXIS = ((0.0, 0.0, 1.0), (0.0, 1.0, 0.0), (-1.0, 0.0, 0.0))


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # one short dosimetry run, as in a parameter scan or an interactive check: call latency counts
        dict(name="dose_short", kind="dose", n=64, voxel=2.0, primaries=10_000, source="xray", energy=0.060, tle=False,
             tracking=False),
        # the small configuration: 64^3 water, 2 mm, 60 keV, edep / edep^2 / hits / dose
        dict(name="dose_water64", kind="dose", n=64, voxel=2.0, primaries=1_000_000, source="xray", energy=0.060,
             tle=False, tracking=False),
        # activity inside a phantom of odd size, track-length estimator and photon counts (brachytherapy style)
        dict(name="dose_emission_tle", kind="dose", n=91, voxel=1.5, primaries=2_500_000, source="voxelized",
             energy=0.140, tle=True, tracking=True),
        # the headline: one full CBCT projection, 256^3 phantom, 120 kVp, 512^2 panel, 1e8 primaries
        dict(name="cbct_256", kind="projection", n=256, voxel=1.0, ex=512, ey=512, element=0.8, primaries=100_000_000,
             spectrum=True, world=0),
        # a small projection of odd sizes with GGEMS's world grid recorded
        dict(name="projection_world", kind="projection", n=117, voxel=1.9, ex=333, ey=250, element=1.1,
             primaries=1_500_000, spectrum=True, world=61),
        # dose in a 245,760-triangle body
        dict(name="mesh_body", kind="mesh", body=6, inner=5, primaries=10_000_000, energy=0.080, dosel=2.0),
        # 36 projections of 1e6 primaries as the jobs of one launch: the surrogate's judge, training data
        dict(name="scan_jobs", kind="jobs", jobs=36, phantoms=1, primaries=1_000_000, side=256),
        # a CT image (Hounsfield units) read into labels: image up, labels back
        dict(name="labels_ct512", kind="labels", nx=512, ny=512, nz=512, met=abi.GG_MET_SHORT, ranges=8),
        # GGEMS's volume creator example: 120^3 MET_INT, a box and inserts, image back for the MHD file
        dict(name="draw_120", kind="draw", nx=120, ny=120, nz=120, voxel=0.1, met=abi.GG_MET_INT, shapes=4),
        # network inputs of a 360-angle scan
        dict(name="integrals_scan", kind="integrals", n=64, voxel=2.0, side=256, count=360),
        # surrogate inference and training at the committed network's size
        dict(name="unet_forward", kind="unet", mode="forward", batch=8, side=256),
        dict(name="unet_train", kind="unet", mode="train", batch=8, side=256),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("dose", "dose", "projection", "projection", "mesh", "jobs", "labels", "draw", "integrals", "unet",
                       "unet"))
    if kind == "dose":
        return dict(kind=kind, n=rng.randint(16, 160), voxel=rng.choice((0.7, 1.0, 1.5, 2.0, 2.5)),
                    primaries=log_int(1_000, 5_000_000), source=rng.choice(("xray", "xray", "voxelized")),
                    energy=rng.choice((0.030, 0.060, 0.080, 0.140, 0.511)), tle=rng.random() < 0.3,
                    tracking=rng.random() < 0.3)
    if kind == "projection":
        return dict(kind=kind, n=log_int(32, 256), voxel=rng.choice((0.8, 1.0, 1.9, 2.0)), ex=rng.randint(60, 600),
                    ey=rng.randint(60, 600), element=rng.choice((0.4, 0.8, 1.1)), primaries=log_int(10_000, 20_000_000),
                    spectrum=rng.random() < 0.7, world=rng.choice((0, 0, 0, rng.randint(20, 120))))
    if kind == "mesh":
        body = rng.randint(2, 6)
        return dict(kind=kind, body=body, inner=max(body - 1, 1), primaries=log_int(10_000, 1_000_000 if body < 4 else 5_000_000),
                    energy=rng.choice((0.060, 0.080, 0.140)), dosel=rng.choice((2.0, 3.0, 5.0)))
    if kind == "jobs":
        jobs = rng.randint(2, 48)
        return dict(kind=kind, jobs=jobs, phantoms=rng.choice((1, jobs)), primaries=log_int(10_000, 1_000_000),
                    side=rng.choice((64, 128, 256)))
    if kind == "labels":
        return dict(kind=kind, nx=log_int(48, 512), ny=log_int(48, 512), nz=log_int(24, 512), met=rng.randint(0, 6),
                    ranges=rng.randint(2, 40))
    if kind == "draw":
        n = log_int(24, 320)
        return dict(kind=kind, nx=n, ny=rng.choice((n, rng.randint(24, 320))), nz=log_int(24, 320),
                    voxel=rng.choice((0.1, 0.5, 1.0)), met=rng.randint(0, 6), shapes=rng.randint(3, 12))
    if kind == "integrals":
        side = rng.choice((64, 100, 128, 256, 333))
        return dict(kind=kind, n=log_int(32, 256), voxel=rng.choice((1.0, 1.5, 2.0)), side=side,
                    count=log_int(1, max(1, min(360, 360 * 256 * 64 // (side * 256)))))
    return dict(kind=kind, mode=rng.choice(("forward", "forward", "gradients", "train")), batch=rng.randint(1, 12),
                side=rng.choice((64, 128, 256)))


# ----------------------------------------------------------------- scenes --
class Tables:
    """One navigator's physics tables (library builder), GGEMS's default binning."""

    def __init__(self, names, bins=220):
        nm = len(names)
        self.a = dict(energy_bins=np.zeros(bins, F), cross_sections=np.zeros(3 * nm * bins, F),
                      rayleigh=np.zeros(101 * bins, F), density=np.zeros(nm, F), cut=np.zeros(nm, F),
                      elements=np.zeros(nm, np.int32), offset=np.zeros(nm, np.int32), z=np.zeros(nm * 32, np.uint8),
                      atoms=np.zeros(nm * 32, F))
        ctype = {F: C.c_float, np.int32: C.c_int32, np.uint8: C.c_uint8}
        p = {k: abi.ptr(v, ctype[v.dtype.type]) for k, v in self.a.items()}
        total = C.c_int32()
        lib.ggems_build_tables.restype = C.c_int
        check(lib.ggems_build_tables(workloads.MATERIALS.encode(), (C.c_char_p * nm)(*[m.encode() for m in names]), nm,
                                     bins, C.c_float(1.0e-3), C.c_float(1.0), (C.c_int * 3)(0, 1, 2), 3, C.c_float(0.1),
                                     *[p[k] for k in ("energy_bins", "cross_sections", "rayleigh", "density", "cut",
                                                      "elements", "offset", "z", "atoms")], C.byref(total)), "tables")
        self.mu_energies, self.mu_en = _mu_en(names)
        self.struct = abi.gg_physics_tables(bins, nm, 3, (C.c_int32 * 3)(0, 1, 2), p["energy_bins"],
                                            p["cross_sections"], p["rayleigh"], p["density"], p["cut"], p["elements"],
                                            p["offset"], p["z"], p["atoms"], total.value,
                                            abi.ptr(self.mu_energies, C.c_float), abi.ptr(self.mu_en, C.c_float))


def _mu_en(names):
    """220-bin mu_en table (cm^-1) of the materials, from their main elements' data."""
    main = {"Air": ((7, 0.77, 8, 0.23), 1.2e-3), "Water": ((1, 0.11, 8, 0.89), 1.0),
            "Bone185": ((8, 0.45, 20, 0.55), 1.85), "GOS": ((8, 0.08, 64, 0.92), 7.3)}
    pd = workloads.load_physics()
    nb, first, rows = pd["mu_nb_energy_bins"], pd["mu_index_energy"], pd["mu_data"].reshape(-1, 3).astype(np.float64)
    e = np.exp(np.linspace(math.log(1.0e-3), 0.0, abi.GG_ATTENUATION_BINS))
    out = []
    for name in names:
        (z1, w1, z2, w2), density = main[name]
        mu = sum(w * np.exp(np.interp(np.log(e), np.log(r[:, 0]), np.log(r[:, 2])))
                 for w, r in ((w, rows[first[z]:first[z] + nb[z]]) for z, w in ((z1, w1), (z2, w2))))
        out.append(mu * density)
    return e.astype(F), np.ascontiguousarray(np.concatenate(out).astype(F))


def _frame(axis, translation=(0.0, 0.0, 0.0), angle=0.0):
    m = np.eye(4)
    m[:3, :3] = axis
    m[:3, 3] = translation
    c, s = math.cos(angle), math.sin(angle)
    r = np.eye(4)
    r[:2, :2] = ((c, -s), (s, c))
    return (r @ m).astype(F)


def _box(solid, matrix, half):
    solid.obb.matrix[:] = [float(v) for v in matrix.reshape(-1)]
    solid.obb.border_min[:] = [-float(h) for h in half]
    solid.obb.border_max[:] = [float(h) for h in half]
    solid.histogram = solid.scatter_histogram = solid.dose_map = -1


@functools.lru_cache(maxsize=4)
def _ellipsoids(n, seed, bones):
    """uint8 labels (z, y, x): 0 air, 1 water ellipsoid, 2 bone inserts, of an n^3 grid."""
    rng = np.random.default_rng(seed)
    dev = "cuda"
    c = (torch.arange(n, device=dev, dtype=torch.float32) + 0.5) * (2.0 / n) - 1.0

    def inside(centre, axes):
        x, y, z = (((c - float(p)) / float(a)) ** 2 for p, a in zip(centre, axes))
        return z[:, None, None] + y[None, :, None] + x[None, None, :] <= 1.0

    body = inside((0, 0, 0), rng.uniform(0.6, 0.95, 3))
    out = body.to(torch.uint8)
    for _ in range(bones):
        out[inside(rng.uniform(-0.45, 0.45, 3), rng.uniform(0.06, 0.22, 3)) & body] = 2
    return np.ascontiguousarray(out.cpu().numpy())


def _voxelized(labels, voxel, navigator):
    n = labels.shape[0]
    s = abi.gg_solid()
    s.type, s.navigator = abi.GG_SOLID_VOXELIZED, navigator
    _box(s, np.eye(4, dtype=F), [F(F(n) * F(voxel)) * F(0.5)] * 3)
    s.number_of_voxels[:] = [n] * 3
    s.voxel_sizes[:] = [float(F(voxel))] * 3
    s.labels = abi.ptr(labels, C.c_uint8)
    return s


def _panel(ex, ey, element, navigator, angle=0.0):
    """Flat panel of ex x ey elements, 10 mm thick, 500 mm behind the isocentre."""
    s = abi.gg_solid()
    s.type, s.navigator, s.threshold = abi.GG_SOLID_BOX, navigator, float(F(0.010))
    size = [F(ex) * F(element), F(ey) * F(element), F(10.0)]
    _box(s, _frame(DETECTOR_AXIS, (500.0, 0.0, 0.0), angle), [v * F(0.5) for v in size])
    s.virtual_element_number[:] = [ex, ey, 1]
    s.box_size[:] = [float(v) for v in size]
    s.histogram, s.scatter_histogram = 0, 1
    return s


def _dose_map(solid, dosel, tracking=False, tle=False):
    d = abi.gg_dose_map()
    d.size_of_dosels[:] = [float(F(dosel))] * 3
    d.inv_size_of_dosels[:] = [float(F(1.0) / F(dosel))] * 3
    d.border_min[:] = list(solid.obb.border_min)
    d.border_max[:] = list(solid.obb.border_max)
    k = [int(F(F(b) - F(a)) / F(dosel)) for a, b in zip(d.border_min, d.border_max)]
    d.number_of_dosels[:] = k
    d.total_number_of_dosels, d.slice_number_of_dosels = k[0] * k[1] * k[2], k[0] * k[1]
    d.record_edep_squared = d.record_hit = 1
    d.record_photon_tracking, d.tle = int(tracking), int(tle)
    solid.dose_map = 0
    return d


class Source:
    """X-ray cone at 1000 mm from the isocentre (mono-energetic or 120 kVp), or
    a voxelized activity in the phantom's frame."""

    def __init__(self, energy=None, aperture=11.0, angle=0.0, activity=None, voxel=1.0):
        e, w = ([energy], [1.0]) if energy else workloads.xray_spectrum()
        cdf = np.concatenate([[0.0], np.cumsum(np.asarray(w, np.float64)) / np.sum(w)]).astype(F)
        cdf[-1] = 1.0
        self.spectrum, self.cdf = np.append(np.asarray(e, F), F(e[-1])), cdf
        s = self.struct = abi.gg_source()
        s.type, s.beam_aperture = abi.GG_SOURCE_XRAY, float(F(aperture * DEG))
        s.matrix[:] = [float(v) for v in _frame(SOURCE_AXIS, (-1000.0, 0.0, 0.0), angle).reshape(-1)]
        s.number_of_energy_bins, s.is_interp = len(e), 0 if energy else 1
        s.energy_spectrum, s.energy_cdf = abi.ptr(self.spectrum, C.c_float), abi.ptr(self.cdf, C.c_float)
        if activity is not None:
            n = activity.shape[0]
            active = np.flatnonzero(activity).astype(np.int32)
            self.index = np.concatenate([[0], active]).astype(np.int32)
            self.index[-1] = self.index[-2]
            cum = np.cumsum(activity.reshape(-1)[active].astype(np.float64))
            self.activity = np.concatenate([[0.0], cum / cum[-1]]).astype(F)
            s.type = abi.GG_SOURCE_VOXELIZED
            s.matrix[:] = [float(v) for v in np.eye(4).reshape(-1)]
            s.number_of_voxels[:] = [n] * 3
            s.voxel_sizes[:] = [float(F(voxel))] * 3
            s.border_min[:] = [float(-F(F(n) * F(voxel)) * F(0.5))] * 3
            s.number_of_activity_bins = len(self.index)
            s.activity_index, s.activity_cdf = abi.ptr(self.index, C.c_int32), abi.ptr(self.activity, C.c_float)


class Transport:
    """A context with a scene uploaded, its host tallies and its random streams seeded."""

    def __init__(self, tables, solids, dose_maps, histogram_sizes, world, seed):
        self.keep = (tables, solids)
        self.t = (abi.gg_physics_tables * len(tables))(*[t.struct for t in tables])
        self.s = (abi.gg_solid * len(solids))(*solids)
        self.d = (abi.gg_dose_map * max(1, len(dose_maps)))(*dose_maps)
        self.h = np.array(list(histogram_sizes) + [0], np.int32)
        pd = workloads.load_physics()
        self.fit = np.ascontiguousarray(np.stack([pd["rayleigh_pp%d" % i] for i in range(9)]).astype(F))
        self.world, cells = None, 0
        if world:
            w = self.world = abi.gg_world()
            w.dimensions[:] = [world] * 3
            w.sizes[:] = [float(F(2400.0 / world))] * 3
            w.photon_tracking = w.energy_tracking = w.energy_squared_tracking = w.momentum = 1
            cells = world ** 3
        self.scene = abi.gg_scene(len(tables), self.t, len(solids), self.s, len(dose_maps), self.d,
                                  len(histogram_sizes), abi.ptr(self.h, C.c_int32), abi.ptr(self.fit, C.c_float),
                                  C.pointer(self.world) if world else C.cast(None, C.POINTER(abi.gg_world)))
        self.ctx = Context(0)
        self.ctx.upload_scene(self.scene)
        states = np.zeros(5 * SLOTS, np.uint32)
        check(lib.gg_seed_random_states(abi.ptr(states, C.c_uint32), SLOTS, seed & 0x7FFFFFFF, 0), "seeding")
        self.ctx.set_random_states(states)
        self.tallies = abi.Tallies(histogram_sizes, [d.total_number_of_dosels for d in dose_maps], cells)


@functools.lru_cache(maxsize=4)
def _icosphere(subdivisions):
    return workloads.icosphere(subdivisions)


def _mesh(body, inner, seed):
    """Body ellipsoid with eight inner ellipsoids as a meshed solid (library builder, octree depth 4)."""
    rng = np.random.default_rng(seed)

    def part(axes, centre, subdivisions):
        v, f = _icosphere(subdivisions)
        return (v * np.asarray(axes) + np.asarray(centre))[f].astype(F)

    size = np.array([120.0, 100.0, 150.0])
    parts = [part(size, (0.0, 0.0, 0.0), body)]
    for _ in range(8):
        axes = rng.uniform(10.0, 30.0, 3)
        parts.append(part(axes, rng.uniform(-0.45, 0.45, 3) * size, inner))
    with tempfile.TemporaryDirectory() as tmp:
        path = os.path.join(tmp, "body.stl")
        workloads.write_stl(path, np.concatenate(parts))
        eye = np.eye(4, dtype=F)
        nt, nn = C.c_int32(), C.c_int32()
        f = lib.ggems_build_mesh
        f.restype = C.c_int
        head = (path.encode(), abi.ptr(eye, C.c_float), 4, C.byref(nt), C.byref(nn))
        check(f(*head, None, None, None, None, None, None), "mesh")
        tri, nodes = np.zeros(nt.value * abi.GG_TRIANGLE_FLOATS, F), np.zeros(nn.value * 6, F)
        first, order = np.zeros(nn.value + 1, np.int32), np.zeros(nt.value, np.int32)
        lo, hi = np.zeros(3, F), np.zeros(3, F)
        check(f(*head, *[abi.ptr(a, C.c_float) for a in (tri, nodes)], *[abi.ptr(a, C.c_int32) for a in (first, order)],
                *[abi.ptr(a, C.c_float) for a in (lo, hi)]), "mesh")
    s = abi.gg_solid()
    s.type, s.navigator = abi.GG_SOLID_MESHED, 0
    _box(s, eye, (0.0, 0.0, 0.0))
    s.obb.border_min[:] = [float(v) for v in lo]
    s.obb.border_max[:] = [float(v) for v in hi]
    s.number_of_triangles, s.number_of_nodes = nt.value, nn.value
    s.triangles, s.nodes = abi.ptr(tri, C.c_float), abi.ptr(nodes, C.c_float)
    s.node_first, s.node_triangles = abi.ptr(first, C.c_int32), abi.ptr(order, C.c_int32)
    return s, (tri, nodes, first, order)


# ---------------------------------------------------------------- prepare --
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_dose(case, seed):
    n, voxel = case["n"], case["voxel"]
    labels = _ellipsoids(n, seed, 4) if case["source"] == "voxelized" else np.ones((n, n, n), np.uint8)
    solid = _voxelized(labels, voxel, 0)
    dose = _dose_map(solid, voxel, case["tracking"], case["tle"])
    if case["source"] == "voxelized":
        rng = np.random.default_rng(seed + 1)
        activity = np.where(labels == 2, rng.uniform(0.5, 4.0, labels.shape), 0.0).astype(F)
        activity[n // 2, n // 2, n // 2 - 1:n // 2 + 1] = 1.0
        src = Source(case["energy"], activity=activity, voxel=voxel)
    else:
        src = Source(case["energy"], aperture=10.0)
    t = Transport([Tables(["Air", "Water", "Bone185"])], [solid], [dose], [], 0, seed)
    return dict(kind="dose", t=t, src=src, n=case["primaries"], dosels=dose.total_number_of_dosels,
                tracking=case["tracking"], keep=labels)


def _prepare_projection(case, seed):
    labels = _ellipsoids(case["n"], seed, 9)
    solids = [_voxelized(labels, case["voxel"], 0), _panel(case["ex"], case["ey"], case["element"], 1)]
    src = Source(None if case["spectrum"] else 0.060)
    pixels = case["ex"] * case["ey"]
    t = Transport([Tables(["Air", "Water", "Bone185"]), Tables(["GOS"])], solids, [], [pixels, pixels], case["world"],
                  seed)
    return dict(kind="projection", t=t, src=src, n=case["primaries"], keep=labels)


def _prepare_mesh(case, seed):
    solid, keep = _mesh(case["body"], case["inner"], seed)
    dose = _dose_map(solid, case["dosel"])
    t = Transport([Tables(["Water"])], [solid], [dose], [], 0, seed)
    return dict(kind="dose", t=t, src=Source(case["energy"], aperture=8.0), n=case["primaries"],
                dosels=dose.total_number_of_dosels, tracking=False, keep=keep)


def _prepare_jobs(case, seed):
    rng = np.random.default_rng(seed)
    side, count = case["side"], case["jobs"]
    phantoms = [_ellipsoids(64, seed + k, 4) for k in range(case["phantoms"])]
    tables = [Tables(["Air", "Water", "Bone185"]), Tables(["GOS"])]
    base = [_voxelized(phantoms[0], 2.0, 0), _panel(side, side, 256.0 / side, 1)]
    t = Transport(tables, base, [], [side * side] * (2 * count), 0, seed)
    jobs, keep = [], [phantoms]
    for k, angle in enumerate(np.sort(rng.uniform(0.0, 2.0 * math.pi, count))):
        panel = _panel(side, side, 256.0 / side, 1, float(angle))
        panel.histogram, panel.scatter_histogram = 2 * k, 2 * k + 1
        solids = (abi.gg_solid * 2)(_voxelized(phantoms[k % len(phantoms)], 2.0, 0), panel)
        src = Source(0.060, aperture=10.0, angle=float(angle))
        keep.append((src, solids))
        jobs.append((src.struct, case["primaries"], solids))
    return dict(kind="jobs", t=t, jobs=jobs, keep=keep)


def _prepare_labels(case, seed):
    dtype = np.dtype(abi.MET_DTYPES[case["met"]])
    dims = (case["nx"], case["ny"], case["nz"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    # a CT-like image: air, soft tissue and bone values around their means, in the type's range
    lo, hi = (-1000.0, 2000.0) if dtype.kind == "f" or (dtype.kind == "i" and dtype.itemsize > 1) else (0.0, 120.0)
    n = dims[0] * dims[1] * dims[2]
    mode = torch.randint(0, 4, (n // 64 + 1,), generator=g, device="cuda").repeat_interleave(64)[:n]
    image = lo + (hi - lo) * torch.tensor([0.02, 0.33, 0.36, 0.7], device="cuda")[mode]
    image += 0.02 * (hi - lo) * torch.randn(n, generator=g, device="cuda")
    image = image.clamp_(lo, hi).cpu().numpy().astype(dtype)
    edges = np.linspace(lo, hi, case["ranges"] + 1).astype(F)
    return dict(kind="labels", volume=Volume(case["met"], dims, (1.0, 1.0, 1.0)), image=image, first=edges[:-1].copy(),
                last=edges[1:].copy())


def _prepare_draw(case, seed):
    rng = np.random.default_rng(seed)
    extent = np.array([case["nx"], case["ny"], case["nz"]]) * case["voxel"]
    shapes = []
    for k in range(case["shapes"]):
        s = abi.gg_shape()
        s.type = k % 3
        wide = k == 0
        shift = 0.08 if wide else 0.3
        s.position[:] = [float(F(v)) for v in rng.uniform(-shift, shift, 3) * extent]
        size = rng.uniform(0.6, 0.9, 3) * extent if wide else rng.uniform(0.1, 0.35, 3) * extent
        s.size[:] = [float(F(v)) for v in size]
        s.label_value = float(k + 1)
        shapes.append(s)
    dims = (case["nx"], case["ny"], case["nz"])
    return dict(kind="draw", volume=Volume(case["met"], dims, (case["voxel"],) * 3), shapes=shapes)


def _integral_geometry(case, seed):
    rng = np.random.default_rng(seed)
    labels = _ellipsoids(case["n"], seed, 4)
    # attenuation of air, water and bone around 60 keV, mm^-1
    mu = (np.array([2.4e-5, 0.0206, 0.058]) * rng.uniform(0.95, 1.05, 3)).astype(F)
    angles = np.sort(rng.uniform(0.0, 2.0 * math.pi, case["count"]))
    side = case["side"]
    panels = [_panel(side, side, 256.0 / side, 1, float(a)) for a in angles]
    sources = np.ascontiguousarray(np.stack([_frame(SOURCE_AXIS, (-1000.0, 0.0, 0.0), a)[:3, 3] for a in angles]))
    return labels, mu, panels, sources


def _prepare_integrals(case, seed):
    labels, mu, panels, sources = _integral_geometry(case, seed)
    side, count = case["side"], case["count"]
    return dict(kind="integrals", ctx=Context(0), lib=scatter._lib(), solid=_voxelized(labels, case["voxel"], 0),
                panels=(abi.gg_solid * count)(*panels), sources=sources, mu=mu, count=count, side=side, keep=labels)


def _unet_arrays(case, seed):
    """(parameters, input, target) on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    parts = []
    for cin, cout, _ in scatter.LAYERS:
        fan = 9 * (10 if cin == 16 else cin)
        w = torch.randn((9, cout, cin), generator=g, device="cuda") * math.sqrt(2.0 / fan)
        if cin == 16:
            w[:, :, 10:] = 0.0
        parts += [w.reshape(-1), 0.05 * torch.randn(cout, generator=g, device="cuda")]
    parts += [torch.randn(32, generator=g, device="cuda") * math.sqrt(1.0 / 32.0), torch.zeros(1, device="cuda")]
    b, s = case["batch"], case["side"]
    # smooth line-integral maps with some noise, as phantom shadows have
    y, x = torch.meshgrid(*[torch.linspace(-1, 1, s, device="cuda")] * 2, indexing="ij")
    a = torch.rand((b, 1, 1), generator=g, device="cuda") * 0.5 + 0.4
    shadow = 4.0 * torch.sqrt(torch.clamp(1.0 - (x / a) ** 2 - (y / 0.8) ** 2, min=0.0))
    integral = shadow * (1.0 + 0.05 * torch.randn((b, s, s), generator=g, device="cuda"))
    inputs = torch.stack([torch.exp(-integral), integral], -1).contiguous()
    target = 0.5 + 0.3 * shadow + 0.05 * torch.randn((b, s, s), generator=g, device="cuda")
    return torch.cat(parts), inputs, target.contiguous()


def _prepare_unet(case, seed):
    p, x, t = _unet_arrays(case, seed)
    net = scatter.UNet(case["batch"], case["side"], seed=1)
    net.set_parameters(p.cpu().numpy())
    return dict(kind="unet", mode=case["mode"], net=net, x=x, t=t)


# -------------------------------------------------------------------- run --
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_dose(s):
    ctx, ta = s["t"].ctx, s["t"].tallies
    ctx.reset_tallies()
    ctx.run(s["src"].struct, s["n"])
    ctx.read_tallies(ta)
    dose, uncertainty = ctx.compute_dose(0, 0, s["dosels"])
    out = dict(edep=ta.edep[0], edep_squared=ta.edep_squared[0], hit=ta.hit[0], dose=dose, uncertainty=uncertainty)
    if s["tracking"]:
        out["photon_tracking"] = ta.photon_tracking[0]
    return out


def _run_projection(s):
    ctx, ta = s["t"].ctx, s["t"].tallies
    ctx.reset_tallies()
    ctx.run(s["src"].struct, s["n"])
    ctx.read_tallies(ta)
    return dict(total=ta.histograms[0], scatter=ta.histograms[1], **(ta.world or {}))


def _run_jobs(s):
    ctx, ta = s["t"].ctx, s["t"].tallies
    ctx.reset_tallies()
    ctx.run_jobs(s["jobs"])
    ctx.synchronize()
    ctx.read_tallies(ta)
    return [np.concatenate(ta.histograms[0::2]), np.concatenate(ta.histograms[1::2])]


def _run_labels(s):
    s["volume"].upload(s["image"])
    return list(s["volume"].labels(s["first"], s["last"]))


def _run_draw(s):
    s["volume"].draw(s["shapes"])
    return s["volume"].download()


def _run_integrals(s):
    out = torch.empty((s["count"], s["side"], s["side"], 2), dtype=torch.float32, device="cuda")
    check(s["lib"].gg_line_integrals_batch(s["ctx"].handle, C.byref(s["solid"]), s["panels"],
                                           abi.ptr(s["sources"], C.c_float), s["count"], abi.ptr(s["mu"], C.c_float), 3,
                                           C.cast(C.c_void_p(out.data_ptr()), C.POINTER(C.c_float))), "line integrals")
    return out


def _run_unet(s):
    net = s["net"]
    if s["mode"] == "forward":
        return net.forward(s["x"])
    if s["mode"] == "gradients":
        loss, grads = net.gradients(s["x"], s["t"])
        return dict(loss=loss, gradients=grads)
    loss = net.train_step(s["x"], s["t"], 1e-3)
    return dict(loss=loss, parameters=net.parameters())


# ------------------------------------------------------------ work, limits --
def work(case):
    """Bytes and operations of a pass.  Transport: the random streams in and
    out, the final particles, the labels once and the tallies out, and about
    100 operations a voxel step (three uniform draws, logarithms and divisions,
    the slab test, the voxel index)."""
    k = case["kind"]
    if k in ("dose", "projection", "mesh", "jobs"):
        runs = case.get("jobs", 1)
        slots = min(case["primaries"], SLOTS)
        bytes_ = slots * 80.0
        if k == "dose":
            n = case["n"]
            steps = 0.8 * n if case["source"] == "xray" else 0.4 * n
            bytes_ += n ** 3 * (1 + 28 + 8)
        elif k == "projection":
            steps = 0.6 * case["n"] + 3
            bytes_ += case["n"] ** 3 + 8.0 * case["ex"] * case["ey"] + 44.0 * case["world"] ** 3
        elif k == "mesh":
            # two nodes a level and the triangles of two crossed surfaces for each of about 6 steps
            triangles = 20 * 4 ** case["body"] + 160 * 4 ** case["inner"]
            steps = 6 * (0.5 * math.log2(triangles) + 2)
            bytes_ += 48.0 * triangles + 28 * (300 / case["dosel"]) ** 3
        else:
            steps = 50.0
            bytes_ += case["phantoms"] * 64.0 ** 3 + runs * 8.0 * case["side"] ** 2
        return dict(bytes=bytes_, flops=100.0 * steps * case["primaries"] * runs)
    if k in ("labels", "draw"):
        n = float(case["nx"] * case["ny"] * case["nz"])
        size = np.dtype(abi.MET_DTYPES[case["met"]]).itemsize
        if k == "labels":
            return dict(bytes=n * (size + 1), flops=n * 2 * math.log2(case["ranges"] + 1))
        return dict(bytes=n * size, flops=0.2 * n * 12 * case["shapes"])
    if k == "integrals":
        rays = float(case["count"] * case["side"] ** 2)
        return dict(bytes=rays * 8 + case["n"] ** 3, flops=rays * 1.5 * case["n"] * 6)
    pixels = float(case["batch"] * case["side"] ** 2)
    flops = float(scatter.forward_flops(case["side"], case["batch"]))
    weights = float(sum(9 * i * o + o for i, o, _ in scatter.LAYERS) + 33)
    if case["mode"] == "forward":
        return dict(bytes=12 * pixels + 2 * weights, flops=flops)
    # activations of every layer written in the forward pass and read in the backward pass, BF16
    acts = sum(2.0 * o * pixels / d ** 2 for _, o, d in scatter.LAYERS)
    return dict(bytes=16 * pixels + 2 * acts + (32 if case["mode"] == "train" else 8) * weights, flops=3 * flops)


def tolerance(case):
    """Whole numbers (counts, labels, drawn images) are the same whatever the
    order of the histories; energy tallies are fixed point, so they are too;
    squared energies are FP64 atomics in any order."""
    k = case["kind"]
    if k in ("dose", "mesh") or (k == "projection" and case["world"]):
        return dict(rel=1e-9, max=1e-6)
    if k in ("projection", "jobs", "labels", "draw"):
        return "exact"
    if k == "integrals":
        return dict(rel=1e-4, max=1e-2)  # FP32 walk: 1e-5 to 3e-5 from the 64-bit chords
    if case["mode"] == "forward":
        return dict(rel=1e-2)
    if case["mode"] == "gradients":
        return dict(rel=2e-2)
    return dict(rel=5e-3, max=0.5)


# ------------------------------------------------------------------ exact --
def exact(case, seed):
    if case["kind"] == "integrals":
        return _exact_integrals(case, seed)
    if case["kind"] == "unet":
        return _exact_unet(case, seed)
    return None  # random walks have no closed form; labels and images are whole numbers


def _exact_integrals(case, seed):
    """Chord lengths between a ray's sorted plane crossings, times mu of the
    voxel at each chord's middle, in 64 bits."""
    labels, mu, panels, sources = _integral_geometry(case, seed)
    n, side, half = case["n"], case["side"], float(F(F(case["n"]) * F(case["voxel"])) * F(0.5))
    if case["count"] * side * side * 3.0 * n > 6e9:
        return None
    dev = dict(device="cuda", dtype=torch.float64)
    mu_of = torch.tensor(mu.astype(np.float64), **dev)[torch.from_numpy(labels).cuda().long()].reshape(-1)
    planes = torch.arange(n + 1, **dev) * float(F(case["voxel"])) - half
    out = torch.empty((case["count"], side, side, 2), **dev)
    for k, panel in enumerate(panels):
        m = torch.tensor(np.array(list(panel.obb.matrix), np.float64).reshape(4, 4), **dev)
        es = float(F(panel.box_size[0]) / F(side))
        c = panel.obb.border_min[0] + (torch.arange(side, **dev) + 0.5) * es
        y, x = torch.meshgrid(c, c, indexing="ij")
        end = x.reshape(-1, 1) * m[:3, 0] + y.reshape(-1, 1) * m[:3, 1] + m[:3, 3]
        start = torch.tensor(sources[k].astype(np.float64), **dev)
        for r in range(0, side * side, 1 << 16):
            d = end[r:r + (1 << 16)] - start
            t = torch.cat([(planes - start[a]) / d[:, a:a + 1] for a in range(3)], 1)
            t = torch.nan_to_num(t, nan=0.0, posinf=1.0, neginf=0.0).clamp_(0.0, 1.0).sort(1).values
            mid = 0.5 * (t[:, 1:] + t[:, :-1])
            flat, inside = torch.zeros_like(mid, dtype=torch.long), torch.ones_like(mid, dtype=torch.bool)
            for a, stride in ((0, 1), (1, n), (2, n * n)):
                i = torch.floor((start[a] + mid * d[:, a:a + 1] + half) / float(F(case["voxel"]))).long()
                inside &= (i >= 0) & (i < n)
                flat += i.clamp_(0, n - 1) * stride
            length = (t[:, 1:] - t[:, :-1]) * d.norm(dim=1, keepdim=True)
            line = (mu_of[flat] * length * inside).sum(1)
            out[k].reshape(-1, 2)[r:r + (1 << 16)] = torch.stack([torch.exp(-line), line], 1)
    return out


def _exact_unet(case, seed):
    """The network, its loss and its gradients with FP64 weights and activations."""
    p, x, t = _unet_arrays(case, seed)
    p, x, t = p.double().requires_grad_(case["mode"] != "forward"), x.double(), t.double()
    s, conv, pool = case["side"], torch.nn.functional.conv2d, torch.nn.functional.avg_pool2d
    maps = x.permute(0, 3, 1, 2)
    ch = [maps[:, 0:1], maps[:, 1:2]]
    for m in (0, 1):
        for r in (4, 16, 64):
            sums = torch.nn.functional.pad(maps[:, m:m + 1], (r + 1, r, r + 1, r)).cumsum(2).cumsum(3)
            w = 2 * r + 1
            ch.append((sums[..., w:, w:] - sums[..., :-w, w:] - sums[..., w:, :-w] + sums[..., :-w, :-w]) / w ** 2)
    ch += [maps[:, m:m + 1].mean((2, 3), keepdim=True).expand(-1, 1, s, s) for m in (0, 1)]
    act, off, skips = torch.cat(ch + [torch.zeros_like(maps[:, :1])] * 6, 1), 0, {}
    for i, (cin, cout, _) in enumerate(scatter.LAYERS):
        w = p[off:off + 9 * cin * cout].reshape(3, 3, cout, cin).permute(2, 3, 0, 1)
        off += 9 * cin * cout
        if i in (2, 4, 6):
            skips[i] = act
            act = pool(act, 2)
        if i in (8, 10, 12):
            up = act.repeat_interleave(2, 2).repeat_interleave(2, 3)
            act = torch.cat([up, skips[14 - i]], 1)
        act = torch.relu(conv(act, w, p[off:off + cout], padding=1))
        off += cout
    y = torch.einsum("bchw,c->bhw", act, p[off:off + 32]) + p[off + 32]
    if case["mode"] == "forward":
        return y.detach()
    loss = ((y - t) ** 2).mean()
    loss.backward()
    g = p.grad
    if case["mode"] == "gradients":
        return dict(loss=float(loss), gradients=g)
    # the first Adam step: m / c1 = g, v / c2 = g^2
    return dict(loss=float(loss), parameters=p.detach() - 1e-3 * g / (g.abs() + 1e-8))
