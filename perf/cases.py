"""The work that programs have this framework do, as cases that can be timed one by one.

A case is a dict of plain values. `listed()` names the usual ones, `draw(rng)` gives another one of the same
ranges, `prepare(case, seed)` makes what a program holds before the call (on the GPU, from the seed alone),
`run(state)` is one pass through the public entry points, `work(case)` the bytes and operations that the pass
cannot do without, and `exact(case, seed)` the same outputs in 64 bits where they have such a value.

Kinds of work:
  frame    Simulation.step_frame: one frame of one tank that is already running
  tanks    step_frames: one frame of many independent tanks
  sort     sort_particles_static: the spatial sort of a caller's particle records
  surface  Simulation.build_surface: the density field and the surface-nets mesh of a tank's particles
  train    WarmStartNet.train_step: one step of the learned warm start's training
"""
import ctypes
import math

import numpy as np
import torch

import slosh_b200 as S
from slosh_b200 import _abi as A
from slosh_b200 import scenes, warmstart

# The preconditioner that the benchmark runs with (the library's defaults are the reference's V-cycle).
TUNED = {"mg_correction_scale": 1.9, "mg_smoothing_sweeps": 2, "mg_coarse_iterations": 4, "mg_smoother_weight": 1.15}
PRECISION = {"fp32": A.PRECISION_FP32, "fp16": A.PRECISION_FP16_STORAGE, "bf16": A.PRECISION_BF16_STORAGE}


def _frame(name, grid, scene, **options):
    """A frame case: the options that a case does not give are the library's defaults, one substep per frame."""
    case = {"name": name, "kind": "frame", "nx": grid[0], "ny": grid[1], "nz": grid[2], "scene": scene, "fill_x": 0.4, "fill_y": 0.5,
            "transfer": "apic", "solver": "mgpcg", "iterations": 8, "tolerance": 0.0, "tuned": False, "precision": "fp32",
            "viscosity": 0.0, "colliders": 0, "fields": False, "emitter": 0, "substeps": 1, "rate": 120, "sort_interval": 4}
    case.update(options)
    return case


def listed():
    return [
        # A tool or a small effect that sorts a few thousand records of its own: launches and latency only.
        {"name": "sort_3k", "kind": "sort", "count": 3001, "nx": 24, "ny": 24, "nz": 18, "dead": 0.02},
        # The largest snapshots that the allocation-free sort takes (262,144 records).
        {"name": "sort_200k", "kind": "sort", "count": 200_003, "nx": 64, "ny": 64, "nz": 48, "dead": 0.02},
        # The plugin's default volume with its default settings: the smallest tank that is stepped every frame.
        _frame("tank_64x64x48", (64, 64, 48), "dam", fill_x=0.4, fill_y=0.4, substeps=1, rate=60),
        # The size that the reference quotes its substep on, 4 PCG iterations, two substeps a frame.
        _frame("tank_128x128x96", (128, 128, 96), "dam", fill_x=0.4, fill_y=0.35, iterations=4, substeps=2),
        # A viscous liquid in PIC/FLIP with the other pressure solver, moved by colliders and force fields and fed
        # by an emitter, at the second size that the reference quotes.
        _frame("viscous_flip_96x96x72", (96, 96, 72), "dam", fill_x=0.45, fill_y=0.35, transfer="flip", solver="rbgs", iterations=60,
               viscosity=2e-4, colliders=3, fields=True, emitter=400),
        # The benchmark's scene at 192^3 with red-black SOR to a tight residual.
        _frame("rbgs_192", (192, 192, 192), "dam_sphere", solver="rbgs", iterations=200, substeps=1, rate=480),
        # Several pools and static spheres, an elongated domain, 16-bit storage of the coarse levels.
        _frame("boxes_256x128x128_bf16", (256, 128, 128), "boxes", tolerance=1e-6, tuned=True, precision="bf16", colliders=3, rate=240),
        # The benchmark's scene: 20.6 million particles, MGPCG to 1e-6. The largest case.
        _frame("dam_break_sphere_256", (256, 256, 256), "dam_sphere", tolerance=1e-6, tuned=True, rate=480),
        # A level with many small tanks, stepped together.
        {"name": "tanks_24", "kind": "tanks", "tanks": 24, "lo": 32, "hi": 96, "tolerance": 1e-6},
        # The mesh of the small tank, every frame.
        {"name": "surface_64x64x48", "kind": "surface", "nx": 64, "ny": 64, "nz": 48, "fill": 0.45, "resolution": 1.0, "smoothing": 2.0,
         "mesh": True},
        # The mesh of a large tank.
        {"name": "surface_160", "kind": "surface", "nx": 160, "ny": 160, "nz": 160, "fill": 0.25, "resolution": 1.0, "smoothing": 2.0,
         "mesh": True},
        # Training of the learned warm start: forward, backward and Adam (weights and activations in BF16).
        {"name": "train_64_batch2", "kind": "train", "nx": 64, "ny": 64, "nz": 64, "batch": 2},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "tanks", "sort", "surface", "train"])
    if kind == "frame":
        grid = tuple(_size(rng, 28, 200) for _ in range(3))
        scene = rng.choice(["dam", "dam", "dam_sphere", "boxes"])
        solver = rng.choice(["mgpcg", "mgpcg", "rbgs"])
        tolerance = rng.choice([0.0, 1e-6]) if solver == "mgpcg" else 0.0
        case = _frame("", grid, scene, fill_x=round(rng.uniform(0.2, 0.5), 3), fill_y=round(rng.uniform(0.2, 0.5), 3),
                      transfer=rng.choice(["apic", "apic", "flip"]), solver=solver,
                      iterations=rng.randint(4, 16) if solver == "mgpcg" else rng.randint(30, 80), tolerance=tolerance,
                      tuned=rng.random() < 0.5, precision=rng.choice(["fp32", "fp32", "fp16", "bf16"]),
                      viscosity=rng.choice([0.0, 0.0, 1e-4, 5e-4]), colliders=rng.randint(0, 4), fields=rng.random() < 0.25,
                      emitter=rng.choice([0, 0, 50, 1000]), substeps=rng.randint(1, 3), rate=rng.choice([60, 120, 240]),
                      sort_interval=rng.choice([1, 4, 4, 8]))
        del case["name"]
        return case
    if kind == "tanks":
        return {"kind": "tanks", "tanks": rng.randint(2, 32), "lo": rng.randint(24, 48), "hi": rng.randint(56, 112),
                "tolerance": rng.choice([0.0, 1e-6])}
    if kind == "sort":
        return {"kind": "sort", "count": _size(rng, 500, 262_144), "nx": _size(rng, 16, 200), "ny": _size(rng, 16, 200),
                "nz": _size(rng, 16, 200), "dead": rng.choice([0.0, 0.02, 0.3])}
    if kind == "surface":
        return {"kind": "surface", "nx": _size(rng, 24, 160), "ny": _size(rng, 24, 160), "nz": _size(rng, 24, 160),
                "fill": round(rng.uniform(0.1, 0.25), 3), "resolution": rng.choice([0.5, 1.0, 1.0, 1.5]),
                "smoothing": rng.choice([1.0, 2.0, 3.0]), "mesh": rng.random() < 0.8}
    return {"kind": "train", "nx": rng.choice([32, 64, 128]), "ny": rng.choice([32, 64]), "nz": 64, "batch": rng.randint(1, 3)}


# ---- device memory of the library as tensors ------------------------------------------------------------------
class _Memory:
    """A range of the library's device memory, for torch.as_tensor; keeps its owner alive."""

    def __init__(self, ptr, shape, typestr, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": typestr, "strides": None, "version": 3}


def _device(ptr, shape, typestr, owner):
    if not ptr or 0 in shape:
        return torch.empty(tuple(shape), dtype={"<f4": torch.float32, "<f2": torch.float16, "<i4": torch.int32}[typestr], device="cuda")
    return torch.as_tensor(_Memory(ptr, shape, typestr, owner), device="cuda")


def _particles(sim):
    """The tank's particle records: position, age and velocity in float32, the nine APIC terms in float16."""
    ptr, n = sim.particle_device_ptr()
    rec = _device(ptr, (n, 12), "<f4", sim)
    return {"pos_age_vel": rec[:, :7], "affine": rec.view(torch.float16)[:, 14:23]}


# ---- frame ------------------------------------------------------------------------------------------------------
def _collider(rng, extent, kind, two_way):
    c = A.Collider()
    c.type = kind
    c.center[:] = [float(rng.uniform(0.3, 0.7) * e) for e in extent]
    r = float(rng.uniform(0.05, 0.1) * min(extent))
    c.extent[:] = [r, r * 1.5, r * 0.8]
    c.rotation[:] = [0.0, 0.0, math.sin(0.2), math.cos(0.2)]
    c.flags = 1 if two_way else 0
    c.linear_velocity[:] = [float(v) for v in rng.uniform(-0.2, 0.2, 3)] if two_way else [0.0, 0.0, 0.0]
    return c


def _field(kind, shape, center, radius, axis, strength):
    f = A.Manipulator()
    f.kind, f.shape = kind, shape
    f.center[:] = [float(v) for v in center]
    f.rotation[:] = [0.0, 0.0, 0.0, 1.0]
    f.extent[:] = [radius, radius, radius]
    f.axis[:] = [float(v) for v in axis]
    f.strength, f.falloff = strength, radius
    return f


def _frame_parts(case, seed):
    """(settings, first frame's emissions, per-frame input) of a frame case."""
    rng = np.random.default_rng(seed)
    grid = (case["nx"], case["ny"], case["nz"])
    h = 1.0 / max(grid)
    if case["scene"] == "dam_sphere":  # block and falling sphere, as in scenes.dam_break_sphere
        mn, dims = scenes.box_cells(grid, (0.0, 0.0, 0.0), (0.3, 0.5, 1.0))
        emits = [scenes.fill_cells(mn, dims)] + scenes.sphere_rows(grid, (0.7, 0.75, 0.5), 0.12, velocity=(0.0, -2.0, 0.0))
    elif case["scene"] == "boxes":  # pools apart from one another
        emits = []
        for lo, hi in (((0.0, 0.0, 0.0), (0.22, 0.4, 1.0)), ((0.3, 0.1, 0.1), (0.55, 0.45, 0.5)), ((0.6, 0.0, 0.3), (0.72, 0.9, 0.6)),
                       ((0.8, 0.3, 0.0), (1.0, 0.5, 0.7))):
            mn, dims = scenes.box_cells(grid, lo, hi)
            emits.append(scenes.fill_cells(mn, dims))
    else:
        mn, dims = scenes.box_cells(grid, (0.0, 0.0, 0.0), (case["fill_x"], case["fill_y"], 1.0))
        emits = [scenes.fill_cells(mn, dims)]
    count = sum(e.cell_dims[0] * e.cell_dims[1] * e.cell_dims[2] * 8 for e in emits)
    s = S.settings_default()
    s.grid_dim[:] = list(grid)
    s.cell_size = h
    s.particle_capacity = count + (count // 16 + 4096 if case["emitter"] else 0)
    s.gravity[:] = [0.0, -9.81, 0.0]
    s.transfer_mode = A.TRANSFER_APIC if case["transfer"] == "apic" else A.TRANSFER_FLIP
    s.pressure_solver = A.SOLVER_MGPCG if case["solver"] == "mgpcg" else A.SOLVER_RBGS
    s.pcg_iterations = s.pressure_iterations = case["iterations"]
    s.sor_weight = 1.9 if case["solver"] == "rbgs" else s.sor_weight
    s.tolerance, s.max_iterations = case["tolerance"], 200
    s.precision_mode = PRECISION[case["precision"]]
    s.pcg_flexible = 0 if case["precision"] == "fp32" else 1
    s.kinematic_viscosity = case["viscosity"]
    s.min_substeps = s.max_substeps = case["substeps"]
    s.max_frame_dt = 1.0 / 60.0
    s.sort_interval = case["sort_interval"]
    if case["tuned"]:
        for k, v in TUNED.items():
            setattr(s, k, v)
    extent = [g * h for g in grid]
    colliders = [_collider(rng, extent, (A.COLLIDER_SPHERE, A.COLLIDER_BOX, A.COLLIDER_CAPSULE)[k % 3], k % 2 == 0)
                 for k in range(case["colliders"])]
    fields, each = [], []
    if case["fields"]:
        fields = [_field(A.MANIP_SWIRL, A.SHAPE_CAPSULE, [0.5 * e for e in extent], 0.3 * extent[0], (0.0, 1.0, 0.0), 6.0),
                  _field(A.MANIP_DIRECTIONAL, A.SHAPE_BOX, [0.25 * e for e in extent], 0.2 * extent[0], (1.0, 0.0, 0.0), 3.0),
                  _field(A.MANIP_DRAIN, A.SHAPE_SPHERE, [0.9 * e for e in extent], 0.05 * extent[0], (0.0, 1.0, 0.0), 1.0)]
    if case["emitter"]:
        e = A.EmitRequest()
        e.shape, e.count = A.EMIT_SPHERE, case["emitter"]
        e.center[:] = [0.3 * extent[0], 0.8 * extent[1], 0.5 * extent[2]]
        e.extent[:] = [0.05 * extent[0], 0.0, 0.0]
        e.velocity[:] = [1.0, -1.0, 0.0]
        e.rotation[:] = [0.0, 0.0, 0.0, 1.0]
        e.velocity_spread, e.speed_jitter = 0.2, 0.1
        each = [e]
    fi = A.frame_input(s, emits=each, colliders=colliders, manipulators=fields, delta_time=1.0 / case["rate"])
    return s, emits, fi


def _prepare_frame(case, seed):
    s, emits, fi = _frame_parts(case, seed)
    sim = S.Simulation(s)
    sim.set_emit_seed(1 + seed % (1 << 30))
    sim.step_frame(A.frame_input(s, emits=emits, delta_time=1.0 / case["rate"]))
    for _ in range(3):  # a running tank: sorted once, a pressure to start from
        sim.step_frame(fi)
    return {"kind": "frame", "sim": sim, "input": fi}


def _prepare_tanks(case, seed):
    batch = scenes.tank_batch(S.settings_default, count=case["tanks"], seed=3, lo=case["lo"], hi=case["hi"], tolerance=case["tolerance"])
    sims, inputs, first = [], [], []
    for k, t in enumerate(batch):
        s = t["settings"]
        s.min_substeps = s.max_substeps = 2
        sim = S.Simulation(s)
        sim.set_emit_seed(1 + (seed * 1000 + k) % (1 << 30))
        sims.append(sim)
        first.append(A.frame_input(s, emits=t["emits"]))
        inputs.append(A.frame_input(s))
    S.step_frames(sims, first)
    for _ in range(3):
        S.step_frames(sims, inputs)
    return {"kind": "tanks", "sims": sims, "inputs": inputs}


# ---- particle records of a settled tank ------------------------------------------------------------------------------
def _records(grid, count, seed, dead=0.0, fill=0.4):
    """`count` records (12 words each, on the GPU) in the lower `fill` of the domain, in the order of an earlier sort
    from which half of them have drifted by up to two cells; a share `dead` of them removed."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))

    def uniform(*shape):
        return torch.rand(shape, generator=g, device="cuda")

    n = torch.tensor(grid, dtype=torch.float32, device="cuda")
    u = uniform(count, 3)
    u[:, 1] *= fill * (1.0 + 0.15 * torch.sin(2.0 * math.pi * u[:, 0]) * torch.cos(2.0 * math.pi * u[:, 2]))
    pos = 1.0 + u * (n - 2.0)
    block = (pos / 4.0).long()
    pos = pos[torch.argsort(block[:, 0] + 64 * (block[:, 1] + 64 * block[:, 2]), stable=True)]
    pos += (4.0 * uniform(count, 3) - 2.0) * (uniform(count, 1) < 0.5)
    pos = torch.minimum(pos.clamp(min=1.01), n - 1.01)
    half = (2.0 * torch.randn((count, 10), generator=g, device="cuda")).half()
    half[:, 9] = 0.0
    rec = torch.empty((count, 12), dtype=torch.float32, device="cuda")
    rec[:, 0:3] = pos / float(max(grid))
    rec[:, 3] = 5.0 * uniform(count)
    rec[:, 4:7] = 0.5 * torch.randn((count, 3), generator=g, device="cuda")
    rec[:, 7:12] = half.view(torch.float32)
    if dead:
        rec[uniform(count) < dead, 3] = -1.0
    return rec.view(torch.int32)


def _prepare_sort(case, seed):
    grid = (case["nx"], case["ny"], case["nz"])
    src = _records(grid, case["count"], seed, case["dead"])
    keys = ((grid[0] + 3) // 4) * ((grid[1] + 3) // 4) * ((grid[2] + 3) // 4) + 1
    st = {"kind": "sort", "in": src, "out": torch.empty_like(src), "perm": torch.empty(case["count"], dtype=torch.int32, device="cuda"),
          "offsets": torch.empty(keys, dtype=torch.int32, device="cuda"), "live": torch.zeros(1, dtype=torch.int32, device="cuda"),
          "grid": grid, "count": case["count"], "h": 1.0 / max(grid)}
    return st


# ---- surface ----------------------------------------------------------------------------------------------------------
def _surface_count(case):
    return int(8 * case["nx"] * case["ny"] * case["nz"] * case["fill"])


def _surface_records(case, seed):
    return _records((case["nx"], case["ny"], case["nz"]), _surface_count(case), seed, 0.0, case["fill"])


def _prepare_surface(case, seed):
    rec = _surface_records(case, seed).cpu().numpy().view(S.PARTICLE_DTYPE).reshape(-1)
    s = S.settings_default()
    s.grid_dim[:] = [case["nx"], case["ny"], case["nz"]]
    s.cell_size = 1.0 / max(case["nx"], case["ny"], case["nz"])
    s.particle_capacity = len(rec)
    sim = S.Simulation(s)
    sim.upload_particles(rec)
    sim.sort_particles()  # as the tank's own frames leave them
    q = S.surface_params_default()
    q.field_resolution, q.surface_smoothing, q.build_mesh = case["resolution"], case["smoothing"], 1 if case["mesh"] else 0
    n = [math.ceil(g * case["resolution"]) for g in (case["nx"], case["ny"], case["nz"])]
    q.max_vertices = 6 * (n[0] * n[1] + n[1] * n[2] + n[0] * n[2])
    q.max_indices = 6 * q.max_vertices
    st = {"kind": "surface", "sim": sim, "params": q, "mesh": case["mesh"]}
    for name in ("positions", "normals", "tangents"):  # the program's own vertex and index buffers
        st[name] = torch.zeros((q.max_vertices, 3), device="cuda")
    st["indices"] = torch.zeros(q.max_indices, dtype=torch.int32, device="cuda")
    return st


def _run_surface(st):
    sim = st["sim"]
    info = sim.build_surface(st["params"])
    p = [ctypes.c_void_p() for _ in range(5)]
    S._check(S.load_library().slosh_surface_device_ptrs(sim._ctx, *[ctypes.byref(v) for v in p]))
    nx, ny, nz = info.field_dim
    out = {"field": _device(p[0].value, (nz, ny, nx), "<f2", sim)}
    if st["mesh"]:
        nv, ni = info.num_vertices, info.num_indices
        for name, v in zip(("positions", "normals", "tangents"), p[1:4]):
            st[name][:nv] = _device(v.value, (nv, 3), "<f4", sim)
            out[name] = st[name]
        st["indices"][:ni] = _device(p[4].value, (ni,), "<i4", sim)
        out["indices"] = st["indices"]
        out["counts"] = np.array([info.vertices_requested, info.indices_requested], np.int64)
    return out


def _exact_surface(case, seed):
    """The density field by its definition (Zhu and Bridson's surface of spherical kernels) in float64."""
    grid = (case["nx"], case["ny"], case["nz"])
    h, res = np.float32(1.0 / max(grid)), case["resolution"]
    dim = [int(math.ceil(g * res)) for g in grid]
    reach = case["smoothing"] * 0.6 * res  # kernel radius in voxels (particle_radius_scale 0.6)
    radius, box = 0.6 * res, min(case["smoothing"] * 0.6 * res, 4.0)
    pos = _surface_records(case, seed).view(torch.float32)[:, 0:3].double() * (res / float(h))
    acc = torch.zeros((4, dim[0] * dim[1] * dim[2]), dtype=torch.float64, device="cuda")
    for part in pos.split(1 << 18):
        lo, hi = torch.floor(part - box - 0.5).long(), torch.ceil(part + box - 0.5).long()
        span = int((hi - lo).max()) + 1
        for k in range(span ** 3):
            v = lo + torch.tensor([k % span, (k // span) % span, k // (span * span)], device="cuda")
            ok = (v <= hi).all(1) & (v >= 0).all(1) & (v < torch.tensor(dim, device="cuda")).all(1)
            off = v.double() + 0.5 - part
            q = (off * off).sum(1) / (reach * reach)
            ok &= q < 1.0
            w = (1.0 - q[ok]) ** 3
            at = v[ok, 0] + dim[0] * (v[ok, 1] + dim[1] * v[ok, 2])
            acc[0].index_add_(0, at, w)
            for a in range(3):
                acc[1 + a].index_add_(0, at, -off[ok, a] * w)
    dense = acc[0] > 1e-3
    w = torch.where(dense, acc[0], torch.ones_like(acc[0]))
    phi = (acc[1:] / w).square().sum(0).sqrt() - radius
    field = torch.where(dense, (0.5 - 0.5 * phi / radius).clamp(0.0, 1.0), torch.zeros_like(phi))
    out = {"field": field.reshape(dim[2], dim[1], dim[0]).cpu()}
    if case["mesh"]:  # vertices and quads are numbered by tests on the 16-bit field: no value of their own in 64 bits
        out.update({"positions": None, "normals": None, "tangents": None, "indices": None, "counts": None})
    return out


# ---- training of the warm start ------------------------------------------------------------------------------------
# The network's convolutions in order: (inputs, output channels, output). Pooling and upsampling stand between levels.
_CONVS = ((("in",), 16, "e0a"), (("e0a",), 16, "e0"), (("p1",), 32, "e1a"), (("e1a",), 32, "e1"), (("p2",), 64, "e2a"), (("e2a",), 64, "e2"),
          (("p3",), 64, "e3a"), (("e3a",), 64, "e3"), (("u2", "e2"), 64, "d2a"), (("d2a",), 64, "d2"), (("u1", "e1"), 32, "d1a"),
          (("d1a",), 32, "d1"), (("u0", "e0"), 16, "d0a"), (("d0a",), 16, "d0"))
_CHANNELS = {"in": 16, "p1": 16, "p2": 32, "p3": 64, "u2": 64, "u1": 64, "u0": 32}
_POOL = {"e0": "p1", "e1": "p2", "e2": "p3"}
_UP = {"e3": "u2", "d2": "u1", "d1": "u0"}
_RATE = 5e-4  # Adam's rate in the shipped network's training


def _conv_shapes():
    ch = dict(_CHANNELS)
    for ins, n, out in _CONVS:
        yield ins, n, out, sum(ch[i] for i in ins)
        ch[out] = n


def _network_params(seed):
    rng = np.random.default_rng(seed)
    parts = []
    for _, n, out, cin in _conv_shapes():
        fan = 3 if out == "e0a" else cin
        parts += [rng.normal(0.0, math.sqrt(2.0 / (27 * fan)), 27 * n * cin), rng.normal(0.0, 0.02, n)]
    parts += [rng.normal(0.0, 0.25, 16), np.zeros(1)]
    return np.concatenate(parts).astype(np.float32)


def _samples(case, seed):
    """Divergence, fluid and solid masks and target pressures of `batch` tanks: BF16 values in float32."""
    rng = np.random.default_rng(seed + 1)
    shape = (case["nz"], case["ny"], case["nx"])
    inputs, targets = [], []
    for _ in range(case["batch"]):
        z, y, x = np.meshgrid(*[(np.arange(n) + 0.5) / n for n in shape], indexing="ij")
        ph = rng.uniform(0.0, 6.0, 6)
        solid = np.zeros(shape, bool)
        for a in range(3):
            for edge in (0, -1):
                solid[tuple(edge if k == a else slice(None) for k in range(3))] = True
        fluid = (y < 0.5 + 0.1 * np.sin(5.0 * x + ph[0])) & (x < rng.uniform(0.4, 0.9)) & ~solid
        div = 0.5 * np.sin(9.0 * x + ph[1]) * np.cos(7.0 * z + ph[2]) + 0.3 * rng.standard_normal(shape)
        inp = np.zeros(shape + (16,), np.float32)
        inp[..., 0] = np.clip(div, -1.0, 1.0) * fluid
        inp[..., 1], inp[..., 2] = fluid, solid
        inputs.append(torch.from_numpy(inp).bfloat16())
        targets.append((np.sin(4.0 * x + ph[3]) * np.cos(3.0 * y + ph[4]) * 2.0 * fluid).astype(np.float32))
    return inputs, targets


def _prepare_train(case, seed):
    net = warmstart.WarmStartNet(dim=(case["nx"], case["ny"], case["nz"]), batch=case["batch"], seed=seed % (1 << 31), learning_rate=_RATE)
    net.set_params(_network_params(seed))
    inputs, targets = _samples(case, seed)
    for k, (i, t) in enumerate(zip(inputs, targets)):
        net.set_sample(k, i.view(torch.uint16).numpy(), t)
    return {"kind": "train", "net": net}


def _exact_train(case, seed):
    """Loss and updated parameters of the first step in float64 (convolutions by torch, gradients by autograd)."""
    p = torch.from_numpy(_network_params(seed)).double().cuda().requires_grad_(True)
    inputs, targets = _samples(case, seed)
    inp = torch.stack(inputs).double().cuda()
    target = torch.from_numpy(np.stack(targets)).double().cuda()
    t = {"in": inp.permute(0, 4, 1, 2, 3)}
    at = 0
    for ins, n, out, cin in _conv_shapes():
        w = p[at:at + 27 * n * cin].reshape(3, 3, 3, n, cin).permute(3, 4, 0, 1, 2)
        b = p[at + 27 * n * cin:at + 27 * n * cin + n]
        at += 27 * n * cin + n
        t[out] = torch.relu(torch.nn.functional.conv3d(torch.cat([t[i] for i in ins], 1), w, b, padding=1))
        if out in _POOL:
            t[_POOL[out]] = torch.nn.functional.avg_pool3d(t[out], 2)
        if out in _UP:
            t[_UP[out]] = t[out].repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
    guess = torch.einsum("bczyx,c->bzyx", t["d0"], p[at:at + 16]) + p[at + 16]
    fluid = inp[..., 1] > 0.5
    loss = ((guess - target)[fluid] ** 2).sum() / max(int(fluid.sum()), 1)
    loss.backward()
    g = p.grad
    step = _RATE * g / (g.abs() + 1e-8)  # Adam's first step: both moments are the gradient's own
    return {"loss": loss.item(), "params": (p.detach() - step).cpu()}


# ---- the interface -----------------------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"frame": _prepare_frame, "tanks": _prepare_tanks, "sort": _prepare_sort, "surface": _prepare_surface,
            "train": _prepare_train}[case["kind"]](case, int(seed))


def run(state):
    kind = state["kind"]
    if kind == "frame":
        sim = state["sim"]
        sim.step_frame(state["input"])
        r = sim.results()
        return {**_particles(sim), "max_speed": float(np.float32(r.max_particle_speed)), "fluid_cells": r.fluid_cells,
                "live_particles": r.live_particles}
    if kind == "tanks":
        S.step_frames(state["sims"], state["inputs"])
        return [_particles(sim)["pos_age_vel"] for sim in state["sims"]]
    if kind == "sort":
        S.sort_particles_static(state["in"].data_ptr(), state["out"].data_ptr(), state["count"], state["grid"], state["h"],
                                perm_out=state["perm"].data_ptr(), key_offsets_out=state["offsets"].data_ptr(),
                                live_count_out=state["live"].data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        return {"records": state["out"], "perm": state["perm"], "offsets": state["offsets"], "live": state["live"]}
    if kind == "surface":
        return _run_surface(state)
    net = state["net"]
    loss = net.train_step()
    return {"loss": float(loss), "params": net.params()}


def exact(case, seed):
    if case["kind"] == "surface":
        return _exact_surface(case, int(seed))
    if case["kind"] == "train" and case["nx"] * case["ny"] * case["nz"] * case["batch"] <= 1 << 20:
        return _exact_train(case, int(seed))
    # A frame is a chain of marks, lists and counts (cell types, brick slots, iterations to a residual) that a
    # 64-bit run would take other branches of; a sort's outputs are whole numbers.
    return None


def _frame_cells(case):
    cells = case["nx"] * case["ny"] * case["nz"]
    if case["scene"] == "dam_sphere":
        return 0.157 * cells
    if case["scene"] == "boxes":
        return 0.22 * cells
    return case["fill_x"] * case["fill_y"] * cells


def _substep_bytes(fluid, solver, iterations, viscosity):
    """Per substep: P2G reads the records (48 bytes) and writes 6 sums and a count per active cell, G2P reads and
    writes the records and reads the velocities; the grid passes read and write each field once (64 bytes a cell);
    a solver iteration reads the system and reads and writes its vectors once. 8 particles per fluid cell, the
    active bricks hold about 1.35 cells per fluid cell."""
    active = 1.35 * fluid
    per_iteration = 36.0 if solver == "rbgs" else 60.0
    return 144.0 * 8.0 * fluid + (28.0 + 12.0 + 64.0) * active + iterations * per_iteration * fluid + (12 * 36.0 * fluid if viscosity else 0.0)


def work(case):
    kind = case["kind"]
    if kind == "frame":
        fluid = _frame_cells(case)
        it = 10 if case["tolerance"] > 0 else case["iterations"]
        b = case["substeps"] * _substep_bytes(fluid, case["solver"], it, case["viscosity"] > 0)
        return {"bytes": b, "flops": case["substeps"] * fluid * (8.0 * 700.0 + it * 60.0)}
    if kind == "tanks":
        batch = scenes.tank_batch(S.settings_default, count=case["tanks"], seed=3, lo=case["lo"], hi=case["hi"])
        fluid = sum(t["particles"] for t in batch) / 8.0
        return {"bytes": 2.0 * _substep_bytes(fluid, "mgpcg", 10, False), "flops": 2.0 * fluid * (8.0 * 700.0 + 600.0)}
    if kind == "sort":
        keys = case["nx"] * case["ny"] * case["nz"] / 64.0
        return {"bytes": 100.0 * case["count"] + 4.0 * keys, "flops": 0.0}
    if kind == "surface":
        voxels = case["nx"] * case["ny"] * case["nz"] * case["resolution"] ** 3
        reach = case["smoothing"] * 0.6 * case["resolution"]
        return {"bytes": 16.0 * _surface_count(case) + 2.0 * voxels, "flops": _surface_count(case) * 4.19 * reach ** 3 * 25.0}
    voxels = case["nx"] * case["ny"] * case["nz"] * case["batch"]
    params = flops = 0
    for ins, n, out, cin in _conv_shapes():
        level = {"0": 0, "1": 1, "2": 2, "3": 3}[out[1]]
        params += 27 * n * cin + n
        flops += 3 * 2 * 27 * n * cin * voxels / 8 ** level
    return {"bytes": 24.0 * params + 36.0 * voxels, "flops": float(flops)}
