"""The work this framework is timed on: the solves and the steps around them of a FLIP substep, called through the
public Python classes (and, for the steps around the solve, the ``*_device`` entry points of the C ABI).

Every case is a dict of plain values.  ``prepare`` makes its inputs on the GPU from a seed: the liquid is the
repository's plain geometry ({y < 0.4} and a sphere) or its large one ({y < 0.45} and four spheres) in a box with solid
walls, its surface moved by a part of a voxel by the seed; face velocities are uniform in [-1, 1].  Sides need not be
multiples of 8: the outermost leaves then hold voxels that are not active.
"""
import ctypes
import math

import numpy as np
import torch

from uaamg_b200 import _lib
from uaamg_b200.batch import PoissonBatch
from uaamg_b200.extrapolate import prepare_channel, run_layers_device
from uaamg_b200.grids import LeafGrid
from uaamg_b200.packed3 import packed_FloatGrid3
from uaamg_b200.poisson import LaplacianWithLevel, PoissonSolver, _as_c
from uaamg_b200.viscosity import L_with_level, simd_viscosity3d

DEVICE = "cuda"
SMOOTHERS = {"jacobi": 0, "weighted_jacobi": 1, "rbgs": 2, "spai0": 3}
SIDES = (32, 64, 96, 128, 192)  # boxes of a batch


def listed():
    return [
        # a preview or a droplet: the whole pressure step (matrix, hierarchy, rhs, solve) where launches count
        {"name": "pressure step 40", "kind": "pressure_step", "n": 40, "host": False},
        # the repository's headline step: what a FLIP substep does with inputs that are on the GPU already
        {"name": "pressure step 128", "kind": "pressure_step", "n": 128, "host": False},
        # the same step for a simulation whose grids live in pinned host memory and whose pressure goes back there
        {"name": "pressure step 128 host", "kind": "pressure_step", "n": 128, "host": True},
        # a production-size step, with a side that is no multiple of a leaf
        {"name": "pressure step 250", "kind": "pressure_step", "n": 250, "host": False},
        # a hierarchy that is kept while the liquid's cells stay, solved from the last pressure: the red-black smoother
        {"name": "pressure solve 160 rbgs", "kind": "pressure_solve", "n": 160, "smoother": "rbgs",
         "precision": "fp32", "warm": True},
        # the mixed-precision form at a size where it is chosen
        {"name": "pressure solve 320 fp16", "kind": "pressure_solve", "n": 320, "smoother": "jacobi",
         "precision": "fp16", "warm": False},
        # the largest domain of the repository's configurations, in FP32
        {"name": "pressure solve 512", "kind": "pressure_solve", "n": 512, "smoother": "jacobi",
         "precision": "fp32", "warm": False},
        # many small uneven domains at once (a farm of simulations, a training set)
        {"name": "pressure batch 40", "kind": "pressure_batch", "count": 40},
        # a small viscous object: matrix, hierarchy, rhs, warm start and solve
        {"name": "viscosity step 44", "kind": "viscosity_step", "n": 44, "mu": 1e3},
        # the repository's viscosity configuration
        {"name": "viscosity step 128", "kind": "viscosity_step", "n": 128, "mu": 1e3},
        # a large viscous liquid whose matrix is kept over substeps: rhs, warm start and solve
        {"name": "viscosity solve 240", "kind": "viscosity_solve", "n": 240, "mu": 1e3},
        # what a substep does around its pressure solve: the vec3 velocity split into channels, face weights, liquid
        # SDF in solids, pressure gradient on three channels, extrapolation of three channels
        {"name": "velocity update 128", "kind": "velocity_update", "n": 128, "layers": 3, "friction": 0.5},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pressure_step", "pressure_step", "pressure_solve", "pressure_solve", "pressure_batch",
                       "viscosity_step", "viscosity_solve", "velocity_update"])
    if kind == "pressure_step":
        return {"kind": kind, "n": _log_uniform(rng, 24, 300), "host": rng.random() < 0.3}
    if kind == "pressure_solve":
        precision = rng.choice(["fp32", "fp32", "fp16", "bf16"])
        smoother = rng.choice(["jacobi", "weighted_jacobi", "rbgs", "spai0"] if precision == "fp32" else
                              ["jacobi", "weighted_jacobi"])
        return {"kind": kind, "n": _log_uniform(rng, 32, 400), "smoother": smoother, "precision": precision,
                "warm": rng.random() < 0.5}
    if kind == "pressure_batch":
        return {"kind": kind, "count": _log_uniform(rng, 2, 48)}
    if kind == "velocity_update":
        return {"kind": kind, "n": _log_uniform(rng, 24, 200), "layers": rng.randint(1, 5),
                "friction": rng.choice([0.0, 0.5])}
    return {"kind": kind, "n": _log_uniform(rng, 24, 200), "mu": rng.choice([1.0, 1e2, 1e3])}


# ---------------------------------------------------------------------------------------------- inputs on the GPU
def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _up8(n):
    return -(-n // 8) * 8


def _to_leaves(dense):
    """[X, Y, Z(, C)] with sides that are multiples of 8 -> [leaves, 512(, C)], x slowest."""
    X, Y, Z = dense.shape[:3]
    v = dense.reshape(X // 8, 8, Y // 8, 8, Z // 8, 8, -1).permute(0, 2, 4, 1, 3, 5, 6)
    return (v.reshape(-1, 512) if dense.dim() == 3 else v.reshape(-1, 512, dense.shape[3])).contiguous()


def _origins(sides, lo):
    ax = [np.arange(s // 8, dtype=np.int32) * 8 + lo for s in sides]
    return np.ascontiguousarray(np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3))


def _masks(active):
    """bool [leaves, 512] -> uint64 [leaves, 8] on the host."""
    weights = torch.ones(64, dtype=torch.int64, device=active.device) << torch.arange(64, device=active.device)
    return (active.reshape(-1, 8, 64).to(torch.int64) * weights).sum(2).cpu().numpy().view(np.uint64)


def _grid(dense, background, lo=0, masks=None, pinned=False):
    comps = 1 if dense.dim() == 3 else dense.shape[3]
    g = LeafGrid(origins=np.zeros((0, 3), np.int32),
                 values=np.zeros((0, 512) if comps == 1 else (0, 512, comps), np.float32),
                 background=np.full(comps, background, np.float32))
    g.origins, g.masks = _origins(dense.shape[:3], lo), masks
    g.values = _to_leaves(dense)
    if pinned:
        host = torch.empty(g.values.shape, dtype=torch.float32, pin_memory=True)
        host.copy_(g.values)
        g.pinned = host  # owns the memory behind the array
        g.values = host.numpy()
    return g


def _empty(components, background):
    shape = (0, 512) if components == 1 else (0, 512, components)
    return LeafGrid(origins=np.zeros((0, 3), np.int32), values=np.zeros(shape, np.float32),
                    background=np.full(components, background, np.float32))


def _liquid(n, seed, large):
    """The liquid's signed distance at the voxel centres, float32 [n, n, n]."""
    moved = 0.1 / n * np.random.RandomState(seed % (1 << 31)).uniform(-1, 1)
    if not large:
        return _distance(n, 0.4 + moved, [((0.5, 0.7, 0.5), 0.15)])
    r = np.random.RandomState(2)
    balls = [((r.uniform(0.15, 0.85), 0.5 + 0.4 * r.uniform(0.15, 0.85), r.uniform(0.15, 0.85)), 0.1) for _ in range(4)]
    return _distance(n, 0.45 + moved, balls)


def _balls(n, index):
    """An instance of a batch: one to six balls, radii log-uniform in [0.05, 0.3]."""
    r = np.random.RandomState(index)
    balls = [(tuple(r.uniform(0, 1, 3)), math.exp(r.uniform(math.log(0.05), math.log(0.3))))
             for _ in range(r.randint(1, 7))]
    return _distance(n, None, balls)


def _distance(n, slab, balls):
    c = (torch.arange(n, device=DEVICE, dtype=torch.float32) + 0.5) / n
    X, Y, Z = c.view(n, 1, 1), c.view(1, n, 1), c.view(1, 1, n)
    phi = torch.full((n, n, n), 12.0, device=DEVICE)
    if slab is not None:
        phi = torch.minimum(phi, Y - slab)
    for p, radius in balls:
        phi = torch.minimum(phi, torch.sqrt((X - p[0]) ** 2 + (Y - p[1]) ** 2 + (Z - p[2]) ** 2) - radius)
    return phi


def _wall_weights(n):
    """Open face fractions on the face lattice: 1 inside, 0 on the six walls, 1 in the padding."""
    m, f = _up8(n + 1), n + 1
    w = torch.ones((m, m, m, 3), device=DEVICE)
    w[0, :f, :f, 0] = 0.0
    w[n, :f, :f, 0] = 0.0
    w[:f, 0, :f, 1] = 0.0
    w[:f, n, :f, 1] = 0.0
    w[:f, :f, 0, 2] = 0.0
    w[:f, :f, n, 2] = 0.0
    return w


def _velocities(n, gen):
    m, f = _up8(n + 1), n + 1
    v = torch.zeros((3, m, m, m), device=DEVICE)
    v[:, :f, :f, :f] = torch.rand((3, f, f, f), generator=gen, device=DEVICE) * 2 - 1
    return v


def _padded(phi, background):
    """The box's field with its last leaves filled up, and those leaves' masks (None where there is nothing to fill)."""
    n = phi.shape[0]
    m = _up8(n)
    if m == n:
        return phi, None
    full = torch.full((m, m, m), background, device=DEVICE)
    full[:n, :n, :n] = phi
    on = torch.zeros((m, m, m), dtype=torch.bool, device=DEVICE)
    on[:n, :n, :n] = True
    return full, _masks(_to_leaves(on))


def _liquid_grid(phi, pinned=False):
    bg = 3.0 / phi.shape[0]
    full, masks = _padded(phi, bg)
    return _grid(full, bg, masks=masks, pinned=pinned)


def _pressure_inputs(phi, gen, pinned=False):
    n = phi.shape[0]
    v = _velocities(n, gen)
    return {"phi": _liquid_grid(phi, pinned), "weights": _grid(_wall_weights(n), 1.0, pinned=pinned),
            "velocity": [_grid(v[k], 0.0, pinned=pinned) for k in range(3)], "solid_velocity": _empty(3, 0.0),
            "dt": 1.0, "dx": 1.0 / n}


def _viscosity_inputs(phi, gen, mu):
    n = phi.shape[0]
    m = _up8(n) + 16
    c = torch.arange(m, device=DEVICE, dtype=torch.float32) - 7.5
    a = torch.minimum(c, n - c)
    wall = torch.minimum(torch.minimum(a.view(m, 1, 1), a.view(1, m, 1)), a.view(1, 1, m)) - 0.25
    v = _velocities(n, gen)
    return {"phi": _liquid_grid(phi), "solid": _grid((wall / n).contiguous(), -3.0 / n, lo=-8),
            "viscosity": _empty(1, mu), "velocity": [_grid(v[k], 0.0) for k in range(3)],
            "solid_velocity": _empty(3, 0.0), "dt": 1.0 / 240.0, "rho": 1.0, "dx": 1.0 / n}


# ------------------------------------------------------------------------------------------------------- prepare
def prepare(case, seed):
    return {"pressure_step": _prepare_step, "pressure_solve": _prepare_solve, "pressure_batch": _prepare_batch,
            "viscosity_step": _prepare_viscosity, "viscosity_solve": _prepare_viscosity,
            "velocity_update": _prepare_update}[case["kind"]](case, seed)


def _prepare_step(case, seed):
    gen = _generator(seed)
    s = _pressure_inputs(_liquid(case["n"], seed, False), gen, pinned=case["host"])
    s.update(kind=case["kind"], host=case["host"])
    return s


def _kept_solver(i, smoother):
    lap = LaplacianWithLevel.createPressurePoissonLaplacian(i["phi"], i["weights"], i["dt"], i["dx"])
    rhs = torch.empty((lap.leaf_count(0), 512), device=DEVICE)
    lap.createPressurePoissonRightHandSide(i["weights"], *i["velocity"], i["solid_velocity"], i["dt"], out=rhs)
    solver = PoissonSolver(lap)
    solver.mSmoother = SMOOTHERS[smoother]
    return solver, rhs


def _prepare_solve(case, seed):
    gen = _generator(seed)
    phi = _liquid(case["n"], seed, case["n"] > 300)
    solver, rhs = _kept_solver(_pressure_inputs(phi, gen), case["smoother"])
    if case["precision"] != "fp32":
        solver.prepare_mixed(case["precision"])
    guess = torch.zeros_like(rhs)
    if case["warm"]:  # the last substep's pressure: near this one's
        solver.mRelativeTolerance = 1e-2
        solver.solveMultigridPCG(guess, rhs)
        solver.mRelativeTolerance = 1e-7
    return {"kind": case["kind"], "solver": solver, "rhs": rhs, "guess": guess, "x": torch.empty_like(rhs),
            "precision": case["precision"]}


def _batch_side(index):
    return SIDES[index % len(SIDES)]


def _prepare_batch(case, seed):
    solvers, rhss = [], []
    for k in range(case["count"]):
        gen = _generator(seed * 1009 + k)
        solver, rhs = _kept_solver(_pressure_inputs(_balls(_batch_side(k), k), gen), "jacobi")
        solvers.append(solver)
        rhss.append(rhs)
    return {"kind": case["kind"], "batch": PoissonBatch(solvers), "rhs": rhss,
            "x": [torch.empty_like(b) for b in rhss]}


def _prepare_viscosity(case, seed):
    s = _viscosity_inputs(_liquid(case["n"], seed, False), _generator(seed), case["mu"])
    s["kind"] = case["kind"]
    if case["kind"] == "viscosity_solve":
        s["level0"] = L_with_level.create_viscosity_matrix(s["viscosity"], s["phi"], s["solid"], s["dt"], s["rho"],
                                                           s["dx"])
        shape = (3, s["level0"].leaf_count(0), 512)
        s["rhs"], s["x"] = torch.empty(shape, device=DEVICE), torch.empty(shape, device=DEVICE)
        s["solver"] = simd_viscosity3d(s["level0"])
    return s


def _solid(n):
    """Walls 1.3 voxels thick and a ball as the solid's signed distance, with a margin of a leaf (and the voxels that
    the face weights of the margin read)."""
    m = _up8(n + 2) + 16
    c = torch.arange(m, device=DEVICE, dtype=torch.float32) - 8
    a = torch.minimum(c - 1.3, n - 1.3 - c)
    wall = torch.minimum(torch.minimum(a.view(m, 1, 1), a.view(1, m, 1)), a.view(1, 1, m))
    X, Y, Z = (c - p * n for p in (0.5, 0.25, 0.5))
    ball = torch.sqrt(X.view(m, 1, 1) ** 2 + Y.view(1, m, 1) ** 2 + Z.view(1, 1, m) ** 2) - n / 8
    return torch.minimum(wall, ball) / n


def _weight_topology(n):
    """The box dilated by two voxels: origins and masks of the face weights' leaves, from -8 on."""
    m = _up8(n + 2) + 8
    on = torch.zeros((m, m, m), dtype=torch.bool, device=DEVICE)
    on[6:8 + n + 2, 6:8 + n + 2, 6:8 + n + 2] = True
    return _origins((m, m, m), -8), _masks(_to_leaves(on)), on


def _update_fields(case, seed):
    """The dense fields of a velocity update: what prepare() cuts into leaves and exact() computes from."""
    n, gen = case["n"], _generator(seed)
    m = _up8(n + 1)
    phi = _liquid(n, seed, False)
    velocity = _velocities(n, gen)
    c = torch.arange(n, device=DEVICE, dtype=torch.float32) / n
    depth = torch.clamp(0.42 - c, min=0.0).view(1, n, 1)
    pressure = (9.8 * depth + 0.01 * torch.rand((n, n, n), generator=gen, device=DEVICE)) / n
    solid_velocity = torch.rand((m, m, m, 3), generator=gen, device=DEVICE) * 2 - 1
    return phi, velocity, pressure, solid_velocity


def _prepare_update(case, seed):
    n = case["n"]
    phi, velocity, pressure, solid_velocity = _update_fields(case, seed)
    s = {"kind": case["kind"], "dt": 1.0 / n, "dx": 1.0 / n, "layers": case["layers"], "friction": case["friction"]}
    s["phi"], s["solid"] = _liquid_grid(phi), _grid(_solid(n), -3.0 / n, lo=-8)
    s["vec3"] = _grid(velocity.permute(1, 2, 3, 0).contiguous(), 0.0)
    s["solid_velocity"] = _grid(solid_velocity, 0.0)
    s["origins"], s["masks"], _ = _weight_topology(n)
    s["weights"] = _empty(3, 1.0)
    s["weights"].origins, s["weights"].masks = s["origins"], s["masks"]
    s["weights"].values = torch.empty((s["origins"].shape[0], 512, 3), device=DEVICE)
    s["liquid"] = torch.empty((s["phi"].leaf_count, 512), device=DEVICE)
    _face_weights(s)
    s["lap"] = LaplacianWithLevel.createPressurePoissonLaplacian(s["phi"], s["weights"], s["dt"], s["dx"])
    # the pressure over the matrix's leaves
    origins, masks = s["lap"].dof_topology(0)
    m = _up8(n)
    full = torch.zeros((m, m, m), device=DEVICE)
    full[:n, :n, :n] = pressure
    at = torch.from_numpy(((origins // 8).astype(np.int64) * np.array([(m // 8) ** 2, m // 8, 1])).sum(1)).to(DEVICE)
    bits = torch.from_numpy(np.unpackbits(masks.view(np.uint8), axis=1, bitorder="little")).to(DEVICE)
    s["pressure"] = _to_leaves(full)[at] * bits
    v = s["vec3"]
    s["mask"] = [torch.empty((v.leaf_count, 8), dtype=torch.int64, device=DEVICE) for _ in range(3)]
    s["update"] = [torch.empty((v.leaf_count, 512), device=DEVICE) for _ in range(3)]
    s["reflected"] = [torch.empty((v.leaf_count, 512), device=DEVICE) for _ in range(3)]
    # where the extrapolation goes: the liquid's voxels that a channel has no value for after the update
    on = np.full((s["phi"].leaf_count, 8), np.uint64(0xFFFFFFFFFFFFFFFF)) if s["phi"].masks is None else s["phi"].masks
    channels = _split(s)
    _gradient(s, channels)
    torch.cuda.synchronize()
    s["fill"] = []
    for k in range(3):
        g = LeafGrid(origins=v.origins, values=np.zeros((v.leaf_count, 512), np.float32), background=0.0,
                     masks=s["mask"][k].cpu().numpy().view(np.uint64))
        org, _, _, leaf, fill = prepare_channel(g, (s["phi"].origins, on))
        s["fill"].append((org, leaf, fill))
    return s


# ----------------------------------------------------------------------------------------------------------- run
def run(state):
    return {"pressure_step": _run_step, "pressure_solve": _run_solve, "pressure_batch": _run_batch,
            "viscosity_step": _run_viscosity, "viscosity_solve": _run_viscosity,
            "velocity_update": _run_update}[state["kind"]](state)


def _run_step(s):
    lap = LaplacianWithLevel.createPressurePoissonLaplacianWithRhs(
        s["phi"], s["weights"], *s["velocity"], s["solid_velocity"], s["dt"], s["dx"])
    solver = PoissonSolver(lap)
    shape = (lap.leaf_count(0), 512)
    x = np.empty(shape, np.float32) if s["host"] else torch.empty(shape, device=DEVICE)
    solver.solveMultigridPCGResident(x)
    return {"pressure": x, "iterations": solver.mIterationTaken}


def _run_solve(s):
    s["x"].copy_(s["guess"])
    if s["precision"] == "fp32":
        s["solver"].solveMultigridPCG(s["x"], s["rhs"])
    else:
        s["solver"].solveMultigridPCGMixed(s["x"], s["rhs"], s["precision"])
    return {"pressure": s["x"], "iterations": s["solver"].mIterationTaken}


def _run_batch(s):
    for x in s["x"]:
        x.zero_()
    s["batch"].solveMultigridPCG(s["x"], s["rhs"])
    return {"pressure": s["x"], "iterations": np.array(s["batch"].mIterationTaken, np.int64)}


def _run_viscosity(s):
    if s["kind"] == "viscosity_solve":
        level0, solver, rhs, x = s["level0"], s["solver"], s["rhs"], s["x"]
    else:
        level0 = L_with_level.create_viscosity_matrix(s["viscosity"], s["phi"], s["solid"], s["dt"], s["rho"], s["dx"])
        solver = simd_viscosity3d(level0)
        shape = (3, level0.leaf_count(0), 512)
        rhs, x = torch.empty(shape, device=DEVICE), torch.empty(shape, device=DEVICE)
    level0.build_rhs(*s["velocity"], s["solid_velocity"], out=rhs)
    level0.gather_velocity(*s["velocity"], out=x)
    solver.pcg_solve(x, 1e-6, rhs)
    return {"velocity": x, "rhs": rhs, "iterations": solver.m_iteration}


def _face_weights(s):
    solid = _as_c(s["solid"], [])
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(_lib.lib().uaamg_face_weights_device(
        ctypes.byref(solid), s["origins"].shape[0], s["origins"].ctypes.data, s["masks"].ctypes.data,
        s["weights"].values.data_ptr(), stream), "face_weights")


def _split(s):
    """The velocity's channels as grids of their own."""
    packed = packed_FloatGrid3()
    packed.from_vec3(s["vec3"])
    return packed.v


def _gradient(s, channels):
    lib, keep = _lib.lib(), []
    phi, weights, solid_velocity = (_as_c(s[k], keep) for k in ("phi", "weights", "solid_velocity"))
    grids = [_as_c(g, keep) for g in channels]
    touched = [g.values for g in channels] + s["mask"] + s["update"] + s["reflected"]
    with _lib.torch_ordered("poisson", s["lap"]._h, s["pressure"], *touched):
        for k in range(3):
            _lib.check(lib.uaamg_poisson_apply_pressure_gradient_device(
                s["lap"]._h, ctypes.byref(phi), ctypes.byref(weights), ctypes.byref(solid_velocity),
                s["pressure"].data_ptr(), s["dt"], s["friction"], k, ctypes.byref(grids[k]),
                channels[k].values.data_ptr(), s["mask"][k].data_ptr(), s["update"][k].data_ptr(),
                s["reflected"][k].data_ptr()), "apply_pressure_gradient")


def _run_update(s):
    stream = torch.cuda.current_stream().cuda_stream
    channels = _split(s)
    _face_weights(s)
    keep = []
    solid, phi = _as_c(s["solid"], keep), _as_c(s["phi"], keep)
    _lib.check(_lib.lib().uaamg_immerse_liquid_phi_device(ctypes.byref(solid), ctypes.byref(phi), s["dx"],
                                                          s["liquid"].data_ptr(), stream), "immerse_liquid_phi")
    _gradient(s, channels)
    for k, (origins, leaf, fill) in enumerate(s["fill"]):
        run_layers_device(s["layers"], origins, channels[k].values, s["mask"][k], leaf, fill, stream=stream)
    return {"weights": s["weights"].values, "liquid": s["liquid"], "velocity": [g.values for g in channels],
            "mask": s["mask"], "update": s["update"], "reflected": s["reflected"]}


# ---------------------------------------------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once; a solve's iterations each read the operator and the vectors of the
    conjugate gradients once more, and do the arithmetic of the cycle (seven stencil passes on level 0 and, on the
    coarser levels of a W-cycle, a third of that again)."""
    kind = case["kind"]
    if kind == "pressure_batch":
        parts = [_solve_work(0.13 * _batch_side(k) ** 3, 7) for k in range(case["count"])]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    n3 = float(case["n"]) ** 3
    liquid = 0.414 * n3
    if kind == "velocity_update":
        # split: 24; weights: 4 + 12; SDF: 8 + 4; gradient of a channel: velocity and four fields in, three out
        return {"bytes": n3 * (24 + 16 + 12 + 3 * (32 + 4) + 12), "flops": n3 * 60}
    if kind.startswith("viscosity"):
        dof, iterations = 3 * liquid, 9
        b, f = dof * 4 * (3 + iterations * (10 + 5)), dof * iterations * 4 * 4 / 3 * 2 * 30
        return {"bytes": b + (n3 * 4 * 2 + dof * 4 * 10 if kind == "viscosity_step" else 0), "flops": f}
    b, f = _solve_work(liquid * (1.15 if case["n"] > 300 else 1.0), 5 if case.get("smoother") == "rbgs" else 7)
    if kind == "pressure_step":
        b += n3 * 4 + liquid * 4 * (3 + 3 + 5)
    return {"bytes": b, "flops": f}


def _solve_work(dof, iterations):
    return dof * 4 * (2 + iterations * (5 + 5)), dof * iterations * 7 * 4 / 3 * 14


# --------------------------------------------------------------------------------------------------------- exact
def exact(case, seed):
    kind = case["kind"]
    if kind in ("pressure_step", "pressure_solve") and case["n"] <= 420:
        phi = _liquid(case["n"], seed, kind == "pressure_solve" and case["n"] > 300)
        x = _exact_pressure(phi, _generator(seed))
        return {"pressure": x, "iterations": None}
    if kind == "pressure_batch":
        xs = [_exact_pressure(_balls(_batch_side(k), k), _generator(seed * 1009 + k))
              for k in range(case["count"])]
        return {"pressure": xs, "iterations": None}
    if kind == "velocity_update":
        return _exact_update(case, seed)
    return None


def _shift(a, axis, step, fill):
    """b[i] = a[i + step] along an axis, `fill` where that is outside."""
    b = torch.full_like(a, fill)
    n = a.shape[axis]
    src, dst = [slice(None)] * a.dim(), [slice(None)] * a.dim()
    src[axis], dst[axis] = (slice(1, n), slice(0, n - 1)) if step > 0 else (slice(0, n - 1), slice(1, n))
    b[tuple(dst)] = a[tuple(src)]
    return b


def _inside(a, b):
    """The part of a segment with these end values that is inside."""
    cut = torch.where(a < 0, a / (a - b), b / (b - a))
    return torch.where((a < 0) & (b < 0), torch.ones_like(a), torch.where((a < 0) | (b < 0), cut, torch.zeros_like(a)))


def _tree_order(dof):
    """Leaves of the box [m, m, m] that hold a true voxel, in an OpenVDB tree's order (128^3 nodes, then leaves)."""
    m = dof.shape[0] // 8
    has = _to_leaves(dof).any(1)
    i = torch.arange(m, device=DEVICE)
    X, Y, Z = (t.reshape(-1) for t in torch.meshgrid(i, i, i, indexing="ij"))
    key = ((X >> 4) * 64 + (Y >> 4)) * 64 + (Z >> 4)
    key = ((key * 16 + (X & 15)) * 16 + (Y & 15)) * 16 + (Z & 15)
    at = torch.nonzero(has).reshape(-1)
    return at[torch.argsort(key[at])]


def _exact_pressure(phi32, gen):
    """The pressure in 64 bits: ghost-fluid Laplacian of the box, solved by diagonally preconditioned CG."""
    n, dx = phi32.shape[0], 1.0 / phi32.shape[0]
    phi = phi32.double()
    v = _velocities(n, gen)
    w, v = _wall_weights(n), v.double()
    t, far = 1.0 / (dx * dx), 3.0 * dx
    liquid = phi < 0
    diag, rhs, nz = torch.zeros_like(phi), torch.zeros_like(phi), torch.zeros_like(liquid)
    off = []  # the entry towards the lower neighbour of each axis
    for ax in range(3):
        for step in (1, -1):
            sl = [slice(0, n)] * 3
            if step > 0:
                sl[ax] = slice(1, n + 1)
            weight, vel = w[tuple(sl) + (ax,)].double(), v[ax][tuple(sl)]
            other = _shift(phi, ax, step, far)
            theta = torch.clamp(_inside(phi, other), min=0.02)
            diag += torch.where(other < 0, weight, weight / theta) * t
            rhs -= step * weight * vel / dx
            nz |= weight != 0
            if step < 0:
                off.append(torch.where((other < 0) & liquid, -weight * t, torch.zeros_like(phi)))
    dof = liquid & (diag != 0)
    rhs = torch.where(dof & nz, rhs, torch.zeros_like(rhs))
    inv = torch.where(dof, 1.0 / diag, torch.zeros_like(diag))
    diag = torch.where(dof, diag, torch.zeros_like(diag))

    def matrix(x):
        y = diag * x
        for ax in range(3):
            lo, hi = [slice(None)] * 3, [slice(None)] * 3
            lo[ax], hi[ax] = slice(0, n - 1), slice(1, n)
            lo, hi = tuple(lo), tuple(hi)
            y[hi] += off[ax][hi] * x[lo]
            y[lo] += off[ax][hi] * x[hi]
        return y

    x, r = torch.zeros_like(rhs), rhs.clone()
    z = inv * r
    p, rho = z.clone(), (r * z).sum()
    goal = 1e-11 * float(rhs.norm())
    for k in range(20000):
        q = matrix(p)
        a = rho / (p * q).sum()
        x += a * p
        r -= a * q
        if k % 20 == 0 and float(r.norm()) <= goal:
            break
        z = inv * r
        new = (r * z).sum()
        p = z + (new / rho) * p
        rho = new
    m = _up8(n)
    full, on = torch.zeros((m, m, m), device=DEVICE, dtype=torch.float64), torch.zeros((m, m, m), dtype=torch.bool,
                                                                                    device=DEVICE)
    full[:n, :n, :n], on[:n, :n, :n] = x, dof
    return _to_leaves(full)[_tree_order(on)]


def _square(bl, br, tl, tr):
    """The part of a square with these corner values that is inside."""
    c = [bl, br, tr, tl]
    f = [_inside(c[i], c[(i + 1) % 4]) for i in range(4)]
    neg = [(v < 0) for v in c]
    count = sum(v.to(torch.int32) for v in neg)
    cut_in = sum(torch.where(neg[i], 0.5 * f[i] * f[i - 1], torch.zeros_like(f[i])) for i in range(4))
    cut_out = 1 - sum(torch.where(neg[i], torch.zeros_like(f[i]), 0.5 * (1 - f[i]) * (1 - f[i - 1])) for i in range(4))
    sides = 0.5 * sum(torch.where(neg[i] != neg[(i + 1) % 4], f[i], torch.zeros_like(f[i])) for i in range(4))
    diagonal = (count == 2) & (neg[0] == neg[2])
    two = torch.where(diagonal, torch.where(sum(c) < 0, cut_out, cut_in), sides)
    one = torch.where(count == 1, cut_in, torch.where(count == 2, two, cut_out))
    return torch.where(count == 0, torch.zeros_like(one), torch.where(count == 4, torch.ones_like(one), one))


def _exact_update(case, seed):
    n, dx = case["n"], 1.0 / case["n"]
    phi32, velocity, pressure, solid_velocity = _update_fields(case, seed)
    phi, solid = phi32.double(), _solid(n).double()
    _, _, on = _weight_topology(n)
    size, m = on.shape[0], _up8(n + 1)
    corner = {}
    for i in (0, 1):
        for j in (0, 1):
            for k in (0, 1):
                c = torch.full((size,) * 3, -3.0 * dx, device=DEVICE, dtype=torch.float64)
                part = solid[i:i + size, j:j + size, k:k + size]
                c[:part.shape[0], :part.shape[1], :part.shape[2]] = part
                corner[i, j, k] = c
    faces = [((0, 0, 0), (0, 1, 0), (0, 0, 1), (0, 1, 1)), ((0, 0, 0), (0, 0, 1), (1, 0, 0), (1, 0, 1)),
             ((0, 0, 0), (1, 0, 0), (0, 1, 0), (1, 1, 0))]
    weights = []
    for f in faces:
        w = torch.clamp(1 - _square(*(corner[q] for q in f)), 0, 1)
        weights.append(torch.where(on, torch.where(w < 1e-2, torch.zeros_like(w), w), torch.ones_like(w)))
    weights = torch.stack(weights, -1)

    # the liquid's SDF inside the solid: every voxel of the box is active
    centre = sum(corner.values())[8:8 + n, 8:8 + n, 8:8 + n] / 8
    inside = centre < 0
    first = torch.where(inside, phi - 0.5 * dx, phi)
    bg = 3.0 * dx
    least, found = torch.full_like(first, 3.0 * dx), torch.zeros_like(inside)
    up = _up8(n)
    stored = torch.full((up,) * 3, bg, device=DEVICE, dtype=torch.float64)
    stored[:n, :n, :n] = first
    for ax in range(3):
        for step in (1, -1):
            v = _shift(stored, ax, step, bg)[:n, :n, :n]
            least = torch.where(found, least, torch.minimum(least, v))
            found |= v < 0
    air = torch.where(first < 0, torch.clamp(-centre, min=bg), first)
    second = torch.where(inside, torch.where(found, least, air), first)
    liquid = torch.full((up,) * 3, bg, device=DEVICE, dtype=torch.float64)
    liquid[:n, :n, :n] = second
    if up > n:  # voxels beside the box that its dilation makes active
        liquid = _exact_rim(liquid, stored, corner, n, up, bg)

    # pressure gradient: the matrix's unknowns are the liquid voxels with an open face
    def box(a, fill, dtype=torch.float64):
        b = torch.full((m,) * 3, fill, device=DEVICE, dtype=dtype)
        b[:n, :n, :n] = a
        return b

    open_face = torch.zeros((n, n, n), dtype=torch.bool, device=DEVICE)
    for ax in range(3):
        for step in (0, 1):
            sl = [slice(8, 8 + n)] * 3
            sl[ax] = slice(8 + step, 8 + step + n)
            open_face |= weights[tuple(sl) + (ax,)] > 0
    dof = box((phi < 0) & open_face, False, torch.bool)
    p = torch.where(dof, box(pressure.double(), 0.0), torch.zeros((), device=DEVICE, dtype=torch.float64))
    value = box(phi, bg)
    target = box(torch.ones_like(phi32, dtype=torch.bool), False, torch.bool)
    out = {"weights": _to_leaves(weights), "liquid": _to_leaves(liquid), "velocity": [], "mask": [None] * 3,
           "update": [], "reflected": []}
    dt, friction = 1.0 / n, case["friction"]
    for ax in range(3):
        u = velocity[ax].double()
        w = torch.ones((m,) * 3, device=DEVICE, dtype=torch.float64)
        part = weights[8:8 + m, 8:8 + m, 8:8 + m, ax]
        w[:part.shape[0], :part.shape[1], :part.shape[2]] = part
        below = _shift(value, ax, -1, bg)
        has = (w > 0) & (dof | _shift(dof, ax, -1, False))
        theta = torch.where((value >= 0) | (below >= 0), torch.clamp(_inside(below, value), min=0.02),
                            torch.ones_like(u))
        d = -dt * (p - _shift(p, ax, -1, 0.0)) / dx / theta
        s = (1 - w) * friction
        moved = torch.where(w < 1, (1 - s) * (u + d) + s * solid_velocity[..., ax].double(), u + d)
        out["update"].append(_to_leaves(torch.where(has, d, u)))
        out["reflected"].append(_to_leaves(torch.where(has, u + 2 * d, u)))
        u, known = torch.where(has, moved, u), has
        for _ in range(case["layers"]):
            total, count = torch.zeros_like(u), torch.zeros_like(u)
            for k in range(3):
                for step in (-1, 1):
                    near = _shift(known, k, step, False)
                    total += torch.where(near, _shift(u, k, step, 0.0), torch.zeros_like(u))
                    count += near
            new = target & ~known & (count > 0)
            u = torch.where(new, total / count.clamp(min=1), u)
            known = known | new
        out["velocity"].append(_to_leaves(u))
    return out


def _exact_rim(liquid, stored, corner, n, up, bg):
    """The voxels one beside the box, inside its last leaves: active once the box is dilated."""
    rim = torch.zeros((up,) * 3, dtype=torch.bool, device=DEVICE)
    rim[:n + 1, :n + 1, :n + 1] = True
    rim[:n, :n, :n] = False
    centre = sum(c[8:8 + up, 8:8 + up, 8:8 + up] for c in corner.values()) / 8
    least, found = torch.full_like(stored, bg), torch.zeros_like(rim)
    for ax in range(3):
        for step in (1, -1):
            v = _shift(stored, ax, step, bg)
            least = torch.where(found, least, torch.minimum(least, v))
            found |= v < 0
    return torch.where(rim & (centre < 0) & found, least, liquid)
