"""The calls a user of this lattice-Boltzmann engine makes, as cases to be timed.

Every case is one batch of a study (`Lattice.run`, `MultiLattice.run`: the
step list in, the forces per step out, the slice sampled at the batch's end
read back) or one gradient of a design loop (`GrayLattice.set_field` and
`backward`).  The number of steps in a batch is the study layer's: about a
quarter second at 2,800 million updates a second, from 16 to (here) 256.

Kinds of case:

* `tunnel`: a body held still in a wind tunnel on one D3Q19 level (velocity
  inlet holding the total pressure, open sides and outlet, sponges,
  Smagorinsky closure), body `sphere` or `arm`.  The study layer cuts its
  grids to the part's size, so extents are ragged as a rule, and stores FP32
  unless only 16 bits fit; the large throughput cases store 16 bits.
* `plain`: the laminar validation sphere (BGK, free-slip sides) with the
  whole field read back.
* `array`: a sphere in a periodic box driven by a body force (drag of a
  packed array), the whole field read back.
* `rotor`: a two-blade rotor spinning on one D3Q19 level.
* `levels`: a still sphere on D3Q27, one level or two nested ones.
* `rotor_levels`: the rotor spinning on the finest of three D3Q27 levels.
* `grad`: objective and gradient of the gray-level (Brinkman) solver.

The seed moves the body by fractions of a cell and sets the inflow speed (or
draws the solid fraction), as the runs of a parameter study differ.  Spheres
come with analytic links (the engine takes any StaticVoxels), so that the
same flow can be computed in 64 bits without the engine.

Forces of lattices whose arithmetic is 32-bit, and gradients taken through
it, are logged in 32 bits: their terms carry no more.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from simlab_b200.cases import BODY_TO_LATTICE
from simlab_b200.gray import AdjointSpec, GrayLattice, GraySetup
from simlab_b200.lbm import (STEP_DTYPE, WALL_DTYPE, Collision, FaceBc, Lattice, LatticeSetup, Probes, SliceDef, SpinGeometry, StaticVoxels, Storage,
                             steps_array, voxelize_spin, voxelize_static)
from simlab_b200.mlattice import LevelBox, MultiLattice, MultiSetup
from simlab_b200.shapes import arm, propeller

STORAGE = {"fp32": Storage.FP32, "fp16": Storage.FP16, "bf16": Storage.BF16, "fp64": Storage.FP64}
SIZE = {"fp32": 4, "fp16": 2, "bf16": 2, "fp64": 8}


def listed():
    return [
        # the laminar validation case: the smallest lattice, where launches count
        dict(name="plain_fp32_96x48x48", kind="plain", storage="fp32", nx=96, ny=48, nz=48, r=6.0),
        # a single-level study as the planner cuts it: FP32, no extent a multiple of anything
        dict(name="tunnel_fp32_203x131x117", kind="tunnel", body="sphere", storage="fp32", nx=203, ny=131, nz=117, r=12.0),
        # a ragged study stored in bfloat16
        dict(name="tunnel_bf16_301x157x157", kind="tunnel", body="sphere", storage="bf16", nx=301, ny=157, nz=157, r=16.0),
        # the headline throughput case
        dict(name="tunnel_fp16_512x256x256", kind="tunnel", body="arm", storage="fp16", nx=512, ny=256, nz=256, r=1.0),
        # the same body at twice the resolution: the largest lattice
        dict(name="tunnel_fp16_1024x512x512", kind="tunnel", body="arm", storage="fp16", nx=1024, ny=512, nz=512, r=2.0),
        # drag of a packed array: periodic box, body force
        dict(name="array_fp32_131x130x129", kind="array", storage="fp32", nx=131, ny=130, nz=129, r=30.0),
        # a spinning rotor on one level, re-voxelized every step
        dict(name="rotor_fp16_256x128x128", kind="rotor", storage="fp16", nx=256, ny=128, nz=128, r=40.0),
        # one D3Q27 level, 16-bit storage
        dict(name="levels1_fp16_256x128x128", kind="levels", storage="fp16", nx=256, ny=128, nz=128, r=12.0, boxes=0),
        # a still part as the planner refines it: two nested levels, FP32
        dict(name="levels2_fp32_121x73x71", kind="levels", storage="fp32", nx=121, ny=73, nz=71, r=14.0, boxes=1),
        # the refined rotor: three levels, 28 million cells
        dict(name="rotor_levels_fp16_256x128x128", kind="rotor_levels", storage="fp16", nx=256, ny=128, nz=128, r=60.0),
        # the design case, every segment recomputed from its checkpoint
        dict(name="grad_fp32_192x96x96", kind="grad", storage="fp32", nx=192, ny=96, nz=96, steps=200, every=50, recompute=True),
        # the gradient at scale: FP16 forward, moments kept
        dict(name="grad_fp16_384x192x192", kind="grad", storage="fp16", nx=384, ny=192, nz=192, steps=60, every=20, recompute=False),
    ]


def draw(rng):
    kind = rng.choice(["tunnel"] * 5 + ["plain", "array", "array", "rotor", "levels", "levels", "levels", "rotor_levels", "grad", "grad"])

    def extents(lo, hi, ax=2.0):
        cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        ny = cells / (ax * rng.uniform(0.8, 1.25))
        ny = ny ** (1.0 / 3.0)
        nz = ny * rng.uniform(0.8, 1.25)
        nx = cells / (ny * nz)
        nx, ny, nz = int(round(nx)), int(round(ny)), int(round(nz))
        if rng.random() < 0.25:  # rows of whole 16-byte units, as a user who picks round numbers has them
            nx = max(nx // 16, 3) * 16
        return dict(nx=nx, ny=ny, nz=nz)

    if kind == "plain":
        d = extents(6e4, 1e6)
        return dict(kind=kind, storage="fp32", r=round(min(d["ny"], d["nz"]) * rng.uniform(0.08, 0.14), 2), **d)
    if kind == "tunnel":
        d = extents(3e5, 3e7)
        return dict(kind=kind, body="sphere", storage=rng.choice(["fp32", "fp32", "fp32", "fp16", "fp16", "bf16", "fp64"]),
                    r=round(min(d["ny"], d["nz"]) * rng.uniform(0.06, 0.12), 2), **d)
    if kind == "array":
        d = extents(2e5, 6e6, ax=1.0)
        return dict(kind=kind, storage=rng.choice(["fp32", "fp32", "fp16"]), r=round(min(d["nx"], d["ny"], d["nz"]) * rng.uniform(0.15, 0.3), 2), **d)
    if kind == "rotor":
        d = extents(1.5e6, 6e6)
        return dict(kind=kind, storage=rng.choice(["fp32", "fp16"]), r=round(min(d["ny"], d["nz"]) * rng.uniform(0.25, 0.33), 2), **d)
    if kind == "levels":
        boxes = rng.choice([0, 1, 1])
        d = extents(2e5, 2e6 if boxes else 8e6)
        return dict(kind=kind, storage=rng.choice(["fp32", "fp32", "fp16", "bf16"]), r=round(min(d["ny"], d["nz"]) * rng.uniform(0.08, 0.16), 2),
                    boxes=boxes, **d)
    if kind == "rotor_levels":
        ny = rng.randrange(56, 112)
        return dict(kind=kind, storage=rng.choice(["fp32", "fp16"]), nx=2 * ny + rng.randrange(0, 9), ny=ny, nz=ny + rng.randrange(-4, 5),
                    r=round(0.45 * ny, 2))
    d = extents(2e5, 6e6)
    every = rng.randrange(10, 40)
    return dict(kind=kind, storage=rng.choice(["fp32", "fp16"]), steps=rng.randrange(40, 120), every=every, recompute=rng.random() < 0.5, **d)


# ------------------------------------------------------------------ inputs
def _cells(case):
    return case["nx"] * case["ny"] * case["nz"]


def _level_boxes(case):
    """The nested boxes: about 0.63 of the parent per axis for the rotor, the
    part and its near wake for a still sphere."""
    out, d = [], [case["nx"], case["ny"], case["nz"]]
    n_boxes = 2 if case["kind"] == "rotor_levels" else case["boxes"]
    for _ in range(n_boxes):
        n = [max(int(v * 0.63), 8) for v in d]
        out.append(([(d[k] - n[k]) // 2 for k in range(3)], n))
        d = [2 * (v - 1) + 1 for v in n]
    return out, d


def _updates(case):
    """Cell updates of one (finest) step, averaged over the levels' sub-cycling."""
    if case["kind"] not in ("levels", "rotor_levels"):
        return float(_cells(case))
    boxes, _ = _level_boxes(case)
    cells = [_cells(case)] + [math.prod(2 * (v - 1) + 1 for v in n) for _, n in boxes]
    return sum(c / 2.0 ** (len(cells) - 1 - l) for l, c in enumerate(cells))


def _batch(case):
    ss = 2 ** len(_level_boxes(case)[0]) if case["kind"] in ("levels", "rotor_levels") else 1
    n = int(min(max(0.25 * 2800e6 / _updates(case), 16), 256))
    return (n + ss - 1) // ss * ss


def _flow(case, seed):
    """What the seed sets: the inflow speed and the body's place in its cell."""
    g = np.random.RandomState(seed % (2 ** 32))
    return 0.05 * g.uniform(0.9, 1.1), g.uniform(-0.45, 0.45, 3)


def _center(dims, off, front=0.3):
    return [dims[0] * front + off[0], dims[1] * 0.5 + off[1], dims[2] * 0.5 + off[2]]


C19 = np.array([[0, 0, 0], [1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1], [1, 1, 0], [-1, -1, 0], [1, 0, 1], [-1, 0, -1],
                [0, 1, 1], [0, -1, -1], [1, -1, 0], [-1, 1, 0], [1, 0, -1], [-1, 0, 1], [0, 1, -1], [0, -1, 1]])
C27 = np.array([[i % 3 - 1, (i // 3) % 3 - 1, i // 9 - 1] for i in range(27)])


def _sphere_links(dims, c, r, cset):
    """Solid cells and wall cells of a sphere: every link that ends inside it,
    with the distance to its surface, rounded to the 16 bits a record keeps."""
    lo = [max(int(math.floor(c[k] - r)) - 2, 0) for k in range(3)]
    hi = [min(int(math.ceil(c[k] + r)) + 2, dims[k] - 1) for k in range(3)]
    z, y, x = np.meshgrid(*[np.arange(lo[k], hi[k] + 1) for k in (2, 1, 0)], indexing="ij")
    rel = np.stack([x - c[0], y - c[1], z - c[2]], -1).astype(np.float64)
    inside = (rel ** 2).sum(-1) < r * r
    cell = ((z.astype(np.int64) * dims[1] + y) * dims[0] + x)
    mask = np.zeros(inside.shape, dtype=np.uint32)
    q = np.ones(inside.shape + (27,), dtype=np.float32)
    for i, ci in enumerate(cset):
        if not ci.any():
            continue
        end = np.zeros_like(inside)
        src = tuple(slice(max(ci[k], 0), inside.shape[2 - k] + min(ci[k], 0)) for k in (2, 1, 0))
        dst = tuple(slice(max(-ci[k], 0), inside.shape[2 - k] + min(-ci[k], 0)) for k in (2, 1, 0))
        end[dst] = inside[src]
        cut = end & ~inside
        a, b, g = float((ci ** 2).sum()), rel[cut] @ ci, (rel[cut] ** 2).sum(-1) - r * r
        t = (-b - np.sqrt(np.maximum(b * b - a * g, 0.0))) / a
        q[cut, i] = np.clip(t, 0.001, 1.0).astype(np.float16).astype(np.float32)
        mask[cut] |= np.uint32(1 << i)
    walls = np.zeros(int((mask != 0).sum()), dtype=WALL_DTYPE)
    walls["cell"] = cell[mask != 0]
    walls["mask"] = mask[mask != 0]
    walls["q"] = q[mask != 0]
    return StaticVoxels(solid=cell[inside].astype(np.uint32), walls=walls)


def _gray_inputs(case, seed):
    dims = [case["nx"], case["ny"], case["nz"]]
    lo, bn = [v // 4 for v in dims], [v // 3 for v in dims[:1]] + [v // 2 for v in dims[1:]]
    g = torch.Generator(device="cpu").manual_seed(seed)
    f = torch.rand((1, 1, bn[2], bn[1], bn[0]), generator=g)
    for _ in range(3):  # a smooth solid fraction, as the filtered fields of a design loop
        f = torch.nn.functional.avg_pool3d(f, 3, 1, 1, count_include_pad=False)
    return dims, lo, bn, f.reshape(-1).double().numpy()


def _slice(dims, center):
    return Probes(slices=[SliceDef(origin=[0, 0, int(center[2])], u=[1, 0, 0], v=[0, 1, 0], nu=int(dims[0]), nv=int(dims[1]))])


def _sponge(dims):
    side = max(min(dims[1], dims[2]) // 16, 3)
    return [side, 2 * side] + [side] * 4


def _setup(case, seed):
    """(setup, geometry, dims of the body's level, centre) of a still part."""
    F = FaceBc
    u, off = _flow(case, seed)
    dims = [case["nx"], case["ny"], case["nz"]]
    st = STORAGE[case["storage"]]
    if case["kind"] == "levels":
        boxes, fd = _level_boxes(case)
        c = _center(fd, off, 0.4 if boxes else 0.3)
        s = MultiSetup(dims0=dims, boxes=[LevelBox(lo=lo, n=n) for lo, n in boxes], faces=[F.VELOCITY] + [F.OPEN] * 5, nu0=0.002, smagorinsky=0.1,
                       u_inf=[u, 0.0, 0.0], u_init=[u, 0.0, 0.0], sponge=_sponge(dims), sponge_tau=1.0, sponge_sigma=0.1, total_pressure_inlet=True,
                       storage=st, center=c)
        return s, _sphere_links(fd, c, case["r"], C27), fd, c
    if case["kind"] == "plain":
        c = _center(dims, off, 0.25)
        s = LatticeSetup(dims=dims, faces=[F.VELOCITY, F.OPEN] + [F.FREE_SLIP] * 4, nu=0.8 * u * 2 * case["r"] / 40.0, u_inf=[u, 0.0, 0.0],
                         u_init=[u, 0.0, 0.0], collision=Collision.BGK, storage=st, center=c, debug_dump=True)
    elif case["kind"] == "array":
        c = _center(dims, off, 0.5)
        s = LatticeSetup(dims=dims, faces=[F.PERIODIC] * 6, nu=0.05, u_init=[u, 0.0, 0.0], body_force=[1e-5, 0.0, 0.0], storage=st, center=c,
                         debug_dump=True)
    else:
        c = _center(dims, off, 0.25)
        s = LatticeSetup(dims=dims, faces=[F.VELOCITY] + [F.OPEN] * 5, nu=u * 12.0 / 1e5 if case["body"] == "arm" else 1e-3, smagorinsky=0.17,
                         u_inf=[u, 0.0, 0.0], u_init=[u, 0.0, 0.0], sponge=_sponge(dims), sponge_tau=1.0, sponge_sigma=0.1,
                         total_pressure_inlet=True, storage=st, center=c)
        if case["body"] == "arm":
            v, t = arm(center=c, scale=case["r"])
            return s, voxelize_static(v, t, dims), dims, c
    return s, _sphere_links(dims, c, case["r"], C19), dims, c


WARM = 16  # steps a study has run before the timed batch: the field is under way


def prepare(case, seed):
    kind = case["kind"]
    n = _batch(case) if kind != "grad" else 0
    if kind == "grad":
        dims, lo, bn, gamma = _gray_inputs(case, seed)
        c = [lo[k] + 0.5 * (bn[k] - 1) for k in range(3)]
        lat = GrayLattice(GraySetup(dims=dims, box_lo=lo, box_n=bn, nu=0.02, u_in=[0.04, 0.0, 0.0], center=c, storage=STORAGE[case["storage"]]))
        spec = AdjointSpec(steps=case["steps"], t0=case["steps"] // 2 + 1, t1=case["steps"], checkpoint_every=case["every"], recompute=case["recompute"])
        return dict(kind=kind, lat=lat, gamma=gamma, spec=spec)
    real = np.float64 if case["storage"] == "fp64" else np.float32
    if kind in ("rotor", "rotor_levels"):
        F = FaceBc
        u, off = _flow(case, seed)
        st = STORAGE[case["storage"]]
        v, t = propeller(radius=case["r"])
        sv = voxelize_spin(v, t, [0.0, 0.0, 1.0], 0.125)
        dims = [case["nx"], case["ny"], case["nz"]]
        boxes, fd = _level_boxes(case) if kind == "rotor_levels" else ([], dims)
        c = _center(fd, off, 0.5 if boxes else 0.37)
        r = int(math.ceil(sv.radius)) + 3
        ax = [int(math.floor(c[0] + sv.axial[0])) - 3, int(math.ceil(c[0] + sv.axial[1])) + 3]
        geo = SpinGeometry(vox=sv, box_lo=[ax[0], int(c[1]) - r, int(c[2]) - r], box_n=[ax[1] - ax[0] + 1, 2 * r + 2, 2 * r + 2])
        wind = dict(u_inf=[0.4 * u, 0.0, 0.0], u_init=[0.4 * u, 0.0, 0.0], total_pressure_inlet=True, storage=st, center=c)
        if boxes:
            lat = MultiLattice(MultiSetup(dims0=dims, boxes=[LevelBox(lo=lo, n=b) for lo, b in boxes], faces=[F.VELOCITY] + [F.OPEN] * 5, nu0=1e-5,
                                          sponge=[0] + _sponge(dims)[1:], sponge_tau=1.0, sponge_sigma=0.1, **wind), geo, _slice(fd, c))
        else:
            lat = Lattice(LatticeSetup(dims=dims, faces=[F.VELOCITY] + [F.OPEN] * 5, nu=4e-4, **wind), geo, _slice(dims, c))
        state = dict(kind=kind, lat=lat, n=n, omega=0.08 / case["r"], theta=0.0, real=real)
        lat.run(_turn(state, 16, False))
        return state
    s, vox, fd, c = _setup(case, seed)
    if kind == "levels":
        lat = MultiLattice(s, vox, _slice(fd, c))
    else:
        lat = Lattice(s, vox, None if s.debug_dump else _slice(fd, c))
    lat.advance(WARM)
    lat.synchronize()
    steps = steps_array(n)
    steps[-1]["sample"] = 1
    return dict(kind=kind, lat=lat, steps=steps, real=real)


def _turn(state, n, sample=True):
    """The step records of the next n steps of a part at its full speed."""
    w = state["omega"]
    th = state["theta"] + w * np.arange(n + 1)
    rot = np.zeros((n + 1, 3, 3))
    rot[:, 0, 0] = 1.0
    rot[:, 1, 1] = rot[:, 2, 2] = np.cos(th)
    rot[:, 2, 1] = np.sin(th)
    rot[:, 1, 2] = -rot[:, 2, 1]
    rot = rot @ BODY_TO_LATTICE
    a = np.zeros(n, dtype=STEP_DTYPE)
    a["rot"], a["rot_prev"] = rot[1:], rot[:-1]
    a["omega"] = [w, 0.0, 0.0]
    a["sample"][-1] = int(sample)
    state["theta"] = th[-1]
    return a


# ------------------------------------------------------------------ one pass
def run(state):
    lat = state["lat"]
    if state["kind"] == "grad":
        lat.set_field(state["gamma"])
        j, grad = lat.backward(state["spec"])
        return {"objective": np.float32(j), "gradient": grad.astype(np.float32)}
    forces = lat.run(_turn(state, state["n"]) if "theta" in state else state["steps"]).astype(state["real"])
    if state["kind"] in ("plain", "array"):
        return {"forces": forces, "field": lat.macros()}
    return {"forces": forces, "slice": lat.slice_means()}


def work(case):
    """Every population read once and written once per update, and the cell's
    flag; the reverse sweep of a gradient reads and writes the adjoint and
    reads the 4 moments, and a recomputed segment is one more forward step."""
    size = SIZE[case["storage"]]
    if case["kind"] == "grad":
        n = case["steps"] * _cells(case)
        fwd, rev = 2 * 19 * size + 4, 2 * 19 * 4 + 20
        return {"bytes": float(n * (fwd + rev + 16 + (fwd if case["recompute"] else 0))), "flops": float(n * (600 + (250 if case["recompute"] else 0)))}
    q = 27 if case["kind"] in ("levels", "rotor_levels") else 19
    n = _batch(case) * _updates(case)
    return {"bytes": float(n * (2 * q * size + 4)), "flops": float(n * (250 if q == 19 else 520))}


# ------------------------------------------------------------------ in 64 bits
def _t(v):
    return torch.as_tensor(v, dtype=torch.float64, device="cuda")


def _weights(cset):
    n = len(cset)
    m = (cset ** 2).sum(1)
    table = {19: [1 / 3, 1 / 18, 1 / 36], 27: [8 / 27, 2 / 27, 1 / 54, 1 / 216]}[n]
    return [table[k] for k in m]


def _opposite(cset):
    return [int(np.where((cset == -c).all(1))[0][0]) for c in cset]


def _moments(f, cset):
    """(rho - 1, j, second moments) of the populations' deviations from the weights."""
    d = f.sum(0)
    j = [sum(int(c[a]) * f[i] for i, c in enumerate(cset) if c[a]) for a in range(3)]
    s = [sum(int(c[a] * c[b]) * f[i] for i, c in enumerate(cset) if c[a] * c[b]) for a, b in PAIRS]
    return d, j, s


PAIRS = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]


def _stress(d, s, rho, u):
    return [s[k] - rho * u[a] * u[b] - (d / 3 if a == b else 0) for k, (a, b) in enumerate(PAIRS)]


def _fneq(cset, w, p, i):
    c = cset[i]
    tr = (p[0] + p[1] + p[2]) / 3
    t = -tr
    for k, (a, b) in enumerate(PAIRS):
        if c[a] * c[b]:
            t = t + (1 if a == b else 2) * int(c[a] * c[b]) * p[k]
    return 4.5 * w[i] * t


def _feq19(w, i, d, rho, u):
    c = C19[i]
    cu = sum(int(c[a]) * u[a] for a in range(3))
    return w[i] * (d + rho * (3 * cu + 4.5 * cu * cu - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])))


def _feq27(w, i, rho, u):
    f = rho
    for a in range(3):
        c = int(C27[i][a])
        f = f * ((2 / 3 - u[a] * u[a]) if c == 0 else 0.5 * (1 / 3 + u[a] * u[a] + c * u[a]))
    return f - w[i]


class _Exact:
    """One level in 64 bits: post-collision populations P of every cell, pulled,
    collided, faces rebuilt from the cell inside, links after Bouzidi."""

    def __init__(self, s, dims, cset, vox, center, nu, u_inf, top=True):
        self.s, self.dims, self.c, self.q = s, dims, cset, len(cset)
        self.w, self.opp = _weights(cset), _opposite(cset)
        self.u_inf = u_inf
        shape = (dims[2], dims[1], dims[0])
        one = torch.ones(shape, dtype=torch.float64, device="cuda")
        u = [float(v) for v in s.u_init]
        self.P = torch.stack([(_feq19(self.w, i, 0.0, 1.0, u) if self.q == 19 else _feq27(self.w, i, 1.0, u)) * one for i in range(self.q)])
        self.tau0, self.smag2 = 0.5 + 3 * nu, s.smagorinsky ** 2
        self.g = list(getattr(s, "body_force", (0.0, 0.0, 0.0)))
        # faces: type per cell (0 none, 1 velocity, 2 open, 3 free slip) and the cell inside
        idx = [torch.arange(n, device="cuda") for n in (dims[2], dims[1], dims[0])]
        Z, Y, X = torch.meshgrid(*idx, indexing="ij")
        pos = (X, Y, Z)
        self.ty = torch.zeros(shape, dtype=torch.int64, device="cuda")
        self.mirror = []
        inner = []
        for a in range(3):
            per = s.faces[2 * a] == FaceBc.PERIODIC
            inner.append(pos[a] if per or not top else pos[a].clamp(1, dims[a] - 2))
            m = torch.zeros(shape, dtype=torch.bool, device="cuda")
            for f in (2 * a, 2 * a + 1):
                if not top or s.faces[f] == FaceBc.PERIODIC:
                    continue
                on = pos[a] == (0 if f % 2 == 0 else dims[a] - 1)
                t = {FaceBc.VELOCITY: 1, FaceBc.OPEN: 2, FaceBc.FREE_SLIP: 3}[s.faces[f]]
                self.ty = torch.where(on & (self.ty != 1), torch.full_like(self.ty, t), self.ty)
                if t == 3:
                    m |= on
            self.mirror.append(m)
        flat = (Z * dims[1] + Y) * dims[0] + X
        self.face = flat[self.ty > 0]
        self.fty = self.ty.reshape(-1)[self.face]
        self.inner = ((inner[2] * dims[1] + inner[1]) * dims[0] + inner[0]).reshape(-1)[self.face]
        self.fmir = [m.reshape(-1)[self.face] for m in self.mirror]
        sp = torch.zeros(shape, dtype=torch.float64, device="cuda")
        for f in range(6):
            if top and s.sponge[f] > 0:
                a = f // 2
                p = pos[a].double() if f % 2 == 0 else (dims[a] - 1 - pos[a]).double()
                sp = torch.maximum(sp, 1 - p / s.sponge[f])
        self.sp = sp.clamp(0, 1)
        self.sponge = top and any(v > 0 for v in s.sponge)
        self.hold = (self.ty > 0).clone()  # cells the step leaves alone
        self.links = []
        self.solid = torch.zeros(shape, dtype=torch.bool, device="cuda")
        self.wall = torch.zeros(0, dtype=torch.int64, device="cuda")
        if vox is not None:
            self.solid.reshape(-1)[torch.as_tensor(vox.solid.astype(np.int64), device="cuda")] = True
            self.hold |= self.solid
            cell = torch.as_tensor(vox.walls["cell"].astype(np.int64), device="cuda")
            self.wall = cell
            mask = torch.as_tensor(vox.walls["mask"].astype(np.int64), device="cuda")
            qs = _t(vox.walls["q"])
            xyz = torch.stack([cell % dims[0], (cell // dims[0]) % dims[1], cell // (dims[0] * dims[1])]).double()
            rel = xyz - _t(center)[:, None]
            for i in range(self.q):
                cut = ((mask >> i) & 1) == 1
                if cset[i].any() and bool(cut.any()):
                    open_ = ((mask[cut] >> self.opp[i]) & 1) == 0
                    self.links.append((i, cell[cut], qs[cut, i].clamp(min=0.001), open_, rel[:, cut]))

    def faces(self):
        if not len(self.face):
            return
        g = self.P.reshape(self.q, -1)[:, self.inner]
        d, j, s2 = _moments(g, self.c)
        rho = 1 + d
        u = [j[a] / rho - (0.5 * self.g[a] if self.q == 19 else 0.0) for a in range(3)]
        p = _stress(d, s2, rho, u)
        if self.q == 27:
            tr = (p[0] + p[1] + p[2]) / 3
            p = [p[k] - (tr if k < 3 else 0) for k in range(6)]
        vel = self.fty == 1
        ui2 = sum(v * v for v in self.u_inf)
        if self.s.total_pressure_inlet:
            rho = torch.where(vel, (1 / 3 + 0.5 * ui2) / (1 / 3 + 0.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)), torch.ones_like(rho))
        else:
            u = [torch.where(vel, torch.full_like(u[a], float(self.u_inf[a])), u[a]) for a in range(3)]
            rho = torch.where(vel, rho, torch.ones_like(rho))
        out = []
        for i in range(self.q):
            v = (_feq19(self.w, i, rho - 1, rho, u) if self.q == 19 else _feq27(self.w, i, rho, u)) + _fneq(self.c, self.w, p, i)
            if bool((self.fty == 3).any()):
                m = torch.zeros_like(self.face)
                for bits in range(8):
                    cm = self.c[i] * np.array([-1 if bits >> a & 1 else 1 for a in range(3)])
                    sel = sum((self.fmir[a].long() << a) for a in range(3)) == bits
                    m[sel] = int(np.where((self.c == cm).all(1))[0][0])
                v = torch.where(self.fty == 3, torch.gather(g, 0, m[None])[0], v)
            out.append(v)
        self.P.reshape(self.q, -1)[:, self.face] = torch.stack(out)

    def step(self):
        f = torch.stack([torch.roll(self.P[i], tuple(int(v) for v in self.c[i][::-1]), (0, 1, 2)) for i in range(self.q)])
        ff, own = f.reshape(self.q, -1), self.P.reshape(self.q, -1)
        F, T, sub = torch.zeros(3, dtype=torch.float64, device="cuda"), torch.zeros(3, dtype=torch.float64, device="cuda"), []
        for i, cell, q, open_, rel in self.links:
            o, w = self.opp[i], self.w[i]
            fpi, fpo, fin = own[i, cell] + w, own[o, cell] + w, ff[i, cell] + w
            fb = torch.where(q >= 0.5, (fpi + (2 * q - 1) * fpo) / (2 * q), torch.where(open_, 2 * q * fpi + (1 - 2 * q) * fin, fpi))
            sub.append((o, cell, fb - w))
            c = _t(self.c[i].astype(float))[:, None]
            fl = c * (fpi + fb)
            F += fl.sum(1)
            T += torch.linalg.cross(rel + q * c, fl, dim=0).sum(1)
        for o, cell, v in sub:
            ff[o, cell] = v
        d, j, s2 = _moments(f, self.c)
        rho = 1 + d
        u = [(j[a] / rho + 0.5 * self.g[a]) for a in range(3)]
        p = _stress(d, s2, rho, u)
        tr = (p[0] + p[1] + p[2]) / 3
        dv = [p[k] - (tr if self.q == 27 and k < 3 else 0) for k in range(6)]
        tau = torch.full_like(rho, self.tau0)
        if self.smag2 > 0:
            pp = dv[0] ** 2 + dv[1] ** 2 + dv[2] ** 2 + 2 * (dv[3] ** 2 + dv[4] ** 2 + dv[5] ** 2)
            tau = 0.5 * (self.tau0 + torch.sqrt(self.tau0 ** 2 + 18 * self.smag2 * torch.sqrt(2 * pp) / rho))
        sp2 = self.sp ** 2
        if self.sponge:
            tau = torch.where((self.sp > 0) & (tau < self.s.sponge_tau), tau + sp2 * (self.s.sponge_tau - tau), tau)
        om = 1 / tau
        out = self._collide19(f, d, rho, u, p, om, sp2) if self.q == 19 else self._collide27(rho, u, dv, om, sp2)
        self.P = torch.where(self.hold, self.P, out)
        self.last = (rho, u, p, tau)
        return torch.cat([F, T])

    def _collide19(self, f, d, rho, u, p, om, sp2):
        sg = self.s.sponge_sigma * sp2
        bgk = self.s.collision == Collision.BGK
        out = []
        for i in range(19):
            fe = _feq19(self.w, i, d, rho, u)
            v = (1 - om) * f[i] + om * fe if bgk else fe + (1 - om) * _fneq(self.c, self.w, p, i)
            if self.sponge:
                v = v + sg * (_feq19(self.w, i, 0.0, 1.0, u) - fe)
            if any(self.g):
                c = C19[i]
                cg = sum(int(c[a]) * self.g[a] for a in range(3))
                cu = sum(int(c[a]) * u[a] for a in range(3))
                ug = sum(u[a] * self.g[a] for a in range(3))
                v = v + self.w[i] * rho * ((1 - 0.5 * om) * (9 * cu * cg - 3 * ug + 3 * cg) - (0 if bgk else 1.5 * (1 - om) * cg))
            out.append(v)
        return torch.stack(out)

    def _collide27(self, rho, u, dv, om, sp2):
        a, b, cc = [1 / 3 + (1 - om) / rho * dv[k] for k in range(3)]
        d, e, g = [(1 - om) / rho * dv[k] for k in range(3, 6)]
        k = {(0, 0, 0): torch.ones_like(rho), (2, 0, 0): a, (0, 2, 0): b, (0, 0, 2): cc, (1, 1, 0): d, (1, 0, 1): e, (0, 1, 1): g,
             (2, 2, 0): a * b + 2 * d * d, (2, 0, 2): a * cc + 2 * e * e, (0, 2, 2): b * cc + 2 * g * g,
             (2, 1, 1): a * g + 2 * d * e, (1, 2, 1): b * e + 2 * d * g, (1, 1, 2): cc * d + 2 * e * g,
             (2, 2, 2): a * b * cc + 2 * (a * g * g + b * e * e + cc * d * d) + 8 * d * e * g}
        zero = torch.zeros_like(rho)
        val = {(x, y, z): k.get((x, y, z), zero) for x in range(3) for y in range(3) for z in range(3)}
        for ax in (2, 1, 0):  # central moments to populations, one axis at a time
            new = {}
            for key in val:
                if key[ax]:
                    continue
                k0, k1, k2 = [val[key[:ax] + (m,) + key[ax + 1:]] for m in range(3)]
                r1 = k1 + u[ax] * k0
                r2 = k2 + 2 * u[ax] * k1 + u[ax] ** 2 * k0
                for m, v in enumerate((0.5 * (r2 - r1), k0 - r2, 0.5 * (r2 + r1))):
                    new[key[:ax] + (m,) + key[ax + 1:]] = v
            val = new
        out = []
        for i in range(27):
            v = rho * val[tuple(int(t) + 1 for t in C27[i])] - self.w[i]
            if self.sponge:
                v = v + self.s.sponge_sigma * sp2 * (_feq27(self.w, i, 1.0, u) - _feq27(self.w, i, rho, u))
            out.append(v)
        return torch.stack(out)

    def field(self):
        """(rho, u) between steps: from the populations, for wall cells of the
        D3Q19 lattice as the collision left them; nothing on solid and (D3Q19) face cells."""
        d, j, _ = _moments(self.P, self.c)
        rho = 1 + d
        v = torch.stack([rho] + [j[a] / rho - 0.5 * self.g[a] for a in range(3)], -1).reshape(-1, 4)
        if self.q == 19 and len(self.wall):
            v[self.wall] = torch.stack([self.last[0]] + list(self.last[1]), -1).reshape(-1, 4)[self.wall]
        v[(self.hold if self.q == 19 else self.solid).reshape(-1)] = float("nan")
        return v


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return _exact_grad(case, seed)
    # the arm's links come from the engine's voxelizer, a spinning part's from
    # its re-voxelizer and nested levels from its interpolation: no value here
    if kind in ("rotor", "rotor_levels") or case.get("body") == "arm" or case.get("boxes") or _cells(case) * _batch(case) > 1.5e9:
        return None
    s, vox, dims, c = _setup(case, seed)
    L = _Exact(s, dims, C27 if kind == "levels" else C19, vox, c, s.nu0 if kind == "levels" else s.nu, list(s.u_inf))
    forces = []
    for k in range(WARM + _batch(case)):
        L.faces()
        forces.append(L.step())
    forces = torch.stack(forces[WARM:]).cpu().numpy()
    v = L.field()
    if kind in ("plain", "array"):
        return {"forces": forces, "field": v.cpu().numpy()}
    v = v.reshape(dims[2], dims[1], dims[0], 4)[int(c[2])].clone()
    if kind == "levels":
        v[0], v[-1], v[:, 0], v[:, -1] = [float("nan")] * 4
    return {"forces": forces, "slice": v.reshape(-1, 4).cpu().numpy()}


def _exact_grad(case, seed):
    """The gray-level step and its derivative by automatic differentiation,
    step by step backwards from stored states."""
    if _cells(case) * case["steps"] > 2e9:
        return None
    dims, lo, bn, gamma = _gray_inputs(case, seed)
    nx, ny, nz = dims
    w = _weights(C19)
    om = 1 / (0.5 + 3 * 0.02)
    u = [0.04, 0.0, 0.0]
    inlet = _t([_feq19(w, i, 0.0, 1.0, u) for i in range(19)])
    box = (slice(lo[2], lo[2] + bn[2]), slice(lo[1], lo[1] + bn[1]), slice(lo[0], lo[0] + bn[0]))

    def step(P, gam):
        g = torch.stack([torch.roll(P[i], tuple(int(v) for v in C19[i][::-1]), (0, 1, 2)) for i in range(19)])
        d = g.sum(0)
        j = [sum(int(c[a]) * g[i] for i, c in enumerate(C19) if c[a]) for a in range(3)]
        a = torch.zeros(nz, ny, nx, dtype=torch.float64, device="cuda")
        a[box] = gam
        jj = j[0] * j[0] + j[1] * j[1] + j[2] * j[2]
        rho, B = 1 + d, om - 1 + (1 - a) ** 2
        out = []
        for i in range(19):
            cj = sum(int(C19[i][k]) * j[k] for k in range(3))
            out.append((1 - om) * g[i] + w[i] * (om * d + 3 * (om - a) * cj + B / rho * (4.5 * cj * cj - 1.5 * jj)))
        out = torch.stack(out)[..., 1:-1]
        out = torch.cat([inlet[:, None, None, None].expand(19, nz, ny, 1), out, out[..., -1:]], -1)
        return out, (a * j[0])[box].sum()

    T, t0 = case["steps"], case["steps"] // 2 + 1
    start = inlet[:, None, None, None].expand(19, nz, ny, nx).clone()
    gam = _t(gamma).reshape(bn[2], bn[1], bn[0])
    K = max(int(math.sqrt(T)), 1)
    kept, J, P = [], 0.0, start
    with torch.no_grad():
        for t in range(T):
            if t % K == 0:
                kept.append(P)
            P, F = step(P, gam)
            if t + 1 >= t0:
                J += float(F) / (T - t0 + 1)
    lam, grad = torch.zeros_like(P), torch.zeros_like(gam)
    for seg in reversed(range(len(kept))):
        states = [kept[seg]]
        with torch.no_grad():
            for t in range(seg * K, min((seg + 1) * K, T) - 1):
                states.append(step(states[-1], gam)[0])
        for k in reversed(range(len(states))):
            t = seg * K + k
            x, y = states[k].detach().requires_grad_(True), gam.detach().requires_grad_(True)
            P, F = step(x, y)
            weight = 1.0 / (T - t0 + 1) if t + 1 >= t0 else 0.0
            lam, dg = torch.autograd.grad((P * lam).sum() + weight * F, (x, y))
            grad += dg
            states.pop()
    return {"objective": np.float64(J), "gradient": grad.reshape(-1).cpu().numpy()}
