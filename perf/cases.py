"""Performance cases of the tet FEM step.

Every case is a call a program of this framework makes in earnest, through its public entry points:

* a frame of one body whose state lives in host memory (the drop-in call);
* a few frames of a resident system, from a state that is set to a state that is read back;
* a rollout with its gradients.

The bodies are the framework's own: boxes of 0.1 m cubes split into six Kuhn tets, E, nu, yield and push of the
elastic block, the plastic block and the uneven batch.  Each pass starts from the same mid-motion state, made from
the seed: a smooth displacement of a fraction of a percent of the body, a smooth velocity and acceleration.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import talus_b200 as tb
from talus_b200 import _capi as capi

DT = 1.0 / 60.0
GRAVITY = (0.0, -9.81, 0.0)
VOXEL = 0.1
DENSITY = 1000.0
KUHN = np.array([[0, 1, 3, 7], [0, 3, 2, 7], [0, 2, 6, 7], [0, 6, 4, 7], [0, 4, 5, 7], [0, 5, 1, 7]])


def _case(kind, cells, precision, frames, **more):
    """One case; `more` overrides the defaults, which are the framework's own settings."""
    c = dict(kind=kind, cx=cells[0], cy=cells[1], cz=cells[2], precision=precision, frames=frames, law="corotated",
             bodies=1, youngs=1e6, poisson=0.3, tolerance=1e-3, iterations=64, jitter=0.01)
    c.update(more)
    return c


PLASTIC = dict(youngs=2e7, poisson=0.35, jitter=0.0)


def listed():
    return [
        # the smallest use: one prop, one frame, its state in host memory, FP64
        dict(_case("host", (8, 8, 8), "fp64", 1, law="snh"), name="prop frame fp64"),
        # a small resident prop with odd sizes, FP32-mixed
        dict(_case("elastic", (7, 5, 9), "mixed", 4), name="prop frames mixed"),
        # the framework's headline: a large yielding block pushed from above, in both precisions
        dict(_case("plastic", (64, 32, 32), "mixed", 2, **PLASTIC), name="plastic block mixed"),
        dict(_case("plastic", (41, 27, 25), "fp64", 2, **PLASTIC), name="plastic block fp64"),
        # a yielding body too small to fill the GPU
        dict(_case("plastic", (16, 8, 8), "fp64", 4, **PLASTIC), name="plastic small fp64"),
        # many uneven bodies in one system, solved to convergence, and at the default settings in FP64
        dict(_case("batch", (4, 24, 0), "mixed", 2, bodies=96, tolerance=1e-6, iterations=4000, jitter=0.0),
             name="batch mixed"),
        dict(_case("batch", (4, 24, 0), "fp64", 2, bodies=96, jitter=0.0), name="batch fp64"),
        # finite-strain plasticity
        dict(_case("hencky", (33, 20, 15), "mixed", 4, **PLASTIC), name="hencky block mixed"),
        # stiffness damping
        dict(_case("damped", (20, 14, 11), "fp64", 4), name="damped block fp64"),
        # a free body: thrown and spinning
        dict(_case("floating", (12, 10, 9), "mixed", 4), name="floating mixed"),
        # a caller-held solver state: the Cholesky preconditioner kept between frames
        dict(_case("factor", (16, 8, 8), "fp64", 4, youngs=2e7, poisson=0.35), name="solver state fp64"),
        # gradients of a rollout with respect to stiffness and start
        dict(_case("rollout", (16, 16, 16), "fp64", 10, law="snh", tolerance=1e-11, iterations=4000),
             name="rollout fp64"),
    ]


def _cells(rng, least, most):
    """Three axes whose number of cells is spread over its logarithm between least and most."""
    total = math.exp(rng.uniform(math.log(least), math.log(most)))
    side = total ** (1.0 / 3.0)
    a = side * math.exp(rng.uniform(-0.4, 0.4))
    b = side * math.exp(rng.uniform(-0.4, 0.4))
    a, b = max(2, round(a)), max(2, round(b))
    return a, b, max(2, min(int(most / (a * b)), round(total / (a * b))))


def draw(rng):
    kind = rng.choice(["host", "elastic", "plastic", "plastic", "batch", "batch", "hencky", "damped", "floating",
                       "factor", "rollout"])
    precision = rng.choice(["fp64", "mixed"])
    law = rng.choice(["corotated", "snh"])
    frames = rng.randint(1, 4)
    if kind == "host":
        return _case(kind, _cells(rng, 27, 1000), "fp64", 1, law=law)
    if kind == "elastic":
        return _case(kind, _cells(rng, 60, 40000), precision, frames, law=law)
    if kind == "plastic":
        return _case(kind, _cells(rng, 300, 60000), precision, min(frames, 2), **PLASTIC)
    if kind == "batch":
        lo = rng.randint(3, 8)
        more = dict(tolerance=1e-6, iterations=4000) if precision == "mixed" else {}
        return _case(kind, (lo, rng.randint(lo + 4, 24), rng.randint(0, 1000)), precision, min(frames, 2),
                     bodies=rng.randint(5, 96), jitter=0.0, **more)
    if kind == "hencky":
        return _case(kind, _cells(rng, 300, 12000), precision, frames, **PLASTIC)
    if kind in ("damped", "floating"):
        return _case(kind, _cells(rng, 100, 8000), precision, frames)
    if kind == "factor":
        return _case(kind, _cells(rng, 200, 1100), "fp64", frames, youngs=2e7, poisson=0.35)
    return _case(kind, _cells(rng, 200, 4096), "fp64", rng.randint(3, 10), law="snh", tolerance=1e-11, iterations=4000)


# ------------------------------------------------------------------------------------------------------- inputs --

@functools.lru_cache(maxsize=128)
def _box(cells, jitter, free, push):
    """A box of cubes, each split into six tets; nodes numbered as the cells first use them, base fixed unless `free`,
    top held too where it is pushed.  Rest positions are floats."""
    cx, cy, cz = cells
    k, j, i = (a.ravel() for a in np.meshgrid(np.arange(cz), np.arange(cy), np.arange(cx), indexing="ij"))
    bit = np.arange(8)
    corner = ((i[:, None] + (bit & 1)) * (cy + 1) + j[:, None] + ((bit >> 1) & 1)) * (cz + 1) + k[:, None] + (bit >> 2)
    sample, first, use = np.unique(corner.ravel(), return_index=True, return_inverse=True)
    order = np.argsort(first)
    rank = np.empty(order.size, np.int64)
    rank[order] = np.arange(order.size)
    node = rank[use].reshape(-1, 8)
    sample = sample[order]
    lattice = np.stack([sample // ((cy + 1) * (cz + 1)), sample // (cz + 1) % (cy + 1), sample % (cz + 1)], 1)
    rest = VOXEL * (lattice + jitter * np.random.default_rng(11).uniform(-1.0, 1.0, lattice.shape))
    rest = rest.astype(np.float32).astype(np.float64)
    tets = node[:, KUHN].reshape(-1, 4)
    edges = np.stack([rest[tets[:, c]] - rest[tets[:, 0]] for c in (1, 2, 3)], 2)
    flip = np.linalg.det(edges) < 0.0
    tets[flip, 1], tets[flip, 2] = tets[flip, 2].copy(), tets[flip, 1].copy()
    edges = np.stack([rest[tets[:, c]] - rest[tets[:, 0]] for c in (1, 2, 3)], 2)
    volume = np.linalg.det(edges) / 6.0
    mass = np.bincount(tets.ravel(), np.repeat(DENSITY * volume * 0.25, 4), rest.shape[0])
    anchored = np.zeros(rest.shape[0], np.uint8)
    prescribed = None
    if not free:
        anchored[lattice[:, 1] == 0] = 1
    if push:
        top = lattice[:, 1] == cy
        anchored[top] = 1
        prescribed = np.zeros_like(rest)
        prescribed[top, 1] = -0.5 * cy / 32.0
    return tb.PreparedMesh(rest_positions=rest, node_mass=mass, anchored=anchored, tet_nodes=tets.astype(np.uint32),
                           rest_inverse=np.linalg.inv(edges), volume=volume,
                           material=np.zeros(tets.shape[0], np.uint32), prescribed_velocity=prescribed)


def _smooth(rng, where, scale):
    """A smooth vector field over the unit box, of about `scale`."""
    out = np.zeros_like(where)
    for _ in range(3):
        wave = math.pi * rng.uniform(0.3, 1.5, 3)
        out += rng.uniform(-1.0, 1.0, 3) * np.sin(where @ wave + rng.uniform(0.0, 6.28))[:, None]
    return scale * out


@functools.lru_cache(maxsize=16)
def _bodies(kind, cx, cy, cz, bodies, jitter):
    """The meshes of a case."""
    if kind != "batch":
        return [_box((cx, cy, cz), jitter, kind == "floating", kind in ("plastic", "hencky", "factor"))]
    dims = np.random.default_rng(3 + cz).integers(cx, cy + 1, (bodies, 3))
    return [_box(tuple(int(c) for c in d), jitter, False, False) for d in dims]


def _inputs(case, seed):
    """Meshes, per-body materials and start states of a case."""
    rng = np.random.default_rng([seed, 17])
    kind = case["kind"]
    meshes = _bodies(kind, case["cx"], case["cy"], case["cz"], case["bodies"], case["jitter"])
    materials, states = [], []
    for mesh in meshes:
        youngs, poisson = case["youngs"] * math.exp(rng.uniform(-0.1, 0.1)), case["poisson"]
        if kind == "batch":
            youngs, poisson = math.exp(rng.uniform(math.log(1e5), math.log(1e8))), rng.uniform(0.25, 0.45)
        yields = kind in ("plastic", "hencky", "factor")
        materials.append([tb.PhysicalMaterial(
            density=DENSITY, youngs_modulus=youngs, poissons_ratio=poisson,
            stiffness_damping=0.02 if kind == "damped" else 0.0,
            yield_stress=1e5 if yields else math.inf, hardening_modulus=2e5 if yields else 0.0)])
        rest = mesh.rest_positions
        span = rest.max(0) - rest.min(0)
        unit = (rest - rest.min(0)) / span
        free = np.ones((mesh.nodes, 1))
        if kind != "floating":
            free = unit[:, 1:2] * (1.0 - unit[:, 1:2]) if mesh.prescribed_velocity is not None else unit[:, 1:2]
        size = float(span.max())
        moved = free * _smooth(rng, unit, (2e-4 if yields else 2e-3) * size)
        velocity = free * _smooth(rng, unit, 0.1)
        acceleration = free * _smooth(rng, unit, 0.5)
        if yields:  # pushed to about its yield strain
            moved[:, 1] -= rng.uniform(0.004, 0.007) * rest[:, 1]
            velocity[:, 1] -= 0.5 * span[1] / 3.2 * unit[:, 1]
        if kind == "floating":
            spin, arm = rng.uniform(-2.0, 2.0, 3), rest - rest.mean(0)
            velocity += rng.uniform(-1.0, 1.0, 3) + np.cross(spin, arm)
            acceleration += np.cross(spin, np.cross(spin, arm)) + GRAVITY
        held = mesh.anchored != 0
        velocity[held] = 0.0 if mesh.prescribed_velocity is None else mesh.prescribed_velocity[held]
        acceleration[held] = 0.0
        state = tb.DeformableState(rest + moved, velocity, acceleration, np.tile(np.eye(3), (mesh.tets, 1, 1)),
                                   np.zeros((mesh.tets, 10)))
        if kind == "hencky":
            state.plastic[:, [0, 4, 8]] = 1.0
        if case["precision"] == "mixed":  # what a caller with float buffers holds
            state.position, state.velocity, state.acceleration = (
                a.astype(np.float32).astype(np.float64) for a in (state.position, state.velocity, state.acceleration))
        states.append(state)
    return meshes, materials, states


def _settings(case):
    return tb.Settings(law=tb.NEO_HOOKEAN if case["law"] == "snh" else tb.COROTATED, tolerance=case["tolerance"],
                       cg_iterations=case["iterations"])


def _slots(sizes, width, dtype):
    """One page-locked buffer, and each body's part of it."""
    whole = torch.zeros(sum(sizes) * width, dtype=dtype).pin_memory()
    parts, at = [], 0
    for n in sizes:
        parts.append(whole[at:at + n * width].view(n, width))
        at += n * width
    return whole, parts


def prepare(case, seed):
    meshes, materials, states = _inputs(case, seed)
    settings = _settings(case)
    kind = case["kind"]
    mixed = case["precision"] == "mixed"
    if kind == "host":
        return dict(kind=kind, mesh=meshes[0], material=materials[0], start=states[0], settings=settings)
    system = tb.System(meshes, materials, tb.FP32_MIXED if mixed else tb.FP64)
    if kind == "rollout":
        rng = np.random.default_rng([seed, 23])
        mesh = meshes[0]
        system.set_youngs(materials[0][0].youngs_modulus * np.exp(0.3 * rng.standard_normal(mesh.tets)))
        roll = tb.Rollout(system, case["frames"], checkpoint_every=5, newton_reads=4, settings=settings)
        return dict(kind=kind, system=system, roll=roll, start=states[0],
                    target=mesh.rest_positions + _smooth(rng, mesh.rest_positions, 0.02))
    if kind == "hencky":
        system.set_plasticity("hencky")
    if kind == "factor":
        system.use_factor(True)
    # the caller's state buffers, page-locked, in the precision it works in
    dtype = torch.float32 if mixed else torch.float64
    nodes, tets = [m.nodes for m in meshes], [m.tets for m in meshes]
    start, out = [], []
    fields = ("position", "velocity", "acceleration", "rotation", "plastic")
    for name, width in zip(fields, (3, 3, 3, 9, 10)):
        sizes = nodes if width == 3 else tets
        whole, parts = _slots(sizes, width, dtype)
        for part, state in zip(parts, states):
            part.copy_(torch.from_numpy(getattr(state, name).reshape(-1, width)))
        start.append((whole, parts))
        out.append(_slots(sizes, width, dtype))
    yields = kind in ("plastic", "hencky", "factor")
    sets, gets = [], []
    for b in range(len(meshes)):
        p = [parts[b].data_ptr() for _, parts in start]
        # a step writes the rotations before it reads them; a factor is made at those of the state
        sets.append((p[0], p[1], p[2], p[3] if kind == "factor" else None, p[4] if yields else None))
        gets.append(tuple(parts[b].data_ptr() for _, parts in out[:4]) + (out[4][1][b].data_ptr() if yields else None,))
    return dict(kind=kind, system=system, settings=settings, frames=case["frames"], start=start, out=out, sets=sets,
                gets=gets, dtype=capi.TL_DTYPE_F32 if mixed else capi.TL_DTYPE_F64,
                result=dict(zip(fields[:5 if yields else 4], (whole for whole, _ in out))))


def run(state):
    kind = state["kind"]
    if kind == "host":
        body = state["start"].copy()
        tb.step(state["mesh"], body, state["material"], state["settings"], GRAVITY, DT)
        return dict(position=body.position, velocity=body.velocity, acceleration=body.acceleration,
                    rotation=body.rotation)
    system = state["system"]
    if kind == "rollout":
        system.set_state(state["start"])
        state["roll"].forward()
        final = system.get_state()
        g = state["roll"].adjoint(2.0 * (final.position - state["target"]))
        return dict(position=final.position, velocity=final.velocity, youngs=g.youngs, v0=g.velocity, x0=g.position)
    lib, handle, context = capi.lib(), system.handle, system.context.handle
    for b, p in enumerate(state["sets"]):
        capi.check(lib.tl_state_set(handle, b, state["dtype"], *p), context)
    for _ in range(state["frames"]):
        system.step(state["settings"], GRAVITY, DT)
    for b, p in enumerate(state["gets"]):
        capi.check(lib.tl_state_get(handle, b, state["dtype"], *p), context)
    return state["result"]


def _sizes(case):
    if case["kind"] == "batch":
        dims = np.random.default_rng(3 + case["cz"]).integers(case["cx"], case["cy"] + 1, (case["bodies"], 3))
    else:
        dims = np.array([[case["cx"], case["cy"], case["cz"]]])
    return int((dims + 1).prod(1).sum()), int(6 * dims.prod(1).sum())


def work(case):
    """What a pass cannot do without.  Per frame: each element's rest shape, volume, nodes and lane and its
    committed state read once and its new state written; each node's state read and written; the operator's 3x3 node
    blocks (15 a node on a Kuhn lattice) read once by each of the solve's iterations, counted as 3 solves of 20
    iterations, the least that these settings take."""
    V, T = _sizes(case)
    s = 4 if case["precision"] == "mixed" else 8
    blocks = 15 * V
    frames = case["frames"] * (6 if case["kind"] == "rollout" else 1)
    iterations = 60
    per = T * (72 + 8 + 20 + 9 * s + 20 * s) + V * 22 * s + iterations * (blocks * (9 * s + 4) + 6 * V * s)
    return dict(bytes=frames * per, flops=frames * (iterations * (blocks * 18 + V * 40) + 3 * T * 1500))


# -------------------------------------------------------------------------------------------------------- exact --
# The same step restated in 64 bits with torch alone: element laws, generalized-alpha, the three linearised reads or
# the plastic Newton loop, block-Jacobi (or factored) conjugate gradients with the same stops.

def _vdot(a, b):
    return (a * b).sum(-1)


def _cross(a, b):
    a, b = torch.broadcast_tensors(a, b)
    return torch.linalg.cross(a, b)


def _outer(a, b):
    return a.unsqueeze(-1) * b.unsqueeze(-2)


def _dev3(m):
    return m - m.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3.0 * torch.eye(3, dtype=m.dtype, device=m.device)


def _trace(m):
    return m.diagonal(dim1=-2, dim2=-1).sum(-1)


def _cof(m):
    c = [m[..., :, k] for k in range(3)]
    return torch.stack([_cross(c[1], c[2]), _cross(c[2], c[0]), _cross(c[0], c[1])], -1)


def _inv3(m):
    cof = _cof(m)
    return cof.transpose(-1, -2) / _vdot(m[..., :, 0], cof[..., :, 0])[..., None, None]


def _det3(m):
    return _vdot(m[..., :, 0], _cross(m[..., :, 1], m[..., :, 2]))


def _polar(f):
    r = f
    for _ in range(24):
        n = 0.5 * (r + _inv3(r).transpose(-1, -2))
        done = float((n - r).abs().max()) < 1e-9
        r = n
        if done:
            break
    return r


class _Exact:
    """Bodies of one case side by side, with their scalars per body."""

    def __init__(self, case, meshes, materials, states):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, d=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=d, device=dev)  # noqa: E731
        cat = lambda key: t(np.concatenate([np.asarray(getattr(m, key), np.float64) for m in meshes]))  # noqa: E731
        at = np.concatenate([[0], np.cumsum([m.nodes for m in meshes])])
        self.dev, self.case, self.counts = dev, case, t([m.nodes for m in meshes], torch.int64)
        self.B, self.V, self.T = len(meshes), int(at[-1]), sum(m.tets for m in meshes)
        self.rest, self.mass = cat("rest_positions"), cat("node_mass")
        self.held = cat("anchored") != 0
        self.free = (~self.held).double()[:, None]
        self.tets = t(np.concatenate([m.tet_nodes.astype(np.int64) + int(at[i]) for i, m in enumerate(meshes)]),
                      torch.int64)
        self.rinv, self.volume = cat("rest_inverse"), cat("volume")
        self.prescribed = torch.zeros_like(self.rest)
        if meshes[0].prescribed_velocity is not None:
            self.prescribed = cat("prescribed_velocity")
        def lane(f):
            return t(np.concatenate([np.full(m.tets, f(mat[0])) for m, mat in zip(meshes, materials)]))
        self.youngs, nu = lane(lambda m: m.youngs_modulus), lane(lambda m: min(max(m.poissons_ratio, 0.0), 0.49))
        self.nu = nu
        self.set_youngs(self.youngs)
        self.tau = materials[0][0].stiffness_damping
        self.yield_stress, self.hardening = materials[0][0].yield_stress, materials[0][0].hardening_modulus
        self.hencky, self.snh = case["kind"] == "hencky", case["law"] == "snh"
        self.yields = math.isfinite(self.yield_stress) and not self.hencky and not self.snh
        self.floating = case["kind"] == "floating"
        self.x, self.v, self.a = (t(np.concatenate([getattr(s, k) for s in states]))
                                  for k in ("position", "velocity", "acceleration"))
        self.plastic = t(np.concatenate([s.plastic for s in states]))
        self.rotation = torch.eye(3, dtype=torch.float64, device=dev).expand(self.T, 3, 3).clone()
        self.eye = torch.eye(3, dtype=torch.float64, device=dev)
        spectral = 0.5
        self.am, self.af = (2 * spectral - 1) / (spectral + 1), spectral / (spectral + 1)
        self.gamma = 0.5 - self.am + self.af
        self.beta = 0.25 * (1 - self.am + self.af) ** 2
        self.inertia = 1.0 - self.am
        self.factor = None
        self._pattern()

    def set_youngs(self, youngs):
        self.youngs, nu = youngs, self.nu
        self.lam, self.mu = youngs * nu / ((1 + nu) * (1 - 2 * nu)), youngs / (2 * (1 + nu))

    def _pattern(self):
        """Rows and columns of the 3x3 blocks, and where each element's 16 blocks go."""
        a = self.tets[:, :, None].expand(-1, 4, 4).reshape(-1)
        b = self.tets[:, None, :].expand(-1, 4, 4).reshape(-1)
        keys, self.into = torch.unique(a * self.V + b, return_inverse=True)
        self.row, self.col = keys // self.V, keys % self.V
        width = torch.bincount(self.row, minlength=self.V)
        start = torch.cumsum(width, 0) - width
        k = torch.arange(self.row.numel(), device=self.dev) - start[self.row]
        three = torch.arange(3, device=self.dev)
        self.place = (9 * start[self.row] + 3 * k)[:, None, None] + (3 * width[self.row])[:, None, None] * three[:, None] + three
        crow = (9 * start)[:, None] + (3 * width)[:, None] * three
        self.crow = torch.cat([crow.reshape(-1), torch.tensor([9 * self.row.numel()], device=self.dev)])
        cols = torch.empty(9 * self.row.numel(), dtype=torch.int64, device=self.dev)
        cols[self.place.reshape(-1)] = (3 * self.col[:, None, None] + three).expand(-1, 3, 3).reshape(-1)
        self.ccol = cols
        self.on_diagonal = self.row == self.col

    def per_body(self, values):
        """Sum over each body's nodes."""
        if self.B == 1:
            return values.sum(0, keepdim=True)
        return torch.segment_reduce(values, "sum", lengths=self.counts)

    def spread(self, scalars):
        return torch.repeat_interleave(scalars, self.counts, output_size=self.V)[:, None]

    # element pass -------------------------------------------------------------------------------------------------
    def _rest(self):
        if not self.hencky:
            return self.rinv, self.volume
        p = self.plastic[:, :9].view(-1, 3, 3)
        return self.rinv @ p, self.volume / _det3(p)

    def _gradients(self, rinv):
        return torch.cat([-rinv.sum(1, keepdim=True), rinv], 1)

    def _deformation(self, at, rinv):
        c = at[self.tets]
        return torch.stack([c[:, 1] - c[:, 0], c[:, 2] - c[:, 0], c[:, 3] - c[:, 0]], 2) @ rinv

    def _return(self, strain, mapping):
        """J2 radial return: stress, normal, theta, thetaBar, excess, plastic, next point."""
        committed, equivalent0 = self.plastic[:, :9].view(-1, 3, 3), self.plastic[:, 9]
        elastic = strain - committed
        pressure = (self.lam + 2 * self.mu / 3) * _trace(elastic)
        trial = 2 * self.mu[:, None, None] * _dev3(elastic)
        norm = (trial * trial).sum((1, 2)).sqrt()
        equivalent = math.sqrt(1.5) * norm
        radius = self.yield_stress + self.hardening * equivalent0
        over = (equivalent > radius) & (norm > 0) & mapping
        g = torch.where(over, (equivalent - radius) / (3 * self.mu + self.hardening), torch.zeros_like(norm))
        normal = torch.where(over[:, None, None], trial / norm.clamp_min(1e-300)[:, None, None], torch.zeros_like(trial))
        theta = torch.where(over, 1 - 3 * self.mu * g / equivalent.clamp_min(1e-300), torch.ones_like(norm))
        bar = torch.where(over, 3 * self.mu / (3 * self.mu + self.hardening) - (1 - theta), torch.zeros_like(norm))
        stress = theta[:, None, None] * trial + pressure[:, None, None] * self.eye
        excess = torch.where(over, (equivalent - radius) / radius, torch.zeros_like(norm))
        point = torch.cat([(committed + (math.sqrt(1.5) * g)[:, None, None] * normal).reshape(-1, 9),
                           (equivalent0 + g)[:, None]], 1)
        return stress, normal, theta, bar, excess, over, point

    def elements(self, at, consistent, margin, mapping=True, operator=True):
        """Node forces, the element operators (without mass) and the tets that load; sets the rotations."""
        rinv, volume = self._rest()
        g = self._gradients(rinv)
        f = self._deformation(at, rinv)
        loading = 0
        if self.snh:
            h = f - self.eye
            cof, change = _cof(f), _trace(h) + _trace(_cof(h)) + _det3(h)
            stress = self.mu[:, None, None] * (h + h.transpose(1, 2) - _trace(h)[:, None, None] * self.eye - _cof(h)) + \
                ((self.lam + self.mu) * change)[:, None, None] * cof
            self.element_force = -volume[:, None, None] * (g @ stress.transpose(1, 2))
        else:
            self.rotation = r = _polar(f)
            u = r.transpose(1, 2) @ f - self.eye
            strain = 0.5 * (u + u.transpose(1, 2))
            normal = theta = bar = None
            if self.yields:
                stress, normal, theta, bar, excess, over, self.point = self._return(strain, mapping)
                loads = over & (excess > margin)
                loading = int(loads.sum())
                normal = torch.where(loads[:, None, None], normal, torch.zeros_like(normal))
                theta, bar = torch.where(loads, theta, torch.ones_like(theta)), torch.where(loads, bar, torch.zeros_like(bar))
            else:
                stress = self.lam[:, None, None] * _trace(strain)[:, None, None] * self.eye + 2 * self.mu[:, None, None] * strain
            self.element_force = -volume[:, None, None] * (g @ stress.transpose(1, 2) @ r.transpose(1, 2))
        force = torch.zeros_like(self.rest).index_add_(0, self.tets.reshape(-1), self.element_force.reshape(-1, 3))
        if not operator:
            return force, loading
        # blocks [T, a, b, row, col] of dF_a / dx_b, negated: stiffness
        if self.snh:
            axes = self.eye
            ke = torch.empty(self.T, 4, 4, 3, 3, dtype=torch.float64, device=self.dev)
            s = (self.lam + self.mu)
            for b in range(4):
                for k in range(3):
                    df = _outer(axes[k].expand(self.T, 3), g[:, b])
                    dc = [df[..., :, c] for c in range(3)]
                    fc = [f[..., :, c] for c in range(3)]
                    dcof = torch.stack([_cross(dc[1], fc[2]) + _cross(fc[1], dc[2]), _cross(dc[2], fc[0]) + _cross(fc[2], dc[0]),
                                        _cross(dc[0], fc[1]) + _cross(fc[0], dc[1])], -1)
                    dp = self.mu[:, None, None] * df + (s * change - self.mu)[:, None, None] * dcof + \
                        (s * (cof * df).sum((1, 2)))[:, None, None] * cof
                    ke[:, :, b, :, k] = volume[:, None, None] * (g @ dp.transpose(1, 2))
        else:
            lam, mu2 = self.lam, 2 * self.mu
            if consistent and self.yields:
                mu2 = mu2 * theta
                lam = (self.lam + 2 * self.mu / 3) - mu2 / 3
            gr = g @ r.transpose(1, 2)
            ga, gb = gr[:, :, None, :], gr[:, None, :, :]
            w = volume[:, None, None, None, None]
            ke = w * (lam[:, None, None, None, None] * _outer(ga, gb) + (0.5 * mu2)[:, None, None, None, None] *
                      (_outer(gb, ga) + (ga * gb).sum(-1)[..., None, None] * self.eye))
            if consistent and self.yields:
                n = (r @ normal @ r.transpose(1, 2))
                ng = gr @ n
                ke = ke - w * (2 * self.mu * bar)[:, None, None, None, None] * _outer(ng[:, :, None, :].expand(-1, 4, 4, 3), ng[:, None, :, :].expand(-1, 4, 4, 3))
            self.damping = None
            if self.tau:
                arms = at[self.tets] - at[self.tets].mean(1, keepdim=True)
                tensor = ((arms * arms).sum((1, 2))[:, None, None] * self.eye) - arms.transpose(1, 2) @ arms
                inverse = _inv3(tensor)
                cr = torch.zeros(self.T, 4, 3, 3, dtype=torch.float64, device=self.dev)  # arms x
                cr[..., 0, 1], cr[..., 0, 2], cr[..., 1, 2] = -arms[..., 2], arms[..., 1], -arms[..., 0]
                cr = cr - cr.transpose(2, 3)
                # rigid part of unit motions: mean plus spin x arm
                rigid = 0.25 * self.eye.expand(self.T, 4, 4, 3, 3) - cr[:, :, None] @ inverse[:, None, None] @ cr[:, None, :]
                project = torch.eye(12, dtype=torch.float64, device=self.dev) - rigid.permute(0, 1, 3, 2, 4).reshape(-1, 12, 12)
                dense = ke.permute(0, 1, 3, 2, 4).reshape(-1, 12, 12)
                self.damping = self.tau * (project @ dense @ project.transpose(1, 2))
        self.ke = ke
        return force, loading

    def assemble(self, at, consistent=False, margin=0.0, mapping=True):
        """Forces at `at`; the system matrix and its block-Jacobi inverse stay on self."""
        force, loading = self.elements(at, consistent, margin, mapping)
        ke = self.reach * self.ke
        if self.tau:
            scale = (1 - self.af) * self.gamma * self.h
            ke = ke + scale * self.damping.view(-1, 4, 3, 4, 3).permute(0, 1, 3, 2, 4)
        blocks = torch.zeros(self.row.numel(), 3, 3, dtype=torch.float64, device=self.dev)
        blocks.index_add_(0, self.into, ke.reshape(-1, 3, 3))
        blocks[self.on_diagonal] += (self.inertia * self.mass)[:, None, None] * self.eye
        self.matrix_of(blocks)
        return force, loading

    def matrix_of(self, blocks):
        diagonal = blocks[self.on_diagonal]
        bad = self.held | ~(_det3(diagonal) > 0)
        self.jacobi = torch.where(bad[:, None, None], self.eye, _inv3(torch.where(bad[:, None, None], self.eye, diagonal)))
        keep = (~self.held[self.row] & ~self.held[self.col]).double()
        values = torch.empty(9 * self.row.numel(), dtype=torch.float64, device=self.dev)
        values[self.place.reshape(-1)] = (blocks * keep[:, None, None]).reshape(-1)
        self.matrix = torch.sparse_csr_tensor(self.crow, self.ccol, values, (3 * self.V, 3 * self.V))

    def product(self, p):
        return (self.matrix @ p.reshape(-1, 1)).view(-1, 3)

    def condition(self, r):
        if self.factor is None:
            return (self.jacobi @ r[:, :, None])[:, :, 0]
        turned = r @ self.frame
        solved = torch.cholesky_solve(turned.reshape(-1, 1), self.factor).view(-1, 3)
        return self.free * (solved @ self.frame.T)

    def cg(self, right, x, limit):
        """Conjugate gradients of every body with the reference's stops; (solution, iterations, capped) of body 0."""
        tiny = np.finfo(np.float64).tiny
        target = self.tolerance * self.per_body(_vdot(right, right)).sqrt().clamp_min(tiny)
        r = self.free * (right - self.product(x))
        z = self.condition(r)
        p, rz = z, self.per_body(_vdot(r, z))
        live = torch.ones(self.B, dtype=torch.bool, device=self.dev)
        taken = torch.zeros(self.B, dtype=torch.int64, device=self.dev)
        for _ in range(limit):
            live &= self.per_body(_vdot(r, r)).sqrt() > target
            if not bool(live.any()):
                break
            ap = self.product(p)
            curve = self.per_body(_vdot(p, ap))
            live &= (curve > 0) & (rz > 0)
            zero = torch.zeros_like(rz)
            step = self.spread(torch.where(live, rz / curve, zero))
            x, r = x + step * p, r - step * ap
            z = self.condition(r)
            after = self.per_body(_vdot(r, z))
            p = torch.where(self.spread(live.double()) > 0, z + self.spread(torch.where(live, after / rz, zero)) * p, p)
            rz = torch.where(live, after, rz)
            taken += live
        capped = bool((taken[0] == limit) & (self.per_body(_vdot(r, r)).sqrt()[0] > target[0]))
        return x, capped

    # the caller-held factor ---------------------------------------------------------------------------------------
    def refresh(self):
        self.elements_at_rest()
        full = torch.zeros(3 * self.V, 3 * self.V, dtype=torch.float64, device=self.dev)
        b = torch.zeros(self.row.numel(), 3, 3, dtype=torch.float64, device=self.dev)
        b.index_add_(0, self.into, self.reach * self.elastic.reshape(-1, 3, 3))
        b[self.on_diagonal] += (self.inertia * self.mass)[:, None, None] * self.eye
        keep = (~self.held[self.row] & ~self.held[self.col]).double()
        b = b * keep[:, None, None]
        b[self.on_diagonal] += self.held.double()[:, None, None] * self.eye
        three = torch.arange(3, device=self.dev)
        full[(3 * self.row[:, None, None] + three[:, None]).expand(-1, 3, 3), (3 * self.col[:, None, None] + three).expand(-1, 3, 3)] = b
        self.factor = torch.linalg.cholesky(full)
        self.made_at = self.x.clone()

    def elements_at_rest(self):
        gr = self._gradients(self.rinv) @ self.rotation.transpose(1, 2)
        ga, gb = gr[:, :, None, :], gr[:, None, :, :]
        five = lambda s: s[:, None, None, None, None]  # noqa: E731
        self.elastic = five(self.volume) * (five(self.lam) * _outer(ga, gb) + five(self.mu) * (
            _outer(gb, ga) + (ga * gb).sum(-1)[..., None, None] * self.eye))

    def turn_factor(self):
        m = self.mass[:, None]
        now = self.x - (m * self.x).sum(0) / m.sum()
        before = self.made_at - (m * self.made_at).sum(0) / m.sum()
        self.frame = _polar((m * now).T @ before)

    # the step -----------------------------------------------------------------------------------------------------
    def step(self):
        case = self.case
        limit, h = case["iterations"], DT
        self.tolerance = min(case["tolerance"], 1e-5) if self.floating else case["tolerance"]
        shift = lambda: self.x + h * self.v + (0.5 - self.beta) * h * h * self.a  # noqa: E731
        if not self.floating:
            w = (1 - self.af) * shift() + self.af * self.x
            if bool((_det3(self._deformation(w, self.rinv)) <= 0).any()):
                raise ValueError("a predicted inversion: the step would take substeps")
        self.h, self.reach = h, (1 - self.af) * self.beta * h * h
        if case["kind"] == "factor" and self.factor is None:
            self.refresh()
        if self.floating:
            body = self.floating_frame(h)
            arm = self.x - body["centre"]
            moving = self.v - body["velocity"] - _cross(body["spin"], arm)
            carried = self.a - body["acceleration"] - _cross(body["rate"], arm) - \
                _cross(body["spin"], _cross(body["spin"], arm)) - 2 * _cross(body["spin"], moving)
            shifted = arm + h * moving + (0.5 - self.beta) * h * h * carried
            weighted = (1 - self.af) * shifted + self.af * arm
            held, lag = body["mid_spin"], (1 - self.af) * (1 - self.gamma) * h
            drive = -self.mass[:, None] * (_cross(held, _cross(held, weighted)) + _cross(body["mid_rate"], weighted) +
                                           2 * _cross(held, moving + lag * carried))
            self.a, lagged = carried, moving
        else:
            carried, shifted = self.a, shift()
            weighted = (1 - self.af) * shifted + self.af * self.x
            drive = self.mass[:, None] * torch.tensor(GRAVITY, dtype=torch.float64, device=self.dev)
            lagged = self.v
        m = self.mass[:, None]

        def balance(force, taken):
            right = force + drive - self.am * m * carried
            if taken is not None:
                right = right - self.inertia * m * taken
            if self.tau:
                lag = (1 - self.af) * h
                vel = lagged + lag * (1 - self.gamma) * carried + (0 if taken is None else lag * self.gamma * taken)
                vel = self.free * vel
                pushed = (self.damping @ vel[self.tets].reshape(-1, 12, 1)).view(-1, 4, 3)
                right = right.index_add(0, self.tets.reshape(-1), -pushed.reshape(-1, 3))
            return self.free * right

        if self.factor is not None:
            self.turn_factor()

        def solve(right, start, refreshes):
            budget = min(32, limit) if self.factor is not None else limit
            x, capped = self.cg(right, start, budget)
            if capped and self.factor is not None and refreshes:
                self.refresh()
                self.frame = self.eye
                x, capped = self.cg(right, start, limit)
            return x

        zero = torch.zeros_like(self.x)
        if not (self.yields):
            force, _ = self.assemble(weighted)
            a = solve(balance(force, None), self.free * self.a, True)
            for _ in range(2):
                force, _ = self.assemble(weighted + self.reach * a)
                a = a + solve(balance(force, a), zero, False)
        else:
            a = self.newton(weighted, balance, solve)
        if self.floating:
            self.floating_end(body, a, shifted, moving, carried, h)
            return
        self.a = self.free * a
        self.v = torch.where(self.held[:, None], self.prescribed, self.v + h * ((1 - self.gamma) * carried + self.gamma * self.a))
        self.x = torch.where(self.held[:, None], self.x + h * self.prescribed, shifted + self.beta * h * h * self.a)
        if self.yields:
            rotation = self.rotation
            self.elements(self.x, False, 0.0, operator=False)
            self.plastic, self.rotation = self.point, rotation
        if self.hencky:
            self.hencky_flow()

    def newton(self, weighted, balance, solve):
        """The plastic loop: attempts with the consistent operator, halved steps, the hand-off to linear reads and the
        fallback."""
        margin, eps = 1e-3, float(np.finfo(np.float32).eps)
        travel = self.beta * self.h * self.h
        linear_allowed = True
        while True:
            total, step = torch.zeros_like(self.x), None
            accepted = lowest = math.inf
            best, opening, before, solves = total, 0.0, 0, 0
            converged = unloaded = handed = False
            for attempt in range(40):
                at = weighted + self.reach * total
                force, loading = self.assemble(at, attempt != 0, margin)
                right = balance(force, total)
                squared = float((right * right).sum())
                if attempt and (attempt == 1 or squared < lowest):
                    lowest, best = squared, total
                if attempt == 0:
                    unloaded = loading == 0
                if attempt == 1 and linear_allowed and unloaded and squared > accepted:
                    for _ in range(2):
                        force, loading = self.assemble(weighted + self.reach * total, False, margin)
                        if loading:
                            handed = True
                            break
                        total = total + solve(balance(force, total), torch.zeros_like(total), False)
                    converged = not handed
                    break
                if attempt and not squared <= accepted:
                    step = 0.5 * step
                    total = total - step
                    continue
                if attempt and before == 0 and loading == 0:
                    converged = True
                    break
                opening = squared if attempt == 0 else opening
                accepted, before = squared, loading
                step = self.free * solve(right, self.free * self.a if attempt == 0 else torch.zeros_like(total), attempt == 0)
                solves += 1
                total = total + step
                moved = float((self.free * step).norm(dim=1).max())
                extent = float((self.free * at).norm(dim=1).max())
                if solves > 1 and travel * moved <= 8.0 * eps * extent:
                    converged = True
                    break
            if handed:
                linear_allowed = False
                continue
            if not converged:
                total, back = torch.zeros_like(self.x), True
                for read in range(3):
                    force, loading = self.assemble(weighted + self.reach * total, False, margin, read != 0)
                    if loading:
                        back = False
                        break
                    total = total + self.free * solve(balance(force, total), self.free * self.a if read == 0 else torch.zeros_like(total), read == 0)
                if back:
                    force, loading = self.assemble(weighted + self.reach * total, False, margin)
                    right = balance(force, total)
                    back = loading == 0 and float((right * right).sum()) <= 1e-4 * opening
                if not back:
                    total = best
                    self.assemble(weighted + self.reach * total, True, margin)
            return total

    def hencky_flow(self):
        f = self._deformation(self.x, self.rinv)
        p, hard = self.plastic[:, :9].view(-1, 3, 3), self.plastic[:, 9]
        fe = f @ p

        def returned(yield_now):
            value, vector = (a.to(self.dev) for a in torch.linalg.eigh((fe @ fe.transpose(1, 2)).cpu()))
            strain = 0.5 * value.clamp_min(1e-300).log()
            dev = strain - strain.mean(1, keepdim=True)
            stress = math.sqrt(1.5) * 2 * self.mu * dev.norm(dim=1)
            scale = (dev * (yield_now / stress.clamp_min(1e-300) - 1)[:, None]).exp()
            return vector @ (scale[:, :, None] * vector.transpose(1, 2)) @ fe, stress

        start = self.yield_stress + self.hardening * hard
        _, stress = returned(start)
        ratio = self.hardening / (3 * self.mu)
        now = (start + ratio * stress) / (1 + ratio)
        after, _ = returned(now)
        mapped = (stress > start) & (stress > now) & (_det3(f) > 0)
        new = _inv3(f) @ after
        mapped &= (new - p).abs().sum((1, 2)) > 1e-12
        self.plastic = torch.where(mapped[:, None], torch.cat([new.reshape(-1, 9), (hard + (stress - now) / (3 * self.mu))[:, None]], 1), self.plastic)

    def floating_frame(self, h):
        m = self.mass[:, None]
        mean = lambda f: (m * f).sum(0) / m.sum()  # noqa: E731
        c, v, a = mean(self.x), mean(self.v), mean(self.a)
        arm = self.x - c
        tensor = (m * (arm * arm)).sum() * self.eye - (m * arm).T @ arm
        momentum, torque = (m * _cross(arm, self.v - v)).sum(0), (m * _cross(arm, self.a - a)).sum(0)
        inv = torch.linalg.inv(tensor)
        g = torch.tensor(GRAVITY, dtype=torch.float64, device=self.dev)
        after = (g - self.am * a) / (1 - self.am)

        def skew(s):
            z = torch.zeros((), dtype=torch.float64, device=self.dev)
            return torch.stack([torch.stack([z, -s[2], s[1]]), torch.stack([s[2], z, -s[0]]), torch.stack([-s[1], s[0], z])])

        def rate(l, t):
            s = inv @ l
            return _cross(l, s), t @ skew(s)

        def advance(l, t, span):
            d = span / 8
            for _ in range(8):
                a1, b1 = rate(l, t)
                a2, b2 = rate(l + 0.5 * d * a1, t + 0.5 * d * b1)
                a3, b3 = rate(l + 0.5 * d * a2, t + 0.5 * d * b2)
                a4, b4 = rate(l + d * a3, t + d * b3)
                l, t = l + d / 6 * (a1 + 2 * a2 + 2 * a3 + a4), t + d / 6 * (b1 + 2 * b2 + 2 * b3 + b4)
            for _ in range(3):
                t = 0.5 * (t + torch.linalg.inv(t).T)
            return l, t

        ml, mt = advance(momentum, self.eye, (1 - self.af) * h)
        el, et = advance(ml, mt, h - (1 - self.af) * h)
        spin = lambda l: inv @ l  # noqa: E731
        turn = lambda l: inv @ _cross(l, inv @ l)  # noqa: E731
        share = self.am / (1 - self.am)
        return dict(centre=c, velocity=v, acceleration=a, next_a=after,
                    next_c=c + h * v + h * h * ((0.5 - self.beta) * a + self.beta * after),
                    next_v=v + h * ((1 - self.gamma) * a + self.gamma * after),
                    momentum=momentum + h * (1 - self.gamma - self.gamma * share) * torque, torque=-share * torque,
                    spin=spin(momentum), rate=turn(momentum), mid_spin=spin(ml), mid_rate=turn(ml),
                    end_spin=et @ spin(el), end_rate=et @ turn(el), turn=et)

    def floating_end(self, body, a, shifted, moving, carried, h):
        m, span = self.mass[:, None], self.beta * h * h
        turned = a - (m * a).sum(0) / m.sum()
        placed = (shifted + span * turned) @ body["turn"].T
        moved = (moving + h * ((1 - self.gamma) * carried + self.gamma * turned)) @ body["turn"].T
        spin = body["end_spin"]
        reached = body["next_c"] + placed
        acc = body["next_a"] + _cross(body["end_rate"], placed) + _cross(spin, _cross(spin, placed)) + \
            2 * _cross(spin, moved) + turned @ body["turn"].T
        vel = body["next_v"] + _cross(spin, placed) + moved
        base = reached - span * acc
        tensor = (m * (placed * placed)).sum() * self.eye - (m * placed).T @ placed
        inv = torch.linalg.inv(tensor)
        restore = inv @ (body["momentum"] - (m * _cross(placed, vel - body["next_v"])).sum(0))
        settle = inv @ (body["torque"] - (m * _cross(placed, acc - body["next_a"])).sum(0))
        turning = _cross(settle, placed)
        self.v, self.a = vel + _cross(restore, placed), acc + turning
        self.x = base - span * turning + span * self.a
        self.rotation = body["turn"] @ self.rotation

    # the rollout's gradients --------------------------------------------------------------------------------------
    def rollout(self, steps, target):
        """Converged neo-Hookean steps and their adjoint."""
        h, kept = DT, []
        self.h, self.reach, self.tolerance = h, (1 - self.af) * self.beta * h * h, 1e-13
        m, c = self.mass[:, None], (0.5 - self.beta) * h * h
        g = torch.tensor(GRAVITY, dtype=torch.float64, device=self.dev)
        for _ in range(steps):
            x, v, a = self.x, self.v, self.a
            w = x + (1 - self.af) * (h * v + c * a)
            new = self.free * a
            for _ in range(7):
                force, _ = self.assemble(w + self.reach * new)
                right = self.free * (force + m * g - self.am * m * a - self.inertia * m * new)
                new = new + self.cg(right, torch.zeros_like(x), 4000)[0]
            kept.append(w + self.reach * new)
            self.a = self.free * new
            self.v = torch.where(self.held[:, None], self.prescribed, v + h * ((1 - self.gamma) * a + self.gamma * self.a))
            self.x = torch.where(self.held[:, None], x + h * self.prescribed, x + h * v + c * a + self.beta * h * h * self.a)
        dx = 2.0 * (self.x - target)
        dv, da = torch.zeros_like(dx), torch.zeros_like(dx)
        de = torch.zeros(self.T, dtype=torch.float64, device=self.dev)
        for at in reversed(kept):
            self.assemble(at)
            right = self.free * (self.beta * h * h * dx + h * self.gamma * dv + da)
            adj = self.cg(right, torch.zeros_like(dx), 4000)[0]
            corner = adj[self.tets]
            de += (self.element_force * corner).sum((1, 2)) / self.youngs
            pulled = (self.ke.permute(0, 1, 3, 2, 4).reshape(-1, 12, 12) @ corner.reshape(-1, 12, 1)).view(-1, 3)
            dw = torch.zeros_like(dx).index_add_(0, self.tets.reshape(-1), -pulled)
            fx, fv = dx, self.free * dv
            dx, dv, da = (fx + dw, self.free * h * fx + fv + (1 - self.af) * h * dw,
                          self.free * c * fx + h * (1 - self.gamma) * fv + (1 - self.af) * c * dw - self.am * m * adj)
        return dict(position=self.x, velocity=self.v, youngs=de, v0=dv, x0=dx)


def exact(case, seed):
    meshes, materials, states = _inputs(case, seed)
    kind = case["kind"]
    body = _Exact(case, meshes, materials, states)
    if kind == "rollout":
        rng = np.random.default_rng([seed, 23])
        youngs = materials[0][0].youngs_modulus * np.exp(0.3 * rng.standard_normal(meshes[0].tets))
        body.set_youngs(torch.as_tensor(youngs, device=body.dev))
        target = meshes[0].rest_positions + _smooth(rng, meshes[0].rest_positions, 0.02)
        out = body.rollout(case["frames"], torch.as_tensor(target, device=body.dev))
        return {k: x.cpu().numpy() for k, x in out.items()}
    for _ in range(case["frames"]):
        body.step()
    out = dict(position=body.x, velocity=body.v, acceleration=body.a, rotation=body.rotation)
    if kind in ("plastic", "hencky", "factor"):
        out["plastic"] = body.plastic
    if kind == "host":
        return {k: None if k == "rotation" and body.snh else x.cpu().numpy() for k, x in out.items()}
    out = {k: x.reshape(-1).cpu().numpy() for k, x in out.items()}
    if body.snh:  # the neo-Hookean law commits no rotation
        out["rotation"] = None
    return out
