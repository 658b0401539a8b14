"""What is timed when this framework's speed is compared: one pass of each case is one call of a
user's program through the public API (``ExplicitLoop``, ``BatchedLoop``, ``FEMRollout``, ``Server``)
and the read-back of what it computed.

Kinds
  loop     one FEM scene in an ExplicitLoop: ``steps`` substeps queued by one call (0: one
           ``advanceWithTime(1/60)`` frame), then positions and velocities; with ``energy`` also the
           FP64 energy report
  batch    many independent bodies, each on its own voxel grid, in one BatchedLoop
  rollout  FEMRollout: a differentiable rollout forward and backward, from and to CUDA tensors
  pile     disks in FEM-FEM contact with each other on a plane, in an ExplicitLoop
  rigids   a slab under a row of driven rigid primitives, in an ExplicitLoop
  serve    a burst of requests, one for each of a catalog of bodies, through the request loop

Meshes are structured triangulations of rectangles with jittered interior nodes (disks for the pile),
as in this repository's benchmark and tests; a seed gives the jitter, the initial velocities and the
grounds.  Scenes carry gravity and a ground, so that a state that is stepped on and on stays in
contact rather than flying off.
"""

import math

import numpy as np
import torch

import flatworld_b200 as fw
from flatworld_b200.batch import BatchedLoop
from flatworld_b200.diff import DiffSim, FEMRollout
from flatworld_b200.serve import Request, Server
from flatworld_b200.world import SceneLayout

FRAME = 1.0 / 60.0
ELASTIC, NEOHOOKEAN, MISES = "elastic", "neohookean", "mises"


def _loop(name, nx, ny, mat, ground, steps, E, rho, adaptive=True, dt=0.0, energy=False, damping=0.0):
    return {"name": name, "kind": "loop", "nx": nx, "ny": ny, "mat": mat, "ground": ground, "steps": steps,
            "E": E, "rho": rho, "adaptive": adaptive, "dt": dt, "energy": energy, "damping": damping}


def listed():
    return [
        # an interactive loop on a small body that reads the state back after every substep
        _loop("one substep, 2k triangles", 64, 16, ELASTIC, "plane", 1, 2e4, 40.0, False, 1e-4),
        # a frame of the same small body (the benchmark's plain small mesh), 167 substeps
        _loop("frame, 2k triangles", 64, 16, ELASTIC, "plane", 0, 2e4, 40.0, False, 1e-4),
        # a frame of an odd-sized elastoplastic body with damping, and the energy report that goes with it
        _loop("frame and energy, 16k triangles J2", 97, 83, MISES, "plane", 0, 5e4, 500.0, energy=True, damping=0.05),
        # a frame of the benchmark's large single mesh on a height field, adaptive dt
        _loop("frame, 131k triangles", 256, 256, NEOHOOKEAN, "heightfield", 0, 1e5, 100.0),
        # a single mesh that no longer fits on chip
        _loop("64 substeps, 655k triangles", 640, 512, NEOHOOKEAN, "heightfield", 64, 1e5, 100.0),
        # the ragged batch of the benchmark (100 to 20000 nodes per body, three materials, random voxel grids), an
        # eighth of it
        {"name": "batch, 256 ragged bodies", "kind": "batch", "bodies": 256, "lo": 100, "hi": 20000,
         "ground": "noise", "steps": 64, "own_dt": False},
        # many small bodies on voxel terrain, each with its own stable time step, one short frame
        {"name": "batch, 384 small bodies, own steps", "kind": "batch", "bodies": 384, "lo": 60, "hi": 400,
         "ground": "terrain", "steps": 48, "own_dt": True},
        # gradient of a rollout with respect to per-triangle moduli and initial velocities (64 x 64 quads, segments
        # of 50 substeps, as in the benchmark)
        {"name": "rollout gradient, 8k triangles", "kind": "rollout", "n": 64, "steps": 400, "every": 50},
        # disks landing on a plane and on each other
        {"name": "pile of 36 disks", "kind": "pile", "side": 6, "cells": 16, "steps": 64},
        # rolling, indenting and spinning rigids on a soft slab
        {"name": "slab under 12 rigids", "kind": "rigids", "nx": 128, "ny": 32, "rigids": 12, "steps": 64},
        # a burst of requests for bodies of different sizes and substep counts
        {"name": "48 requests", "kind": "serve", "bodies": 48, "lo": 100, "hi": 4000, "least": 50, "most": 400},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop"] * 5 + ["batch"] * 2 + ["rollout", "pile", "rigids", "serve"])
    if kind == "loop":
        nodes, aspect = _log(rng, 300, 250000), rng.uniform(0.25, 4.0)
        nx = max(3, int(round(math.sqrt(nodes * aspect))) - 1)
        ny = max(3, int(round(math.sqrt(nodes / aspect))) - 1)
        return {"kind": "loop", "nx": nx, "ny": ny, "mat": rng.choice([ELASTIC, NEOHOOKEAN, MISES]),
                "ground": rng.choice(["plane", "heightfield", "terrain"]),
                "steps": rng.choice([1, _log(rng, 2, 24), _log(rng, 25, 200)]), "E": rng.uniform(2e4, 1e5),
                "rho": rng.uniform(100.0, 500.0), "adaptive": True, "dt": 0.0, "energy": rng.random() < 0.2,
                "damping": rng.choice([0.0, 0.05])}
    if kind == "batch":
        bodies = _log(rng, 16, 384)
        return {"kind": "batch", "bodies": bodies, "lo": _log(rng, 50, 200), "hi": _log(rng, 300, 20000 if bodies < 200 else 2000),
                "ground": rng.choice(["noise", "terrain"]), "steps": _log(rng, 8, 64), "own_dt": rng.random() < 0.4}
    if kind == "rollout":
        return {"kind": "rollout", "n": _log(rng, 8, 72), "steps": _log(rng, 60, 300), "every": rng.choice([25, 40, 50])}
    if kind == "pile":
        return {"kind": "pile", "side": rng.randint(2, 6), "cells": rng.randint(8, 16), "steps": _log(rng, 8, 64)}
    if kind == "rigids":
        return {"kind": "rigids", "nx": rng.randint(40, 160), "ny": rng.randint(8, 40), "rigids": rng.randint(1, 12),
                "steps": _log(rng, 8, 64)}
    return {"kind": "serve", "bodies": rng.randint(4, 48), "lo": 100, "hi": _log(rng, 200, 4000), "least": 50,
            "most": rng.randint(100, 400)}


# ------------------------------------------------------------------ scenes


def _material(kind, E, nu, rho):
    if kind == ELASTIC:
        return fw.Elastic(E=E, nu=nu, rho=rho)
    if kind == NEOHOOKEAN:
        return fw.HyperElastic(E=E, nu=nu, rho=rho)
    return fw.MisesPlastic(E=E, nu=nu, rho=rho, sigma_y=0.02 * E, H=0.1 * E)


def _rows(xs, rng, amplitude):
    """Heights at xs: eight sinusoids of random phase, at most ``amplitude`` in sum."""
    amps = rng.uniform(0.5, 1.0, size=8)
    amps *= amplitude / amps.sum()
    return sum(a * np.sin(w * xs + p) for a, w, p in zip(amps, 2 * np.pi * rng.uniform(0.5, 6.0, 8), rng.uniform(0, 2 * np.pi, 8)))


def _voxels(rng, width, kind, cells=128, cell=0.02):
    """A square voxel grid below y = -0.01: occupied at random ("noise"), or filled up to a rough surface whose
    highest cell ends there ("terrain")."""
    extent = cells * cell
    lb = np.array([0.5 * (width - extent), -extent - 0.01], np.float32)
    if kind == "noise":
        occ = rng.random((cells, cells)) < 0.15
    else:
        top = np.cumsum(rng.integers(-1, 2, cells))
        top = cells - (top.max() - top)
        occ = np.arange(cells)[None, :] < np.maximum(top, cells // 2)[:, None]
    return fw.VoxelGridDomain(2, cells, cells, lb, lb + np.float32(extent), occupancy_np=occ.astype(np.int32))


def _body(rng, lo, hi, index, cell=0.01, rho=2000.0):
    """Body ``index`` of a catalog: a rectangle of 1 cm cells with a log-uniform node count, an aspect ratio of 1/4 to
    4 (both by the index, so that a catalog has the same sizes whatever the seed) and one of the three materials."""
    size = np.random.default_rng([index, 7])
    nodes, aspect = math.exp(size.uniform(math.log(lo), math.log(hi))), size.uniform(0.25, 4.0)
    nx, ny = (max(1, int(round(math.sqrt(v)) - 1)) for v in (nodes * aspect, nodes / aspect))
    conn, coords = fw.structured_rectangle(nx, ny, nx * cell, ny * cell, jitter=0.1, seed=int(rng.integers(1 << 30)))
    mat = _material((ELASTIC, NEOHOOKEAN, MISES)[index % 3], float(rng.uniform(1e4, 1e6)), float(rng.uniform(0.2, 0.45)), rho)
    return nx * cell, fw.FemDomain(fw.Mesh(2, conn, coords), fw.SolidProp(mat), [fw.Gravity([0.0, -9.8])],
                                   initials=[fw.InitialVel("ALL", [0.0, -float(rng.uniform(0.0, 0.5))])])


def _loop_scene(case, seed):
    rng = np.random.default_rng([seed, 1])
    nx, ny, ground = case["nx"], case["ny"], case["ground"]
    width, height = 1.0, ny / nx
    cell = width / nx
    conn, coords = fw.structured_rectangle(nx, ny, width, height, jitter=0.1, seed=int(rng.integers(1 << 30)))
    bcs = [fw.Gravity([0.0, -1.0 if case["rho"] < 50 else -9.8])]
    vel = [fw.InitialVel("ALL", [float(rng.uniform(-0.1, 0.1)), -0.5])]
    if ground == "plane":
        dom = fw.GroundDomain(2, [0.0, -0.25 * cell], [0.0, 1.0])
    elif ground == "heightfield":
        xs = np.linspace(-1.0, 2.0, 4096)
        h = _rows(xs, rng, 0.05)
        h -= h[(xs > 0.0) & (xs < width)].max() + 0.25 * cell
        dom = fw.HeightFieldDomain(2, h.astype(np.float32), lb=[-1.0, -1.0], ub=[2.0, 1.0])
    else:
        dom = _voxels(rng, width, "terrain")
    fem = fw.FemDomain(fw.Mesh(2, conn, coords), fw.SolidProp(_material(case["mat"], case["E"], 0.3, case["rho"])), bcs,
                       initials=vel)
    return [dom, fem]


def _batch_scenes(case, seed):
    scenes = []
    for i in range(case["bodies"]):
        rng = np.random.default_rng([seed, 2, i])
        width, fem = _body(rng, case["lo"], case["hi"], i)
        scenes.append([_voxels(rng, width, case["ground"]), fem])
    return scenes


def _served_body(case, seed, i):
    rng = np.random.default_rng([seed, 3, i])
    _, fem = _body(rng, case["lo"], case["hi"], i)
    return [fw.GroundDomain(2, [0.0, -0.002], [0.0, 1.0]), fem]


def _rollout_scene(case, seed):
    n = case["n"]
    conn, coords = fw.structured_rectangle(n, n, 0.4, 0.4, origin=(0.3, 0.002), jitter=0.1, seed=seed)
    fem = fw.FemDomain(fw.Mesh(2, conn, coords), fw.SolidProp(fw.HyperElastic(1e5, 0.3, 1000.0)), [fw.Gravity([0.0, -9.8])])
    return [fw.GroundDomain(2, [0.0, 0.0], [0.0, 1.0]), fem]


def _rollout_dt(case):
    return min(1e-4, 0.1 * (0.4 / case["n"]) / math.sqrt(1e5 / 1000.0))


def _pile_scene(case, seed):
    rng = np.random.default_rng([seed, 4])
    side, cells, radius = case["side"], case["cells"], 0.025
    conn, grid = fw.structured_rectangle(cells, cells, 2.0, 2.0, origin=(-1.0, -1.0))
    u, v = grid.astype(np.float64).T
    disk = radius * np.stack([u * np.sqrt(1.0 - 0.5 * v * v), v * np.sqrt(1.0 - 0.5 * u * u)], axis=1)
    conn = np.ascontiguousarray(conn[:, [0, 2, 1]])  # counter-clockwise: boundary normals point outward
    doms, pitch = [fw.GroundDomain(2, [0.0, 0.0], [0.0, 1.0])], 2 * radius * (1.0 - 2e-4)
    for r in range(side):
        for c in range(side):
            k = r * side + c
            at = np.array([radius + c * pitch + rng.uniform(0.0, 1e-5), radius + r * pitch])
            mat = _material((ELASTIC, NEOHOOKEAN)[k % 2], 1e5, 0.3, 1000.0)
            doms.append(fw.FemDomain(fw.Mesh(2, conn, (disk + at).astype(np.float32)), fw.SolidProp(mat),
                                     [fw.Gravity([0.0, -9.8])], friction=0.2))
    return doms


def _rigids_scene(case, seed):
    rng = np.random.default_rng([seed, 5])
    conn, coords = fw.structured_rectangle(case["nx"], case["ny"], 1.0, 0.25, jitter=0.1, seed=int(rng.integers(1 << 30)))
    slab = fw.FemDomain(fw.Mesh(2, conn, coords), fw.SolidProp(fw.HyperElastic(E=1e5, nu=0.3, rho=500.0)),
                        [fw.Gravity([0.0, -9.8])])
    doms = [fw.GroundDomain(2, [0.0, 0.0], [0.0, 1.0]), slab]
    for k in range(case["rigids"]):
        x = 0.06 + 0.08 * k
        if k % 3 == 0:  # balls that roll slowly enough to keep clear of the next primitive while they are timed
            doms.append(fw.RigidBodyDomain(fw.BallRigid(2, [x, 0.2745], 0.025, 0.5), [fw.EnforceVel([0], [1e-4, 0.0])], friction=0.2))
        elif k % 3 == 1:
            doms.append(fw.RigidBodyDomain(fw.BoxRigid(2, [x, 0.2745], [0.04, 0.05], [0.0], 1.0), [fw.FixedAll([0])]))
        else:
            doms.append(fw.RigidBodyDomain(fw.CapsuleRigid(2, [x - 0.02, 0.2695], [x + 0.02, 0.2695], [0.0], 0.02, 0.5),
                                           [fw.Fixed([0]), fw.EnforceRotVel([0], 0.01)], friction=0.1))
    return doms


# ------------------------------------------------------------------ prepare and run


class _Served:
    """A server with its catalog of bodies, resident after the first burst; closed with the state."""

    def __init__(self, case, seed):
        n = case["bodies"]
        rng = np.random.default_rng([seed, 6])
        self.substeps = [int(k) for k in rng.integers(case["least"], case["most"] + 1, n)]
        self.server = Server(lambda b: _served_body(case, seed, b), arena_nodes=2 * n * case["hi"], arena_elems=4 * n * case["hi"],
                             arena_bodies=n, arena_scenes=n)
        self.server.prepare(range(n))

    def __del__(self):
        self.server.close()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "loop":
        return case, fw.ExplicitLoop(case["dt"], _loop_scene(case, seed), useAdapativeDT=case["adaptive"], damping=case["damping"])
    if kind == "batch":
        loop = BatchedLoop(_batch_scenes(case, seed), dt=5e-5, useAdapativeDT=case["own_dt"])
        return case, loop
    if kind == "rollout":
        domains = _rollout_scene(case, seed)
        sim = DiffSim(domains, _rollout_dt(case), case["steps"], case["every"])
        g = torch.Generator(device="cuda").manual_seed(seed)
        young = 1e5 * torch.exp(0.3 * torch.randn(sim.E, generator=g, device="cuda") - 0.045)
        v0 = torch.randn(sim.N, 2, generator=g, device="cuda") * 0.01
        v0[:, 1] -= 1.0
        target = torch.from_numpy(domains[1].mesh.coords).cuda()
        return case, sim, young.requires_grad_(), v0.requires_grad_(), target
    if kind == "pile":
        doms = _pile_scene(case, seed)
        return case, fw.ExplicitLoop(0.3 * SceneLayout(doms).stableTime, doms, useAdapativeDT=False)
    if kind == "rigids":
        return case, fw.ExplicitLoop(0.0, _rigids_scene(case, seed))
    return case, _Served(case, seed)


def run(state):
    case, kind = state[0], state[0]["kind"]
    if kind in ("loop", "pile", "rigids"):
        loop = state[1]
        if case["steps"] == 0:
            loop.advanceWithTime(FRAME)
        elif case["steps"] == 1:
            loop.advance()
        else:
            loop.advance_n(case["steps"])
        fem = loop.femSpringManager
        out = {"x": fem.coords.numpy(), "v": fem.V.numpy()}
        if case.get("energy"):
            out["energy"] = np.array(list(loop.energy().values()))
        if kind == "rigids":
            out["rigid_x"] = loop.rigidManager.rigidParams.numpy()
        return out
    if kind == "batch":
        loop = state[1]
        if case["own_dt"]:
            loop.advanceWithTime(case["steps"] * 5e-5)
        else:
            loop.advance(case["steps"])
        return {"x": loop.all_coords(), "energy": loop.energies()}
    if kind == "rollout":
        _, sim, young, v0, target = state
        young.grad = v0.grad = None
        x = FEMRollout.apply(young, v0, sim)
        ((x - target) ** 2).sum().backward()
        return {"x": x.detach(), "young_grad": young.grad, "v0_grad": v0.grad}
    served = state[1]
    served.server.run([Request(0.0, i, i, n) for i, n in enumerate(served.substeps)], realtime=False)
    return {"x": np.concatenate([served.server.coords(b) for b in range(case["bodies"])])}


# ------------------------------------------------------------------ work


def _frame(frame_dt, step):
    """Substeps of one advanceWithTime(frame_dt): full steps and what is left."""
    out, rest = [], frame_dt
    while rest > 1e-12:
        out.append(max(min(step, rest), 1e-8))
        rest -= out[-1]
    return out


def _schedule(case, fem, ground):
    if case["steps"]:
        return [_stable(fem, ground) if case["adaptive"] else case["dt"]] * case["steps"]
    return _frame(FRAME, _stable(fem, ground) if case["adaptive"] else case["dt"])


def _stable(fem, ground):
    """The stable time of a body on a ground: the shortest edge over the wave speed, the penalty contact's period,
    and 1 ms where there is a plane."""
    mat, length = fem.prop.mat, fem.mesh.charLength
    penalty = 2.0 * mat.E / (3.0 * (1.0 - 2.0 * min(mat.nu, 0.4999)))
    out = min(0.4 * length / math.sqrt(mat.E / mat.rho), 0.9 * math.sqrt(mat.rho * length * length / 6.0 / penalty))
    return min(out, 1e-3) if isinstance(ground, fw.GroundDomain) else out


def _served_steps(fem, ground, asked):
    return max(asked, math.ceil(FRAME / (0.5 * _stable(fem, ground)) - 1e-9))


#: Operations of one triangle (strain, stress, corner forces) by material and of one node in a substep.
_FLOPS = {ELASTIC: 115, NEOHOOKEAN: 160, MISES: 150}
_NODE_FLOPS = 30


def work(case):
    kind = case["kind"]
    if kind == "loop":
        nodes, elems = (case["nx"] + 1) * (case["ny"] + 1), 2 * case["nx"] * case["ny"]
        dom, fem = None, None
        if case["steps"] == 0:
            dom, fem = _loop_scene(case, 0)
        steps = case["steps"] or len(_schedule(case, fem, dom))
        one = elems * _FLOPS[case["mat"]] + nodes * _NODE_FLOPS
        j2 = 32 if case["mat"] == MISES else 0
        return {"bytes": 44 * nodes + (40 + j2) * elems, "flops": one * steps}
    if kind == "batch":
        nodes = elems = flops = 0
        for i, (dom, fem) in enumerate(_batch_scenes(case, 0)):
            nodes += fem.nnodes
            elems += fem.nelements
            one = fem.nelements * _FLOPS[(ELASTIC, NEOHOOKEAN, MISES)[i % 3]] + fem.nnodes * _NODE_FLOPS
            flops += one * (len(_frame(case["steps"] * 5e-5, _stable(fem, dom))) if case["own_dt"] else case["steps"])
        return {"bytes": 44 * nodes + 51 * elems, "flops": flops}
    if kind == "rollout":
        nodes, elems = (case["n"] + 1) ** 2, 2 * case["n"] ** 2
        # forward, the segment again, and the reverse step (about twice a forward one)
        return {"bytes": 60 * nodes + 48 * elems, "flops": 4 * case["steps"] * (elems * _FLOPS[NEOHOOKEAN] + nodes * _NODE_FLOPS)}
    if kind == "pile":
        disks, cells = case["side"] ** 2, case["cells"]
        return {"bytes": disks * (44 * (cells + 1) ** 2 + 80 * cells * cells),
                "flops": case["steps"] * disks * (2 * cells * cells * 138 + (cells + 1) ** 2 * _NODE_FLOPS)}
    if kind == "rigids":
        nodes, elems = (case["nx"] + 1) * (case["ny"] + 1), 2 * case["nx"] * case["ny"]
        items = 2 * (case["nx"] + case["ny"]) * case["rigids"]
        return {"bytes": 44 * nodes + 40 * elems + 16 * items, "flops": case["steps"] * (elems * 160 + nodes * _NODE_FLOPS + 20 * items)}
    nodes = elems = flops = 0
    rng = np.random.default_rng([0, 6])
    for i, asked in enumerate(rng.integers(case["least"], case["most"] + 1, case["bodies"])):
        ground, fem = _served_body(case, 0, i)
        nodes += fem.nnodes
        elems += fem.nelements
        flops += _served_steps(fem, ground, int(asked)) * (fem.nelements * 140 + fem.nnodes * _NODE_FLOPS)
    return {"bytes": 44 * nodes + 51 * elems, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits


class _Wide:
    """Any number of bodies, each on a ground of its own, stepped in 64 bits with plain torch: the substep is
    gated penalty contact, P1 triangle forces, nodal damping and symplectic Euler."""

    def __init__(self, scenes, damping=0.0, young=None):
        f, dev = torch.float64, "cuda"
        self.damping = damping
        x, conn, body, bnd, v, g, nu, E, rho, kind = [], [], [], [], [], [], [], [], [], []
        n0 = 0
        for b, (_, fem) in enumerate(scenes):
            n, mat = fem.nnodes, fem.prop.mat
            x.append(fem.mesh.coords)
            conn.append(fem.mesh.connectivity.astype(np.int64) + n0)
            bnd.append(np.asarray(fem.mesh.boundaryNodes, np.int64) + n0)
            body.append(np.full(n, b))
            v.append(np.tile(fem.initials[0].vel if fem.initials else np.zeros(2, np.float32), (n, 1)))
            g.append(np.tile(np.float32(fem.bcs[0].g), (n, 1)))
            for to, value in ((nu, mat.nu), (E, mat.E), (rho, mat.rho), (kind, int(mat.type))):
                to.append(np.full(fem.nelements, value))
            n0 += n
        t = lambda a, dtype=f: torch.as_tensor(np.concatenate(a), device=dev).to(dtype)  # noqa: E731
        self.x, self.v, self.g = t(x), t(v), t(g)
        self.conn, self.body, self.bnd = t(conn, torch.int64), t(body, torch.int64), t(bnd, torch.int64)
        self.bodies = len(scenes)
        nu, rho = t(nu), t(rho)
        self.E = t(E) if young is None else young
        unit = self.E
        self.lam, self.mu = unit * nu / ((1 + nu) * (1 - 2 * nu)), unit / (2 * (1 + nu))
        kind = t(kind, torch.int64)
        self.sets = {k: torch.nonzero(kind == int(c.type))[:, 0] for k, c in
                     ((ELASTIC, fw.Elastic(1, 0, 1)), (NEOHOOKEAN, fw.HyperElastic(1, 0, 1)), (MISES, fw.MisesPlastic(1, 0, 1, 1)))}
        p = self.x[self.conn]
        dm = torch.stack([p[:, 0] - p[:, 2], p[:, 1] - p[:, 2]], dim=2)
        self.area, self.inv = 0.5 * torch.linalg.det(dm).abs(), torch.linalg.inv(dm)
        share = self.area * rho / 3
        self.mass = torch.zeros(len(self.x), dtype=f, device=dev).index_add_(0, self.conn.reshape(-1), share.repeat_interleave(3))
        self.plastic = torch.zeros(len(self.conn), 4, dtype=f, device=dev)
        first = [fem.prop.mat for _, fem in scenes]
        per_body = lambda vals: torch.tensor(vals, dtype=f, device=dev)  # noqa: E731
        self.penalty = per_body([2.0 * m.E / (3.0 * (1.0 - 2.0 * min(m.nu, 0.4999))) for m in first])
        sizes = [fem.nelements for _, fem in scenes]
        rep = torch.repeat_interleave(torch.arange(self.bodies, device=dev), torch.tensor(sizes, device=dev))
        self.yield_ = per_body([getattr(m, "sigma_y", 0.0) for m in first])[rep]
        self.hard = per_body([getattr(m, "H", 0.0) for m in first])[rep]
        boxes = [dom.getBBox() for dom, _ in scenes]
        self.lo, self.hi = (torch.tensor(np.stack([b[k] for b in boxes]), dtype=f, device=dev) for k in (0, 1))
        self.grounds = [dom for dom, _ in scenes]
        if isinstance(self.grounds[0], fw.VoxelGridDomain):
            self._free_cells()
        elif isinstance(self.grounds[0], fw.HeightFieldDomain):
            self.heights = torch.tensor(self.grounds[0].height, dtype=f, device=dev)
        self.count = torch.zeros(self.bodies, dtype=torch.int64, device=dev)

    def _free_cells(self):
        """Per cell of every grid the index of the nearest free cell to its left, right, below and above (-1 or the
        grid's size where there is none)."""
        occ = torch.tensor(np.stack([d.occ for d in self.grounds]), device="cuda")
        n = occ.shape[1]
        at = torch.arange(n, device="cuda")
        self.occ, self.free = occ, []
        for dim in (1, 2):
            shape = [1, n, 1] if dim == 1 else [1, 1, n]
            here = torch.where(occ == 0, at.view(shape), -1)
            self.free.append(torch.cummax(here, dim).values)
            there = torch.where(occ == 0, at.view(shape), n)
            self.free.append(torch.flip(torch.cummin(torch.flip(there, [dim]), dim).values, [dim]))
        par = [[float(np.float32(a)) for a in (d.lb[0], d.lb[1], d.dx, d.dz)] for d in self.grounds]
        self.grid = torch.tensor(par, dtype=torch.float64, device="cuda")

    def _contact(self, dt):
        """Penalty forces on the boundary nodes."""
        b = self.body[self.bnd]
        x, v = self.x[self.bnd], self.v[self.bnd]
        with torch.no_grad():
            lo = torch.full((self.bodies, 2), math.inf, dtype=x.dtype, device=x.device).scatter_reduce_(0, b[:, None].expand(-1, 2), x, "amin")
            hi = torch.full((self.bodies, 2), -math.inf, dtype=x.dtype, device=x.device).scatter_reduce_(0, b[:, None].expand(-1, 2), x, "amax")
            grown = torch.where(self.count % 100 == 0, 0.1, 0.0)[:, None]
            w, gw = grown * (hi - lo), grown * (self.hi - self.lo)
            gate = ((lo - w <= self.hi + gw) & (hi + w >= self.lo - gw)).all(1)[b]
        ground = self.grounds[0]
        if isinstance(ground, fw.GroundDomain):
            p = torch.tensor([[float(c) for c in d.point] for d in self.grounds], dtype=x.dtype, device=x.device)[b]
            n = torch.tensor([[float(c) for c in d.normal] for d in self.grounds], dtype=x.dtype, device=x.device)[b]
            depth = ((x - p) * n).sum(1)
            return torch.where((gate & (depth < 0))[:, None], -n * (self.penalty[b] * depth)[:, None], torch.zeros_like(x))
        if isinstance(ground, fw.HeightFieldDomain):
            m, lb, span = ground.nx, float(ground.lb[0]), float(ground.ub[0]) - float(ground.lb[0])
            s = ((x[:, 0] - lb) / span).clamp(0, 1) * (m - 1)
            i = s.floor().long()
            h = self.heights
            top = h[i] + (h[(i + 1).clamp(max=m - 1)] - h[i]) * (s - i)
            near = torch.floor(s + 0.5).long().clamp(0, m - 1)
            k0, k1 = (near - 1).clamp(min=0), (near + 1).clamp(max=m - 1)
            slope = (h[k1] - h[k0]) / (span / (m - 1) * (k1 - k0))
            n = torch.stack([-slope, torch.ones_like(slope)], 1)
            n = n / n.norm(dim=1, keepdim=True)
            depth = (x[:, 1] - top) * n[:, 1]
            inside = gate & (depth < 0)
        else:
            g = self.grid[b]
            cells = self.occ.shape[1]
            ij = torch.floor((x - g[:, :2]) / g[:, 2:]).long()
            inside = gate & ((ij >= 0) & (ij < cells)).all(1)
            i, j = ij.clamp(0, cells - 1).unbind(1)
            inside = inside & (self.occ[b, i, j] == 1)
            left, right, down, up = (t[b, i, j] for t in self.free)
            gap = torch.stack([x[:, 0] - (g[:, 0] + (left + 1) * g[:, 2]), g[:, 0] + right * g[:, 2] - x[:, 0],
                               x[:, 1] - (g[:, 1] + (down + 1) * g[:, 3]), g[:, 1] + up * g[:, 3] - x[:, 1]], 1)
            depth, face = gap.min(1)
            depth = -depth
            n = torch.tensor([[-1.0, 0.0], [1.0, 0.0], [0.0, -1.0], [0.0, 1.0]], dtype=x.dtype, device=x.device)[face]
            inside = inside & (depth < 0)
        k, vn = self.penalty[b], (v * n).sum(1)
        push = -k * depth - 0.5 * k * vn.clamp(max=0.0) * (dt[b] if dt.dim() else dt)
        return torch.where(inside[:, None], n * push[:, None], torch.zeros_like(x))

    def _stress(self):
        p = self.x[self.conn]
        F = torch.stack([p[:, 0] - p[:, 2], p[:, 1] - p[:, 2]], dim=2) @ self.inv
        C = F.transpose(1, 2) @ F
        S, eye = torch.zeros_like(C), torch.eye(2, dtype=C.dtype, device=C.device)
        for kind, at in self.sets.items():
            if not len(at):
                continue
            c, lam, mu = C[at], self.lam[at], self.mu[at]
            e = 0.5 * (c - eye)
            if kind == ELASTIC:
                s = lam[:, None, None] * (e[:, 0, 0] + e[:, 1, 1])[:, None, None] * eye + 2 * mu[:, None, None] * e
            elif kind == NEOHOOKEAN:
                inv = torch.linalg.inv(c)
                s = (lam * torch.log(torch.linalg.det(F[at])) - mu)[:, None, None] * inv + mu[:, None, None] * eye
            else:
                old = self.plastic[at]
                t = torch.stack([e[:, 0, 0], e[:, 1, 1], e[:, 0, 1]], 1) - old[:, :3]
                lt = lam * (t[:, 0] + t[:, 1])
                trial = torch.stack([lt + 2 * mu * t[:, 0], lt + 2 * mu * t[:, 1], 2 * mu * t[:, 2]], 1)
                mean = (trial[:, 0] + trial[:, 1]) / 3
                d = trial - torch.stack([mean, mean, torch.zeros_like(mean)], 1)
                vm = (d[:, 0] ** 2 + d[:, 1] ** 2 - d[:, 0] * d[:, 1] + 3 * d[:, 2] ** 2).sqrt()
                over = vm - (self.yield_[at] + self.hard[at] * old[:, 3])
                dg = over.clamp(min=0.0) / (3 * mu + self.hard[at])
                safe = torch.where(over > 0, vm, torch.ones_like(vm))
                back = d * (3 * mu * dg / safe)[:, None]
                flat = trial - back
                s = torch.stack([torch.stack([flat[:, 0], flat[:, 2]], 1), torch.stack([flat[:, 2], flat[:, 1]], 1)], 1)
                self.plastic[at] = old + torch.cat([d / safe[:, None] * dg[:, None], dg[:, None]], 1)
            S = S.index_put((at,), s)
        return F, S

    def step(self, dt):
        """One substep; ``dt`` a number, or one per body (0: the body rests)."""
        dt = torch.as_tensor(dt, dtype=torch.float64, device="cuda").float().double()
        f = torch.zeros_like(self.x).index_add(0, self.bnd, self._contact(dt))
        F, S = self._stress()
        P = -self.area[:, None, None] * (F @ S) @ self.inv.transpose(1, 2)  # column c: the force on corner c
        f = f.index_add(0, self.conn[:, 0], P[:, :, 0]).index_add(0, self.conn[:, 1], P[:, :, 1])
        f = f.index_add(0, self.conn[:, 2], -P[:, :, 0] - P[:, :, 1])
        a = self.g + (f - self.damping * self.v) / self.mass[:, None]
        h = dt if dt.dim() == 0 else dt[self.body][:, None]
        self.v = self.v + a * h
        self.x = self.x + self.v * h
        self.count = self.count + ((dt > 0).long() if dt.dim() else 1)

    def energies(self):
        """Per body: kinetic, strain, external, contact."""
        p = self.x[self.conn]
        F = torch.stack([p[:, 0] - p[:, 2], p[:, 1] - p[:, 2]], dim=2) @ self.inv
        C = F.transpose(1, 2) @ F
        e = 0.5 * (C - torch.eye(2, dtype=C.dtype, device=C.device))
        ep = self.plastic
        e = e - torch.stack([torch.stack([ep[:, 0], ep[:, 2]], 1), torch.stack([ep[:, 2], ep[:, 1]], 1)], 1)
        W = 0.5 * self.lam * (e[:, 0, 0] + e[:, 1, 1]) ** 2 + self.mu * (e * e).sum((1, 2))
        at = self.sets[NEOHOOKEAN]
        if len(at):
            lj = torch.log(torch.linalg.det(F[at]))
            W[at] = 0.5 * self.mu[at] * (C[at, 0, 0] + C[at, 1, 1] - 2) - self.mu[at] * lj + 0.5 * self.lam[at] * lj * lj
        out = torch.zeros(self.bodies, 4, dtype=torch.float64, device="cuda")
        out[:, 0].index_add_(0, self.body, 0.5 * self.mass * (self.v ** 2).sum(1))
        out[:, 1].index_add_(0, self.body[self.conn[:, 0]], self.area * W)
        out[:, 2].index_add_(0, self.body, -self.mass * (self.g * self.x).sum(1))
        keep, self.v = self.v, torch.zeros_like(self.v)
        lo, hi, self.lo, self.hi = self.lo, self.hi, self.lo - math.inf, self.hi + math.inf  # not gated
        c = self._contact(torch.zeros((), dtype=torch.float64, device="cuda"))
        self.lo, self.hi, self.v = lo, hi, keep
        b = self.body[self.bnd]
        out[:, 3].index_add_(0, b, 0.5 * (c ** 2).sum(1) / self.penalty[b])
        return out.cpu().numpy()


def _padded(t):
    """Node values as ExplicitLoop hands them out: in an array with room for at least 1024 more rows."""
    out = np.zeros((max(len(t) + 1024, 2048), 2))
    out[: len(t)] = t.cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "loop":
        scene = _loop_scene(case, seed)
        w = _Wide([scene], case["damping"])
        for dt in _schedule(case, scene[1], scene[0]):
            w.step(dt)
        out = {"x": _padded(w.x), "v": _padded(w.v)}
        if case["energy"]:
            e = w.energies()[0]
            out["energy"] = np.append(e, e.sum())
        return out
    if kind == "batch":
        scenes = _batch_scenes(case, seed)
        w = _Wide(scenes)
        if case["own_dt"]:
            plans = [_frame(case["steps"] * 5e-5, _stable(fem, dom)) for dom, fem in scenes]
            for k in range(max(len(p) for p in plans)):
                w.step([p[k] if k < len(p) else 0.0 for p in plans])
        else:
            for _ in range(case["steps"]):
                w.step(5e-5)
        return {"x": w.x.cpu().numpy(), "energy": w.energies()}
    if kind == "serve":
        scenes = [_served_body(case, seed, i) for i in range(case["bodies"])]
        asked = np.random.default_rng([seed, 6]).integers(case["least"], case["most"] + 1, case["bodies"])
        plans = [_frame(FRAME, FRAME / _served_steps(fem, dom, int(n))) for (dom, fem), n in zip(scenes, asked)]
        if max(len(p) for p in plans) > 4000:
            return None
        w = _Wide(scenes)
        for k in range(max(len(p) for p in plans)):
            w.step([p[k] if k < len(p) else 0.0 for p in plans])
        return {"x": w.x.cpu().numpy()}
    if kind == "rollout":
        _, fem = scene = _rollout_scene(case, seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        young = 1e5 * torch.exp(0.3 * torch.randn(fem.nelements, generator=g, device="cuda") - 0.045)
        v0 = torch.randn(fem.nnodes, 2, generator=g, device="cuda") * 0.01
        v0[:, 1] -= 1.0
        young, v0 = young.double().requires_grad_(), v0.double().requires_grad_()
        w = _Wide([scene], young=young)
        w.v, target = v0, w.x.clone()
        for _ in range(case["steps"]):
            w.step(_rollout_dt(case))
        ((w.x - target) ** 2).sum().backward()
        return {"x": w.x.detach(), "young_grad": young.grad, "v0_grad": v0.grad}
    return None  # friction between deformable bodies and rigids has no short plain form
