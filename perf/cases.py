"""The work a user of the framework has it do, as cases that can be timed and
compared: time steps of blobs and batches, the surface interactions between
blobs, the linear-solver plugin and the training step of the learned
preconditioner, each through the entry points a program calls.

Meshes are the synthetic spheres of ffea_gb300.mesh (Freudenthal-split grids at
a 1.25 nm cell); positions, moduli and RNG words come from the seed.  A step
case returns node positions (float64, as the state is held) and node
velocities in the arithmetic of its solve: float64 in FP64 precision, float32
in mixed precision, whose vectors are FP32.
"""
from __future__ import annotations

import ctypes
import dataclasses
import functools
import math

import numpy as np
import torch

from ffea_gb300 import _lib as L
from ffea_gb300 import learned
from ffea_gb300 import params as P
from ffea_gb300.mesh import make_blob, sphere_mesh
from ffea_gb300.partition import estimate_sizes
from ffea_gb300.surface import SSINT_TYPES, SurfaceSolver, surface_faces
from ffea_gb300.world import (PRECOND_JACOBI, PRECOND_LEARNED, PRECOND_TWO_LEVEL, ConjugateGradientSolver,
                              NoMassCGSolver, World)

CELL_NM = 1.25
PRECOND = {"jacobi": PRECOND_JACOBI, "two-level": PRECOND_TWO_LEVEL, "learned": PRECOND_LEARNED}
SOLVER = {"nomass": P.SOLVER_NOMASS, "mass": P.SOLVER_MASS, "lumped": P.SOLVER_LUMPED}
M1, M2 = 4294967087, 4294944443   # MRG32k3a's moduli


# ---------------------------------------------------------------- the cases
def _step(name, radii, steps=1, solver="nomass", precision="mixed", precond="learned"):
    return {"name": name, "kind": "step", "radii": " ".join(f"{r:g}" for r in radii), "steps": steps,
            "solver": solver, "precision": precision, "precond": precond}


def listed():
    return [
        # one protein domain of ~450 nodes, a step per call as a coupled program makes it: bound by latency
        _step("domain_5nm", [5.0]),
        # the plain FFEA method in FP64 with the mass solver on the 16^3-cell blob, 10 steps
        _step("mass_fp64_10nm_x10", [10.0], steps=10, solver="mass", precision="fp64", precond="jacobi"),
        # a mid-size protein complex, 4 steps between two looks at it
        _step("complex_20nm_x4", [20.0], steps=4),
        # FFEA's own method (Jacobi-PCG, inertialess) in mixed precision at an odd size
        _step("jacobi_16nm", [16.3], precond="jacobi"),
        # the single-blob throughput workload
        _step("blob_40nm", [40.0]),
        # a blob with more rows than the chip holds in registers
        _step("blob_50nm", [50.0]),
        # an ensemble of uneven blobs (radii 5-20 nm) in one batch
        _step("ensemble_16", [5.0, 5.6, 6.3, 7.1, 7.7, 8.4, 9.2, 10.1, 11.0, 12.2, 13.3, 14.6, 16.0, 17.2, 18.6, 20.0]),
        # replicas of one blob, an RNG stream each, for statistics
        _step("replicas_32x15nm", [15.0] * 32),
        # the Solver plugin on host arrays: the call FFEA's own Blob makes each step
        {"name": "plugin_15nm", "kind": "solve", "radius": 15.0, "solver": "nomass", "precision": "fp64"},
        # Lennard-Jones between (and within) two 20 nm blobs 0.6 nm apart
        {"name": "lj_20nm", "kind": "ssint", "radius": 20.0, "type": "lennard-jones", "gap": 0.6, "self": 1},
        # steric repulsion of two blobs pushed into each other
        {"name": "steric_8nm", "kind": "ssint", "radius": 8.0, "type": "steric", "gap": -0.6, "self": 0},
        # one training step of the learned preconditioner: forward, loss and backward
        {"name": "train_15nm", "kind": "train", "radius": 15.0},
    ]


def _log_u(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["single", "single", "single", "batch", "batch", "solve", "ssint", "train"])
    if kind == "single":
        r = round(_log_u(rng, 4.0, 46.0), 2)
        solver = rng.choice(["nomass", "nomass", "nomass", "mass", "lumped"])
        precision = rng.choice(["mixed", "mixed", "mixed", "fp64"])
        precond = rng.choice(["learned", "learned", "two-level", "jacobi"])
        if solver != "nomass" or precision == "fp64":
            precond = "jacobi"
        if precision == "fp64":
            r = min(r, round(rng.uniform(8.0, 24.0), 2))
        return dict(_step("", [r], steps=rng.randint(1, 10 if precision == "fp64" else 2) if r < 20 else 1, solver=solver, precision=precision,
                          precond=precond), name=f"single_{r}")
    if kind == "batch":
        if rng.random() < 0.5:
            r = round(_log_u(rng, 4.0, 20.0), 2)
            n = rng.randint(2, min(48, int(32 * (15.0 / r) ** 3)))
            radii = [r] * n
        else:
            n = rng.randint(2, 24)
            radii = [round(_log_u(rng, 4.0, 20.0), 2) for _ in range(n)]
        return dict(_step("", radii, precond=rng.choice(["learned", "learned", "jacobi"])), name=f"batch_{n}_{radii[0]}")
    if kind == "solve":
        return {"name": "solve", "kind": "solve", "radius": round(_log_u(rng, 4.0, 20.0), 2),
                "solver": rng.choice(["nomass", "mass"]), "precision": rng.choice(["fp64", "mixed"])}
    if kind == "ssint":
        t = rng.choice(["lennard-jones", "lennard-jones", "steric", "ljsteric", "gensoft"])
        steric = t != "lennard-jones"
        return {"name": "ssint", "kind": "ssint", "type": t, "self": rng.randint(0, 1),
                "radius": round(_log_u(rng, 4.0, 10.0 if steric else 20.0), 2),
                "gap": round(rng.uniform(-0.8, -0.3), 2) if steric else round(rng.uniform(0.4, 1.2), 2)}
    return {"name": "train", "kind": "train", "radius": round(_log_u(rng, 5.0, 25.0), 2)}


# ---------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=64)
def _rest_mesh(radius):
    return sphere_mesh(radius, cell_nm=CELL_NM, jitter=0.0)


def _mesh(radius, rng):
    """A sphere with its corner nodes jittered by N(0, 0.05 cell), edge nodes midway."""
    m = _rest_mesh(radius)
    pos = m.pos.copy()
    n = m.num_linear
    pos[:n] += rng.normal(0.0, 0.05 * m.cell, (n, 3))
    t = m.topology
    for k, (a, b) in enumerate(((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))):
        pos[t[:, 4 + k]] = 0.5 * (pos[t[:, a]] + pos[t[:, b]])
    return dataclasses.replace(m, pos=pos)


def _params(solver, precision):
    return P.SimulationParams.from_si(
        dt=1e-14, kT=P.kT_at(300.0) * P.MESO_ENERGY, epsilon=1e-6, max_iterations_cg=10000, rng_seed=1,
        solver=SOLVER[solver], precision=P.PRECISION_FP64 if precision == "fp64" else P.PRECISION_MIXED)


def _blobs(case, seed):
    """Per blob of a step case: its BlobSpec and the six words of its RNG stream."""
    rng = np.random.default_rng(seed)
    out = []
    radii = [float(r) for r in case["radii"].split()]
    for r in radii:
        g = rng.uniform(0.5, 2.0) if len(set(radii)) > 1 else 1.0
        spec = make_blob(_mesh(r, rng), _params(case["solver"], case["precision"]), shear_mod=3.7e8 * g,
                         bulk_mod=1.1e9 * g)
        out.append((spec, rng.integers(1, M2, 6, dtype=np.uint64)))
    return out


def _spheres(case, seed):
    """Two spheres `gap` nm apart along x, with their faces, in a periodic grid of 3 nm cells."""
    rng = np.random.default_rng(seed)
    r = case["radius"]
    meshes = [_mesh(r, rng), _mesh(r, rng)]
    rest = _rest_mesh(r)
    tri, apex = surface_faces(rest.pos, rest.topology, with_apex=True)
    n = rest.num_nodes
    # the spheres' facing points lie on the x axis: the distance between the outermost rest nodes is the gap
    width = float(rest.pos[:, 0].max() - rest.pos[:, 0].min())
    pos = np.concatenate([m.pos - rest.pos.mean(0) for m in meshes])
    pos[n:, 0] += width + P.nm(case["gap"])
    h = P.nm(3.0)
    grid = tuple(int(v) for v in 2 * np.ceil((pos.max(0) - pos.min(0)) / h))
    pos += 0.5 * h * np.array(grid) - pos.mean(0)
    emin = rng.uniform(0.5, 2.0, (2, 2))
    return dict(pos=pos, faces=np.concatenate([tri, tri + n]).astype(np.int32),
                apex=np.concatenate([apex, apex + n]).astype(np.int32),
                blob=np.repeat(np.arange(2, dtype=np.int32), len(tri)),
                ftype=rng.integers(0, 2, 2 * len(tri)).astype(np.int32), emin=0.5 * (emin + emin.T),
                rmin=np.full((2, 2), P.nm(1.0)), k0=np.full((2, 2), 0.3), h=h, grid=grid)


def _solve_inputs(case, seed):
    rng = np.random.default_rng(seed)
    spec = make_blob(_mesh(case["radius"], rng), _params(case["solver"], case["precision"]))
    return spec, rng.normal(0.0, 1.0, (spec.mesh.num_nodes, 3))


def _dptr(t):
    return ctypes.cast(t.data_ptr(), L._dp)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        blobs = _blobs(case, seed)
        mixed = case["precision"] == "mixed"
        w = World([s for s, _ in blobs], true_residual=mixed, preconditioner=PRECOND[case["precond"]])
        for i, (_, words) in enumerate(blobs):
            w.blob(i).set_rng_state(words)
        if case["precond"] == "learned":
            learned.apply(w, learned.load())
        n = sum(w.num_nodes)
        # the program's own device arrays, filled by get_nodes
        pos, vel = (torch.zeros(n, 3, dtype=torch.float64, device="cuda") for _ in range(2))
        return {"kind": kind, "world": w, "steps": case["steps"], "pos": pos, "vel": vel, "mixed": mixed}
    if kind == "solve":
        spec, rhs = _solve_inputs(case, seed)
        s = NoMassCGSolver() if case["solver"] == "nomass" else ConjugateGradientSolver()
        s.init(spec.mesh.pos, spec.mesh.topology, spec.material, spec.params, drag=spec.drag)
        return {"kind": kind, "solver": s, "rhs": rhs, "pos": spec.mesh.pos, "mixed": case["precision"] == "mixed"}
    if kind == "ssint":
        g = _spheres(case, seed)
        s = SurfaceSolver(len(g["pos"]), g["faces"], g["blob"], g["ftype"], g["emin"], g["rmin"], 2, g["h"], g["grid"],
                          inc_self=case["self"], ssint_type=SSINT_TYPES[case["type"]], face_apex=g["apex"],
                          steric_factor=50.0, steric_dr=5e-3, k0=g["k0"])
        pos = torch.tensor(g["pos"], device="cuda")
        return {"kind": kind, "solver": s, "pos": pos, "force": torch.zeros_like(pos),
                "energy": torch.zeros(2, 2, dtype=torch.float64, device="cuda")}
    rng = np.random.default_rng(seed)
    spec = make_blob(_mesh(case["radius"], rng), _params("nomass", "mixed"))
    w = World([spec], true_residual=True, preconditioner=PRECOND_LEARNED)
    w.blob(0).set_rng_state(rng.integers(1, M2, 6, dtype=np.uint64))
    # weights in the middle of a training run
    theta = learned.load() + rng.normal(0.0, 0.02, learned.NUM_PARAMS).astype(np.float32)
    learned.apply(w, theta)
    w.run(1)  # the solve whose (rhs, solution) pair is trained on
    return {"kind": kind, "world": w, "theta": theta}


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "step":
        w = state["world"]
        w.run(state["steps"])
        o = 0
        for i in range(w.num_blobs):
            n = w.num_nodes[i]
            L.check(L.lib().ffea_gpu_get_nodes(w.handle, i, _dptr(state["pos"][o:]), _dptr(state["vel"][o:]), None))
            o += n
        return {"pos": state["pos"], "vel": state["vel"].float() if state["mixed"] else state["vel"]}
    if kind == "solve":
        x = state["solver"].solve(state["rhs"].copy(), state["pos"])
        return {"x": x.astype(np.float32) if state["mixed"] else x}
    if kind == "ssint":
        s = state["solver"]
        s.forces_device(state["pos"].data_ptr(), state["force"].data_ptr(), state["energy"].data_ptr())
        pairs = s.synchronize()
        return {"force": state["force"], "energy": state["energy"], "pairs": pairs}
    loss, grad = learned.loss_grad(state["world"], state["theta"])
    return {"loss": np.float32(loss), "grad": grad}


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Each input read and each output written once; the arithmetic of the
    element forces, the assembly and the products of the solve."""
    kind = case["kind"]
    if kind == "step":
        b = f = 0.0
        t = 8 if case["precision"] == "fp64" else 4
        for r in (float(x) for x in case["radii"].split()):
            n, e, ed = estimate_sizes(r, CELL_NM)
            # per element: corners, rest inverse, volume, material; per node: position, velocity and drag in, and
            # position and velocity of every node (edge nodes too) out
            b += case["steps"] * (e * (16 + 10 * t + 2) + n * 56) + (n + ed) * 48
            iters = (1.6 * r if case["precond"] != "jacobi" else 5.2 * r) if case["solver"] == "nomass" else 20.0
            f += case["steps"] * (e * 400 + ed * 6 * 45 + iters * (18 * 2 * ed + 40 * n))
        return {"bytes": b, "flops": f}
    n, e, ed = estimate_sizes(case["radius"], CELL_NM)
    if kind == "solve":
        t = 8 if case["precision"] == "fp64" else 4
        iters = 5.2 * case["radius"] if case["solver"] == "nomass" else 20.0
        return {"bytes": (n + ed) * 72 + e * (16 + 10 * t + 2), "flops": ed * 6 * 45 + iters * (36 * ed + 40 * n)}
    faces = 7.2 * 4 * math.pi * (case["radius"] / CELL_NM) ** 2
    if kind == "ssint":
        pairs = faces * (30.0 if case["self"] else 2.0)
        return {"bytes": 2 * (n + ed) * 48 + faces * 20, "flops": pairs * (700.0 if case["type"] != "steric" else 20000.0)}
    # training step: the matrix, features and pair in, 4,737 gradients out; three layers of 32, forward and backward
    return {"bytes": (n + 2 * ed) * 36 + n * 24, "flops": 3.0 * 2 * n * (2 * 32 * 8 + 4 * 32 * 32 + 2 * 14 * 32)}


# ---------------------------------------------------------------- the same in 64 bits
def _mrg_draws(words, count):
    """`count` centred MRG32k3a draws: 2^k streams in step, each from its jump of the state."""
    per = 256
    lanes = max(1, -(-count // per))
    out = np.empty((per, lanes))
    A = ([[0, 1, 0], [0, 0, 1], [-810728 % M1, 1403580, 0]], [[0, 1, 0], [0, 0, 1], [-1370589 % M2, 0, 527612]])

    def mul(X, Y, m):
        return [[sum(X[i][k] * Y[k][j] for k in range(3)) % m for j in range(3)] for i in range(3)]

    state = []
    for c, m in enumerate((M1, M2)):
        J = [[int(i == j) for j in range(3)] for i in range(3)]
        B, e = A[c], per
        while e:
            if e & 1:
                J = mul(J, B, m)
            B, e = mul(B, B, m), e >> 1
        s = np.array([[int(w)] for w in words[3 * c:3 * c + 3]], dtype=np.uint64)
        while s.shape[1] < lanes:
            Ju = np.array(J, dtype=np.uint64)
            t = np.stack([sum((Ju[i, k] * s[k]) % np.uint64(m) for k in range(3)) % np.uint64(m) for i in range(3)])
            s = np.concatenate([s, t], axis=1)
            J = mul(J, J, m)
        state.append(s[:, :lanes].astype(np.int64))
    (a0, a1, a2), (b0, b1, b2) = state
    for i in range(per):
        p1 = (1403580 * a1 - 810728 * a0) % M1
        a0, a1, a2 = a1, a2, p1
        p2 = (527612 * b2 - 1370589 * b0) % M2
        b0, b1, b2 = b1, b2, p2
        out[i] = np.where(p1 > p2, p1 - p2, p1 - p2 + M1) * (1.0 / (M1 + 1.0)) - 0.5
    return out.T.reshape(-1)[:count]


class _Exact:
    """One blob in torch float64 on the GPU: element forces, matrix products and CG without preconditioning tricks."""

    def __init__(self, spec):
        dev = "cuda"
        m, p = spec.mesh, spec.params
        n = m.num_linear
        self.p, self.n, self.nt = p, n, m.num_nodes
        self.pos = torch.tensor(m.pos[:n], device=dev)
        self.vel = torch.zeros_like(self.pos)
        self.topo = torch.tensor(m.topology.astype(np.int64), device=dev)
        self.c = self.topo[:, :4].contiguous()
        self.mat = torch.tensor(spec.material, device=dev)
        self.drag = torch.tensor(spec.drag[:n], device=dev)
        self.J0, _, self.vol0 = self._shape(self.pos)
        self.J0i = torch.linalg.inv(self.J0)

    def _shape(self, pos):
        x = pos[self.c]
        J = x[:, 1:] - x[:, :1]                      # rows: edge vectors
        inv = torch.linalg.inv(J)                    # d psi_a / d x_i = inv[i, a - 1] for a = 1..3
        d = torch.cat([-inv.sum(2, keepdim=True), inv], 2)
        return J, d, torch.linalg.det(J).abs() / 6

    def _gather(self, f):
        out = torch.zeros(self.n, 3, dtype=torch.float64, device="cuda")
        return out.index_add_(0, self.c.reshape(-1), f.reshape(-1, 3))

    def _viscous(self, v, d):
        A, B = self.mat[:, 1, None, None], self.mat[:, 2, None, None]
        Lg = torch.einsum("eai,eja->eij", v[self.c], d)
        S = A * (Lg + Lg.transpose(1, 2))
        tr = B[:, 0, 0] * Lg.diagonal(dim1=1, dim2=2).sum(1)
        S.diagonal(dim1=1, dim2=2).add_(tr[:, None])
        return S

    def solve(self, b, pos):
        p = self.p
        if p.solver == P.SOLVER_LUMPED:
            m = torch.zeros(self.n, dtype=torch.float64, device="cuda")
            m.index_add_(0, self.c.reshape(-1), (0.25 * self.mat[:, 0] * self.vol0).repeat_interleave(4))
            return b / m[:, None]
        if p.solver == P.SOLVER_MASS:
            mv = (0.05 * self.mat[:, 0] * self.vol0)[:, None, None]

            def apply(v):
                w = v[self.c]
                return self._gather(mv * (w + w.sum(1, keepdim=True)))
            D = torch.zeros(self.n, dtype=torch.float64, device="cuda")
            D.index_add_(0, self.c.reshape(-1), (2 * mv[:, 0, 0]).repeat_interleave(4))
            D = D[:, None].expand(-1, 3)
        else:
            _, d, vol = self._shape(pos)

            def apply(v):
                S = self._viscous(v, d) * vol[:, None, None]
                return self._gather(torch.einsum("eij,eja->eai", S, d)) + self.drag[:, None] * v
            A, B = self.mat[:, 1, None, None], self.mat[:, 2, None, None]
            dd = (d * d).transpose(1, 2)
            D = self._gather(vol[:, None, None] * (A * (dd.sum(2, keepdim=True) + dd) + B * dd)) + self.drag[:, None]
        x, r = torch.zeros_like(b), b.clone()
        z = r / D
        q, g, stop = z.clone(), (r * z).sum(), 1e-24 * (b * b).sum()
        for k in range(5000):
            w = apply(q)
            a = g / (q * w).sum()
            x, r = x + a * q, r - a * w
            if k % 16 == 15 and bool((r * r).sum() < stop):
                break
            z = r / D
            g2 = (r * z).sum()
            q, g = z + (g2 / g) * q, g2
        return x

    def step(self, draws):
        p, mat = self.p, self.mat
        _, d, vol = self._shape(self.pos)
        x = self.pos[self.c]
        F = torch.einsum("eki,ejk->eij", x[:, 1:] - x[:, :1], self.J0i)
        G, E = mat[:, 3], mat[:, 4]
        S = (G * self.vol0 / vol)[:, None, None] * (F @ F.transpose(1, 2))
        up, dn = vol / self.vol0, self.vol0 / vol
        S.diagonal(dim1=1, dim2=2).add_((-G + G * (1 - dn) + 0.5 * (E - G * 2.0 / 3.0) * (up - dn))[:, None])
        ne = len(self.c)
        u = draws[:7 * ne].reshape(ne, 7)
        A, B = mat[:, 1], mat[:, 2]
        cf = torch.sqrt(24 * p.kT / (vol * p.dt))
        for k in range(3):
            S[:, k, k] += cf * (torch.sqrt(2 * A) * u[:, 1 + k] + torch.sqrt(B) * u[:, 0])
        for k, (i, j) in enumerate(((0, 1), (0, 2), (1, 2))):
            S[:, i, j] += cf * torch.sqrt(A) * u[:, 4 + k]
            S[:, j, i] = S[:, i, j]
        massive = p.solver != P.SOLVER_NOMASS
        if massive:
            S = S + self._viscous(self.vel, d)
        f = self._gather(-vol[:, None, None] * torch.einsum("eij,eja->eai", S, d))
        if massive:
            f = f - self.vel * self.drag[:, None]
        amp = torch.sqrt(24 * p.kT * self.drag / p.dt)
        f = f - draws[7 * ne:7 * ne + 3 * self.n].reshape(self.n, 3) * amp[:, None]
        x = self.solve(f, self.pos)
        self.vel = self.vel + x * p.dt if massive else x
        self.pos = self.pos + self.vel * p.dt

    def nodes(self):
        """Positions and velocities of every node, edge nodes midway and at rest."""
        pos, vel = (torch.zeros(self.nt, 3, dtype=torch.float64, device="cuda") for _ in range(2))
        pos[:self.n], vel[:self.n] = self.pos, self.vel
        for k, (a, b) in enumerate(((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))):
            pos[self.topo[:, 4 + k]] = 0.5 * (self.pos[self.topo[:, a]] + self.pos[self.topo[:, b]])
        return pos, vel


def _exact_step(case, seed):
    pos, vel = [], []
    for spec, words in _blobs(case, seed):
        e = _Exact(spec)
        per = 7 * len(e.c) + 3 * e.nt
        draws = torch.from_numpy(_mrg_draws(words, per * case["steps"])).cuda()
        for k in range(case["steps"]):
            e.step(draws[k * per:(k + 1) * per])
        p, v = e.nodes()
        pos.append(p)
        vel.append(v)
    return {"pos": torch.cat(pos), "vel": torch.cat(vel)}


def _exact_lj(g, inc_self):
    """The Lennard-Jones forces of every pair of faces in neighbouring cells whose normals do not agree."""
    dev = "cuda"
    pos = torch.tensor(g["pos"], device=dev)
    faces = torch.tensor(g["faces"].astype(np.int64), device=dev)
    blob = torch.tensor(g["blob"].astype(np.int64), device=dev)
    kind = torch.tensor(g["ftype"].astype(np.int64), device=dev)
    emin, rmin = torch.tensor(g["emin"], device=dev), torch.tensor(g["rmin"], device=dev)
    n = torch.tensor(g["grid"], device=dev)
    x = pos[faces]
    cr = torch.linalg.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
    mag = cr.norm(dim=1)
    area, normal = 0.5 * mag, cr / mag[:, None]
    cell = torch.floor((1.0 / 3.0) * (x[:, 0] + x[:, 1] + x[:, 2]) / g["h"]).long() % n
    eta = torch.full((3, 3), 0.166666666666667, dtype=torch.float64, device=dev)
    eta.fill_diagonal_(0.666666666666667)
    gauss = torch.einsum("ka,fad->fkd", eta, x)
    w2 = 0.333333333333333 ** 2
    force, energy, pairs = torch.zeros_like(pos), torch.zeros(2, 2, dtype=torch.float64, device=dev), 0
    nf = len(faces)
    for i0 in range(0, nf, 1024):
        i = torch.arange(i0, min(nf, i0 + 1024), device=dev)
        dc = (cell[i][:, None] - cell[None] + 1) % n
        ok = (dc <= 2).all(2) & (i[:, None] < torch.arange(nf, device=dev)[None])
        ok &= (normal[i][:, None] * normal[None]).sum(2) <= 0.0
        if not inc_self:
            ok &= blob[i][:, None] != blob[None]
        a, b = ok.nonzero(as_tuple=True)
        a = i[a]
        pairs += len(a)
        r = gauss[a][:, :, None] - gauss[b][:, None]
        # the pair's force matrix is symmetric: the entry (k, l > k) stands for (l, k) too
        up = torch.triu(torch.ones(3, 3, dtype=torch.bool, device=dev))
        rs = torch.where(up[None, :, :, None], r, r.transpose(1, 2))
        d = rs.norm(dim=3)
        e, r6 = emin[kind[a], kind[b]][:, None, None], rmin[kind[a], kind[b]][:, None, None] ** 6
        f6 = r6 / d ** 6
        fm = 12 * e * f6 * (f6 - 1) / d
        fv = (fm / d)[..., None] * rs
        s = (area[a] * area[b])
        energy.index_put_((blob[a], blob[b]), s * (w2 * e * f6 * (f6 - 2)).sum((1, 2)), accumulate=True)
        fa = w2 * torch.einsum("pkld,lj->pjd", fv, eta) * s[:, None, None]
        force.index_add_(0, faces[a].reshape(-1), fa.reshape(-1, 3))
        force.index_add_(0, faces[b].reshape(-1), -fa.reshape(-1, 3))
    return {"force": force, "energy": energy, "pairs": pairs}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _exact_step(case, seed)
    if kind == "solve":
        spec, rhs = _solve_inputs(case, seed)
        e = _Exact(spec)
        x = rhs.copy()
        x[:e.n] = e.solve(torch.tensor(rhs[:e.n], device="cuda"), e.pos).cpu().numpy()
        return {"x": x}  # edge nodes carry no drag: identity rows
    if kind == "ssint" and case["type"] == "lennard-jones":
        return _exact_lj(_spheres(case, seed), case["self"])
    # steric types: forward differences of clipped volumes, already computed in 64 bits;
    # training: the coarse space's aggregates are the library's own
    return None
