"""The workloads a user of pfem2_b200 runs, for timing and for comparing results.

`listed()` names them, `draw()` gives more of the same ranges, `prepare()` builds
what a driver holds before its time loop (mesh, boundary conditions, seeded
particles, an initial flow, pinned output buffers), `run()` is one turn of the
driver's time loop through pfem2_b200.solver, `work()` the bytes and operations
that turn cannot do without, and `exact()` the same turn in plain torch FP64.

Kinds:
  flow       one whole time step and a host read of its fields and loads
             (pfem2_step_and_read), on the 2D channel, the channel with a disk,
             the 3D pipe, or a batch of channels with disks
  members    the reference driver's own order, one pfem2Solver member after the
             other, with a read of fields, vorticity and particles
  particles  the particle kernels alone on a frozen velocity field, a snapshot
             every few steps
  moving     a time step of the moving-mesh driver: step, loads, mesh
             elasticity, mesh move

Solves stop at |r| <= 1e-11 |b|, as in tests/test_gpu_configs.py. Fields are
FP64 arrays; contexts with FP32 particles carry 24 bits in what they project,
so their fields are kept as FP32.
"""
import functools
import math

import numpy as np
import torch

from pfem2_b200 import _abi as A
from pfem2_b200 import cases as C
from pfem2_b200 import meshes as M
from pfem2_b200.solver import Solver

RTOL = 1e-11
CAPACITY = 4.0  # particle slots per seeded particle: a long run settles at about twice the seeded count
STAGES = {"fp64": (A.PREC_FP64, 0), "mixed": (A.PREC_MIXED, 0), "fp32": (A.PREC_MIXED, A.FP32_ALL)}
KRYLOV = {"cg": A.SOLVER_CG, "bicgstab": A.SOLVER_BICGSTAB}


def listed():
    return [
        # the smallest real flow: 1k cells, where launches and waits are all there is
        dict(name="channel_1k_fp64", kind="flow", mesh="channel", nx=64, ny=16, q=4, precision="fp64",
             vel="bicgstab"),
        # a driver that calls the members one by one, as the reference's run() does, and reads its particles
        dict(name="members_3k_fp64", kind="members", mesh="disk", cells=3300, q=4, precision="fp64", vel="cg"),
        # a coarse study of the benchmark's flow, CG for the velocity systems
        dict(name="disk_13k_cg_mixed", kind="flow", mesh="disk", cells=13000, q=5, precision="mixed", vel="cg"),
        # the benchmark's workload, in its default precision and in plain FP64
        dict(name="disk_52k_mixed", kind="flow", mesh="disk", cells=51653, q=5, precision="mixed", vel="bicgstab"),
        dict(name="disk_52k_fp64", kind="flow", mesh="disk", cells=51653, q=5, precision="fp64", vel="bicgstab"),
        # throughput mode: every stage that can run in FP32
        dict(name="disk_34k_fp32", kind="flow", mesh="disk", cells=34100, q=4, precision="fp32", vel="bicgstab"),
        # a parameter study: uneven instances advanced as one batch
        dict(name="ensemble_16_mixed", kind="flow", mesh="ensemble", n=16, lo=5000, hi=60000, q=5,
             precision="mixed", vel="bicgstab"),
        # 3D: a ragged small pipe in FP64 and the benchmark's pipe at half its resolution
        dict(name="pipe_10k_fp64", kind="flow", mesh="pipe", ny=13, nz=15, nx=53, q=3, precision="fp64",
             vel="bicgstab"),
        dict(name="pipe_131k_mixed", kind="flow", mesh="pipe", ny=32, nz=32, nx=128, q=3, precision="mixed",
             vel="bicgstab"),
        # the particle kernels alone: large in FP32, ragged and smaller in FP64
        dict(name="particles_1M_fp32", kind="particles", nx=1024, ny=1024, q=4, precision="fp32", steps=4),
        dict(name="particles_201k_fp64", kind="particles", nx=517, ny=389, q=3, precision="fp64", steps=4),
        # the oscillating-cylinder driver
        dict(name="moving_8k_mixed", kind="moving", mesh="disk", cells=8200, q=4, precision="mixed", vel="bicgstab"),
    ]


def draw(rng):
    size = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind = rng.choice(["channel", "disk", "disk", "pipe", "ensemble", "particles", "members", "moving"])
    precision = rng.choice(["fp64", "mixed", "mixed", "fp32"])
    vel = rng.choice(["bicgstab", "bicgstab", "cg"])
    if kind == "channel":
        ny = size(12, 110)
        return dict(kind="flow", mesh="channel", nx=ny * rng.randint(3, 5) - rng.randint(0, 3), ny=ny,
                    q=rng.randint(3, 5), precision=precision, vel=vel)
    if kind == "disk":
        return dict(kind="flow", mesh="disk", cells=size(2000, 60000), q=rng.randint(3, 5), precision=precision, vel=vel)
    if kind == "pipe":
        ny = size(8, 26)
        return dict(kind="flow", mesh="pipe", ny=ny, nz=max(8, min(26, ny + rng.randint(-3, 3))),
                    nx=ny * rng.randint(3, 4) + rng.randint(0, 3), q=rng.randint(2, 3), precision=precision, vel=vel)
    if kind == "ensemble":
        return dict(kind="flow", mesh="ensemble", n=rng.randint(3, 16), lo=size(2000, 6000), hi=size(8000, 50000),
                    q=rng.randint(3, 5), precision=precision, vel=vel)
    if kind == "particles":
        nx = size(200, 1000)
        return dict(kind="particles", nx=nx, ny=max(100, nx - rng.randint(0, 150)), q=rng.randint(3, 4),
                    precision=rng.choice(["fp32", "fp64"]), steps=rng.randint(2, 4))
    if kind == "members":
        return dict(kind="members", mesh="disk", cells=size(2000, 30000), q=rng.randint(3, 5),
                    precision=rng.choice(["fp64", "mixed"]), vel=vel)
    return dict(kind="moving", mesh="disk", cells=size(2000, 16000), q=rng.randint(3, 5),
                precision=rng.choice(["fp64", "mixed"]), vel=vel)


# ------------------------------------------------------------------ the driver's side
def _tight(spec, vel):
    spec.case.vel_tol = spec.case.p_tol = 0.0
    spec.case.vel_rtol = spec.case.p_rtol = RTOL
    spec.case.vel_solver = KRYLOV[vel]
    if spec.case.load_patch_id < 0:
        spec.case.load_patch_id = 0  # no body in the flow: the loads on the inlet
    return spec


@functools.lru_cache(maxsize=16)
def _specs(key):
    """the meshes and boundary conditions of a case (a driver reads its mesh from a file)"""
    c = dict(key)
    q = c["q"]
    if c["kind"] == "particles":
        mesh = M.rect_mesh(c["nx"], c["ny"])
        cs = C.make_case(mu=0.01, rho=1.0, dt=1.0, vel_bcs=[[], []], p_bcs=[], open_ids=(), load_patch=0)
        return [C.CaseSpec("particles", mesh, cs, (q, q), 0, 0.5 / q, 1)]
    if c["mesh"] == "channel":
        specs = [C.poiseuille_2d(nx=c["nx"], ny=c["ny"], q=(q, q))]
    elif c["mesh"] == "disk":
        specs = [C.channel_disk(h=math.sqrt(4.0 / c["cells"]), q=(q, q))]
    elif c["mesh"] == "pipe":
        specs = [C.pipe_3d(ny=c["ny"], nz=c["nz"], nx=c["nx"], q=(q, q, q))]
    else:
        specs = C.ensemble(n=c["n"], cells_lo=c["lo"], cells_hi=c["hi"], q=(q, q))
    return [_tight(s, c["vel"]) for s in specs]


def _case_specs(case):
    return _specs(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "precision", "steps"))))


def _initial_flow(spec, rng):
    """a developed-looking velocity with a seeded modulation, zero on the walls"""
    X = spec.mesh.vertices
    mod = 1.0 + 0.05 * np.sin(rng.uniform(1.0, 4.0) * X[:, 0] + rng.uniform(0.0, 6.0))
    if spec.mesh.dim == 3:
        r2 = (X[:, 1] ** 2 + X[:, 2] ** 2) / 0.25
        zero = np.zeros(len(X))
        return [np.maximum(0.0, 1.0 - r2) * mod, zero, zero]
    if spec.name == "poiseuille_2d":
        return [4.0 * X[:, 1] * (1.0 - X[:, 1]) * mod, np.zeros(len(X))]
    # potential flow around the disk under the inflow's parabola, damped to no slip at the disk
    dx, dy, R2 = X[:, 0] - 0.5, X[:, 1] - 0.5, spec.meta["radius"] ** 2
    d2 = np.maximum(dx * dx + dy * dy, R2)
    f = 1.5 * 4.0 * X[:, 1] * (1.0 - X[:, 1]) * (1.0 - (R2 / d2) ** 2) * mod
    return [f * (1.0 - R2 * (dx * dx - dy * dy) / d2 ** 2), -2.0 * f * R2 * dx * dy / d2 ** 2]


def _frozen_flow(spec, rng):
    """divergence-free random Fourier modes scaled to CFL 0.5 (dt = 1), as cases.frozen_stream_field"""
    ux, uy, _ = C.frozen_stream_field(spec.mesh, n_modes=8, seed=int(rng.integers(1 << 30)), cfl=0.5)
    return [ux, uy]


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    specs = _case_specs(case)
    flow = _frozen_flow if case["kind"] == "particles" else _initial_flow
    fields = [flow(s, rng) for s in specs]
    return specs, fields, int(rng.integers(1 << 31))


def _jitter(case, spec):
    return spec.jitter if case["kind"] == "particles" else 0.1


def prepare(case, seed):
    specs, fields, pseed = _inputs(case, seed)
    precision, stages = STAGES[case["precision"]]
    kind = case["kind"]
    s = Solver(specs, precision=precision, fp32_stages=stages, particles_only=kind == "particles",
               moving_mesh=kind == "moving", capacity_factor=CAPACITY)
    vel = (A.FIELD_VX, A.FIELD_VY, A.FIELD_VZ)[:s.dim]
    old = (A.FIELD_OLD_VX, A.FIELD_OLD_VY, A.FIELD_OLD_VZ)[:s.dim]
    pred = (A.FIELD_PRED_VX, A.FIELD_PRED_VY, A.FIELD_PRED_VZ)[:s.dim]
    for i, f in enumerate(fields):
        for d in range(s.dim):
            s.set_field(vel[d], f[d], i)
            s.set_field(old[d], f[d], i)
            if kind == "particles":
                s.set_field(pred[d], f[d], i)
    s.seed_particles(specs[0].q, pseed, _jitter(case, specs[0]))
    read = old if kind == "particles" else vel + (A.FIELD_P,)
    nv = [sp.mesh.n_vertices for sp in specs]
    pinned = lambda n: torch.zeros(n, dtype=torch.float64, pin_memory=True)  # noqa: E731
    state = {"case": case, "solver": s, "read": read, "loads": pinned(5 * len(specs)),
             "out": pinned(sum(nv) * len(read)), "turn": 0}
    if kind == "members":
        slots = int(CAPACITY) * s.n_particles()
        state["particles"] = [np.full(slots, -1, np.int32), np.zeros((slots, s.dim)), np.zeros((slots, s.dim))]
    return state


def _fields_out(st):
    out = st["out"]
    # FP32 particles: what they project has 24 bits
    return out.float() if st["case"]["precision"] == "fp32" else out


def run(state):
    s, kind = state["solver"], state["case"]["kind"]
    state["turn"] += 1
    if kind == "flow":
        s.step_and_read(state["read"], state["loads"].numpy(), state["out"].numpy())
        return {"fields": _fields_out(state), "loads": state["loads"]}
    if kind == "particles":
        for _ in range(state["case"]["steps"] - 1):
            s.step()
        s.step_and_read(state["read"], state["loads"].numpy(), state["out"].numpy())
        return {"fields": _fields_out(state)}
    if kind == "members":
        s.correct_particles_velocities()
        s.move_particles()
        s.distribute_particle_velocities_to_grid()
        s.fem_step()
        loads = s.calculate_loads(3)
        vort = s.calculate_vorticity()
        fields = [s.field(f) for f in state["read"]]
        cell, xi, u = state["particles"]
        n = _keep_particles(s.particles(), state["particles"])
        return {"fields": fields, "loads": loads, "vorticity": vort, "n": n, "cell": cell, "xi": xi, "u": u}
    s.step()
    loads = s.calculate_loads(3)
    s.problem_of_elasticity(1.0, 1.0, (1, 2, 4), 3, _body_step(state["turn"]), rtol=1e-12)
    s.move_mesh()
    return {"fields": [s.field(f) for f in state["read"]], "loads": loads,
            "displacement": [s.field(A.FIELD_DISP_X), s.field(A.FIELD_DISP_Y)], "vertices": s.vertices()}


def _keep_particles(got, slots):
    """the driver's own particle arrays, filled up to the count (cell -1 beyond it)"""
    n = len(got[0])
    for dst, src, rest in zip(slots, got, (-1, 0.0, 0.0)):
        dst[:n] = src
        dst[n:] = rest
    return n


def _body_step(turn):
    return [0.0, 0.0008 * math.cos(0.4 * turn)]


def work(case):
    """Bytes: the particle records and the nodal fields in and out once per step, and for a flow
    step each of its matrices (2 dim + 1 of them, with the shared columns) read once. Operations:
    interpolation, inverse map and projection per particle and sub-step, one product per matrix."""
    specs = _case_specs(case)
    nc = sum(s.mesh.n_cells for s in specs)
    nv = sum(s.mesh.n_vertices for s in specs)
    dim = specs[0].mesh.dim
    n_p = nc * case["q"] ** dim
    rb = 4 if case["precision"] == "fp32" else 8
    steps = case.get("steps", 1)
    nbytes = steps * (n_p * 2 * (4 + 2 * dim * rb) + nv * 8 * 3 * dim)
    flops = steps * n_p * 3 * 60 * dim
    if case["kind"] != "particles":
        nnz = nv * 3 ** dim
        nbytes += nnz * (4 + 8 * (2 * dim + 1)) + nv * 8 * 6 * dim
        flops += 2 * nnz * (2 * dim + 1)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ the same turn in plain torch FP64
class _Plain:
    """The PFEM2 step in FP64 torch: per-cell Q1 element matrices, Newton inverse maps, conjugate gradients."""

    def __init__(self, spec, case, fields, pseed):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        m, self.cs = spec.mesh, spec.case
        self.dim, self.nv, self.nc = m.dim, m.n_vertices, m.n_cells
        self.NV = 1 << self.dim
        t = lambda a, ty=torch.float64: torch.as_tensor(np.ascontiguousarray(a)).to(dev, ty)  # noqa: E731
        self.t, self.dev = t, dev
        self.X, self.cells, self.fb = t(m.vertices), t(m.cells, torch.int64), t(m.face_bid, torch.int64)
        self.bit = t([[(v >> d) & 1 for d in range(self.dim)] for v in range(self.NV)])
        self.S, self.most, self.q = spec.movement_steps, spec.max_per_part, case["q"]
        # cells around every vertex, ascending, padded with -1
        flat = self.cells.reshape(-1)
        order = torch.argsort(flat, stable=True)
        cnt = torch.bincount(flat, minlength=self.nv)
        first = torch.cumsum(cnt, 0) - cnt
        self.patch = torch.full((self.nv, int(cnt.max())), -1, dtype=torch.int64, device=dev)
        self.patch[flat[order], torch.arange(len(flat), device=dev) - first[flat[order]]] = order // self.NV
        self.V = [t(f) for f in fields]
        self.old = [v.clone() for v in self.V]
        self.P = torch.zeros(self.nv, dtype=torch.float64, device=dev)
        self.seed(pseed, _jitter(case, spec))

    # shape functions
    def N(self, xi):
        return torch.where(self.bit.bool(), xi[:, None, :], 1.0 - xi[:, None, :]).prod(2)

    def dN(self, xi):
        f = torch.where(self.bit.bool(), xi[:, None, :], 1.0 - xi[:, None, :])
        sign = 2.0 * self.bit - 1.0
        cols = []
        for d in range(self.dim):
            g = sign[:, d].expand(len(xi), -1).clone()
            for e in range(self.dim):
                if e != d:
                    g = g * f[:, :, e]
            cols.append(g)
        return torch.stack(cols, 2)  # [n, NV, dim]

    def at(self, cell, xi, F):
        N = self.N(xi)
        return torch.stack([(N * f[self.cells[cell]]).sum(1) for f in F], 1)

    def inverse(self, cell, x):
        """reference coordinates of x in its cell (Newton from the centre)"""
        Xc = self.X[self.cells[cell]]
        xi = torch.full_like(x, 0.5)
        for _ in range(12):
            F = (self.N(xi)[:, :, None] * Xc).sum(1)
            J = torch.einsum("nva,nvb->nab", Xc, self.dN(xi))
            step = self.solve_small(J, F - x)
            xi = xi - step
            xi = torch.clamp(xi, -1e3, 1e3)
            if len(xi) == 0 or float(step.abs().max()) < 1e-14:
                break
        return xi

    def solve_small(self, J, r):
        return torch.einsum("nab,nb->na", self.inv(J)[0], r)

    def inv(self, J):
        if self.dim == 2:
            a, b, c, d = J[:, 0, 0], J[:, 0, 1], J[:, 1, 0], J[:, 1, 1]
            det = a * d - b * c
            return torch.stack([d, -b, -c, a], 1).reshape(-1, 2, 2) / det[:, None, None], det
        c0, c1, c2 = J[:, :, 0], J[:, :, 1], J[:, :, 2]
        r0, r1, r2 = torch.cross(c1, c2, dim=1), torch.cross(c2, c0, dim=1), torch.cross(c0, c1, dim=1)
        det = (c0 * r0).sum(1)
        return torch.stack([r0, r1, r2], 1) / det[:, None, None], det

    # particles
    def seed(self, pseed, jitter):
        q, dim = self.q, self.dim
        Q = q ** dim
        t = np.arange(Q)
        idx = np.stack([t // q ** (dim - 1 - d) % q for d in range(dim)], 1)
        x = np.tile((idx + 0.5) * (1.0 / q), (self.nc, 1))
        if jitter:
            key = np.uint64(pseed * 0xD1B54A32D192ED03 % (1 << 64))
            with np.errstate(over="ignore"):
                for d in range(dim):
                    z = key + np.arange(self.nc * Q, dtype=np.uint64) * np.uint64(4) + np.uint64(d)
                    z = z + np.uint64(0x9E3779B97F4A7C15)
                    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
                    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
                    z = z ^ (z >> np.uint64(31))
                    x[:, d] += jitter * (2.0 * ((z >> np.uint64(11)).astype(np.float64) / 2.0 ** 53) - 1.0)
        self.xi = self.t(x)
        self.cell = torch.arange(self.nc, device=self.dev).repeat_interleave(Q)
        self.u = self.at(self.cell, self.xi, self.V)

    def correct(self):
        self.u = self.u + self.at(self.cell, self.xi, [v - o for v, o in zip(self.V, self.old)])

    def first_containing(self, x, cands, eps=0.0):
        """(cell or -1, reference coordinates) of the first candidate cell that contains x"""
        cell = torch.full((len(x),), -1, dtype=torch.int64, device=self.dev)
        xi = torch.zeros_like(x)
        for k in range(cands.shape[1]):
            todo = torch.nonzero((cell < 0) & (cands[:, k] >= 0))[:, 0]
            if len(todo) == 0:
                continue
            y = self.inverse(cands[todo, k], x[todo])
            ok = ((y >= -eps) & (y <= 1 + eps)).all(1)
            cell[todo[ok]] = cands[todo[ok], k]
            xi[todo[ok]] = y[ok]
        return cell, xi

    def move(self):
        live = torch.ones(len(self.cell), dtype=torch.bool, device=self.dev)
        centre = self.X[self.cells].mean(1)
        for _ in range(self.S):
            for lo in range(0, len(self.cell), 1 << 22):
                part = slice(lo, lo + (1 << 22))
                self._substep(part, live, centre)
        keep = torch.nonzero(live)[:, 0]
        keep = keep[torch.argsort(self.cell[keep], stable=True)]
        self.cell, self.xi, self.u = self.cell[keep], self.xi[keep], self.u[keep]

    def _substep(self, part, live, centre):
        cell, xi = self.cell[part], self.xi[part]
        u = self.at(cell, xi, self.V)
        xo = (self.N(xi)[:, :, None] * self.X[self.cells[cell]]).sum(1)
        xn = xo + u * (self.cs.dt / self.S)
        new = self.inverse(cell, xn)
        out = torch.nonzero(~((new >= 0) & (new <= 1)).all(1) & live[part])[:, 0]
        if len(out):
            unit = lambda a: a / a.norm(dim=-1, keepdim=True)  # noqa: E731
            Xc = self.X[self.cells[cell[out]]]
            v = (unit(Xc - xo[out][:, None]) * unit(u[out])[:, None]).sum(2).argmax(1)
            g = self.cells[cell[out], v]
            cand = self.patch[g]
            away = unit(xn[out] - self.X[g])
            dirs = unit(centre[cand.clamp(min=0)] - self.X[g][:, None])
            align = (dirs * away[:, None]).sum(2).masked_fill(cand < 0, -2.0)
            cand = torch.gather(cand, 1, torch.argsort(align, dim=1, descending=True, stable=True))
            c2, x2 = self.first_containing(xn[out], cand)
            lost = c2 < 0
            live[out[lost] + part.start] = False
            c2[lost], x2[lost] = cell[out][lost], xi[out][lost]
            cell[out] = c2
            new[out] = x2
        self.xi[part] = torch.where(live[part][:, None], new, xi)
        self.cell[part] = cell

    def check(self):
        q, dim, n = self.q, self.dim, len(self.cell)
        b = (self.xi / (1.0 / q)).to(torch.int64).clamp(0, q)
        key = self.cell
        for d in range(dim):
            key = key * (q + 1) + b[:, d]
        order = torch.argsort(key, stable=True)
        sk = key[order]
        start = torch.searchsorted(sk, sk, right=False)
        keep = torch.empty(n, dtype=torch.bool, device=self.dev)
        keep[order] = torch.arange(n, device=self.dev) - start < self.most
        full = torch.zeros(self.nc * (q + 1) ** dim, dtype=torch.bool, device=self.dev)
        full[key] = True
        inner = full.reshape((self.nc,) + (q + 1,) * dim)[(slice(None),) + (slice(0, q),) * dim]
        empty = torch.nonzero(~inner.reshape(self.nc, -1))
        idx = torch.stack([empty[:, 1] // q ** (dim - 1 - d) % q for d in range(dim)], 1).double()
        xn = (idx + 0.5) * (1.0 / q)
        un = self.at(empty[:, 0], xn, self.V)
        cell = torch.cat([self.cell[keep], empty[:, 0]])
        order = torch.argsort(cell, stable=True)
        self.cell = cell[order]
        self.xi = torch.cat([self.xi[keep], xn])[order]
        self.u = torch.cat([self.u[keep], un])[order]

    def add(self, vals):
        """[nc, NV] cell contributions summed into the vertices"""
        return torch.zeros(self.nv, dtype=torch.float64, device=self.dev).index_add_(
            0, self.cells.reshape(-1), vals.reshape(-1))

    def project(self):
        N = self.N(self.xi)
        g = self.cells[self.cell].reshape(-1)
        z = lambda v: torch.zeros(self.nv, dtype=torch.float64, device=self.dev).index_add_(0, g, v.reshape(-1))  # noqa: E731
        w = z(N)
        self.V = [torch.where(w != 0, z(N * self.u[:, d:d + 1]) / w, 0.0) for d in range(self.dim)]

    # finite elements
    def quad(self):
        """values at the QGauss(2) points of every cell: (N, gradients, weight x volume)"""
        pts = [0.21132486540518711775, 0.78867513459481288225]
        Xc = self.X[self.cells]
        for iq in range(self.NV):
            xi = self.t([[pts[(iq >> d) & 1] for d in range(self.dim)]])
            yield self._geometry(Xc, xi, 0.5 ** self.dim)

    def _geometry(self, Xc, xi, w):
        N, dN = self.N(xi)[0], self.dN(xi)[0]
        Ji, det = self.inv(torch.einsum("nva,vb->nab", Xc, dN))
        return N, torch.einsum("vb,nba->nva", dN, Ji), det * w, Ji, det

    def open_faces(self):
        """per open boundary face and face quadrature point: cells, N, gradients, n_x, weight"""
        pts = [0.21132486540518711775, 0.78867513459481288225]
        for f in range(2 * self.dim):
            ids = self.fb[:, f]
            on = torch.nonzero((ids >= 0) & ((self.cs.open_boundary_mask >> ids.clamp(min=0)) & 1 > 0))[:, 0]
            if len(on) == 0:
                continue
            ax, others = f // 2, [d for d in range(self.dim) if d != f // 2]
            for iq in range(1 << (self.dim - 1)):
                xi = [0.0] * self.dim
                xi[ax] = float(f & 1)
                for k, d in enumerate(others):
                    xi[d] = pts[(iq >> k) & 1]
                N, G, _, Ji, det = self._geometry(self.X[self.cells[on]], self.t([xi]), 1.0)
                n = Ji[:, ax, :] * (1.0 if f & 1 else -1.0)
                yield on, N, G, n[:, 0] / n.norm(dim=1), det * n.norm(dim=1) * 0.5 ** (self.dim - 1)

    def dirichlet(self, f):
        isd = torch.zeros(self.nv, dtype=torch.bool, device=self.dev)
        g = torch.zeros(self.nv, dtype=torch.float64, device=self.dev)
        for k in range(self.cs.n_dirichlet[f]):
            d = self.cs.dirichlet[f][k]
            v = self.boundary(d.boundary_id)
            isd[v] = True
            x = self.X[v, d.axis]
            g[v] = d.value * 4.0 * (x - d.a) * (d.b - x) / (d.b - d.a) ** 2 if d.kind == A.BC_PARABOLA else d.value
        return isd, g

    def boundary(self, bid):
        got = []
        for f in range(2 * self.dim):
            on = self.fb[:, f] == bid
            got.append(self.cells[on][:, self.bit[:, f // 2] == f % 2].reshape(-1))
        return torch.unique(torch.cat(got))

    def solve(self, Ae, dofs, n, b, isd, g):
        """conjugate gradients (diagonal preconditioner) on the assembled element matrices"""
        flat = dofs.reshape(-1)
        z = lambda: torch.zeros(n, dtype=torch.float64, device=self.dev)  # noqa: E731
        mul = lambda x: z().index_add_(0, flat, torch.bmm(Ae, x[dofs][:, :, None]).reshape(-1))  # noqa: E731
        diag = z().index_add_(0, flat, torch.diagonal(Ae, dim1=1, dim2=2).reshape(-1))
        free = (~isd).double()
        x = torch.where(isd, g, 0.0)
        ref = ((b - mul(x)) * free).norm()
        if float(ref) == 0.0:
            return x
        for _ in range(3):  # restarts from the true residual
            r = (b - mul(x)) * free
            zz = r / diag
            p, rz = zz.clone(), (r * zz).sum()
            for it in range(1, 20001):
                Ap = mul(p) * free
                al = rz / (p * Ap).sum()
                x = x + al * p
                r = r - al * Ap
                zz = r / diag
                rz, prev = (r * zz).sum(), rz
                p = zz + rz / prev * p
                if it % 20 == 0 and not float(r.norm()) > 1e-15 * float(ref):
                    break
            if not torch.isfinite(x).all():
                raise ArithmeticError("the reference solve broke down")
        return x

    def fem(self):
        cs, dim, NV, nc = self.cs, self.dim, self.NV, self.nc
        self.old = [v.clone() for v in self.V]
        zeros = lambda *s: torch.zeros(*s, dtype=torch.float64, device=self.dev)  # noqa: E731
        Me, Ke = zeros(nc, NV, NV), zeros(nc, NV, NV)
        Ce = [zeros(nc, NV, NV) for _ in range(dim)]
        rhs = [zeros(nc, NV) for _ in range(dim)]
        uc = [v[self.cells] for v in self.V]
        mdt = cs.mu * cs.dt
        for N, G, w, _, _ in self.quad():
            Me += torch.outer(N, N)[None] * w[:, None, None]
            for d in range(dim):
                Ce[d] += G[:, :, None, d] * G[:, None, :, d] * w[:, None, None]
            gr = [[(G[:, :, e] * uc[d]).sum(1) for e in range(dim)] for d in range(dim)]
            for c in range(dim):
                t = zeros(nc, NV)
                for d in range(dim):
                    if d != c:
                        t += G[:, :, d] * gr[d][c][:, None] - 2.0 / 3.0 * G[:, :, c] * gr[d][d][:, None]
                rhs[c] += (cs.rho * N[None] * (N * uc[c]).sum(1)[:, None] - mdt * t) * w[:, None]
        Ke = sum(Ce)
        for on, N, G, nx, w in self.open_faces():
            gr = [[(G[:, :, e] * uc[d][on]).sum(1) for e in range(dim)] for d in range(dim)]
            for c in range(dim):
                if dim == 2:
                    T = 4.0 / 3.0 * gr[0][0] - 2.0 / 3.0 * gr[1][1] if c == 0 else gr[0][1] + gr[1][0]
                else:
                    T = -2.0 * (gr[1][1] + gr[2][2]) / 3.0 if c == 0 else gr[0][c]
                rhs[c].index_add_(0, on, mdt * N[None] * (T * nx * w)[:, None])
        pred = []
        for c in range(dim):
            isd, g = self.dirichlet(c)
            Ae = cs.rho * Me + mdt * (Ke + Ce[c] / 3.0)
            pred.append(self.solve(Ae, self.cells, self.nv, self.add(rhs[c]), isd, g))
        pc = [v[self.cells] for v in pred]
        rp = zeros(nc, NV)
        for N, G, w, _, _ in self.quad():
            for d in range(dim):
                rp += cs.rho / cs.dt * G[:, :, d] * ((N * pc[d]).sum(1) * w)[:, None]
        for on, N, G, nx, w in self.open_faces():
            val = (-cs.rho / cs.dt * (N * pc[0][on]).sum(1) + cs.open_boundary_pressure_flux) * nx * w
            rp.index_add_(0, on, N[None] * val[:, None])
        self.P = self.solve(Ke, self.cells, self.nv, self.add(rp), *self.dirichlet(3))
        Pc = self.P[self.cells]
        rc = [zeros(nc, NV) for _ in range(dim)]
        for N, G, w, _, _ in self.quad():
            for c in range(dim):
                rc[c] -= cs.dt / cs.rho * N[None] * ((G[:, :, c] * Pc).sum(1) * w)[:, None]
        self.V = []
        for c in range(dim):
            isd, g = self.dirichlet(c)
            self.V.append(pred[c] + self.solve(Me, self.cells, self.nv, self.add(rc[c]), isd, 0.0 * g))

    def vorticity(self):
        num, den = torch.zeros(self.nc, 4, dtype=torch.float64, device=self.dev), 0.0
        for N, G, _, _, _ in self.quad():
            w = (G[:, :, 0] * self.V[1][self.cells] - G[:, :, 1] * self.V[0][self.cells]).sum(1)
            num += N[None] * w[:, None]
            den = den + N
        return self.add(num) / self.add(den[None].expand(self.nc, -1))

    # moving mesh
    def elasticity(self, lam, mu, fixed, body, disp):
        dofs = torch.cat([self.cells, self.cells + self.nv], 1)
        Ae = torch.zeros(self.nc, 8, 8, dtype=torch.float64, device=self.dev)
        for _, G, w, _, _ in self.quad():
            lap = torch.einsum("nad,nbd->nab", G, G)
            for i in range(2):
                for j in range(2):
                    k = lam * G[:, :, None, i] * G[:, None, :, j] + mu * G[:, :, None, j] * G[:, None, :, i]
                    if i == j:
                        k = k + mu * lap
                    Ae[:, 4 * i:4 * i + 4, 4 * j:4 * j + 4] += k * w[:, None, None]
        isd = torch.zeros(2 * self.nv, dtype=torch.bool, device=self.dev)
        g = torch.zeros(2 * self.nv, dtype=torch.float64, device=self.dev)
        for b, val in [(b, (0.0, 0.0)) for b in fixed] + [(body, disp)]:
            v = self.boundary(b)
            for d in range(2):
                isd[v + d * self.nv] = True
                g[v + d * self.nv] = val[d]
        x = self.solve(Ae, dofs, 2 * self.nv, torch.zeros_like(g), isd, g)
        return [x[:self.nv], x[self.nv:]]

    def reinterpolate(self, disp):
        """fields at the displaced interior vertices in the mesh before the move"""
        edge = torch.unique(torch.cat([self.boundary(b) for b in (1, 2, 3, 4)]))
        inner = torch.ones(self.nv, dtype=torch.bool, device=self.dev)
        inner[edge] = False
        inner = torch.nonzero(inner)[:, 0]
        cell, xi = self.first_containing(self.X[inner] + torch.stack(disp, 1)[inner], self.patch[inner], eps=1e-5)
        ok = cell >= 0
        vals = self.at(cell[ok], xi[ok], self.V + [self.P])
        got = [f.clone() for f in self.V + [self.P]]
        for k, f in enumerate(got):
            f[inner[ok]] = vals[:, k]
        return got


def exact(case, seed):
    specs, fields, pseed = _inputs(case, seed)
    kind, host = case["kind"], lambda x: x.cpu()  # noqa: E731
    if kind in ("flow", "moving", "members"):
        made = []
        for spec, f in zip(specs, fields):
            p = _Plain(spec, case, f, pseed)
            p.correct()
            p.move()
            p.check()
            p.project()
            p.fem()
            made.append(p)
        if kind == "flow":
            return {"fields": torch.cat([host(x) for p in made for x in p.V + [p.P]]), "loads": None}
        p = made[0]
        if kind == "members":
            slots = int(CAPACITY) * p.nc * p.q ** p.dim
            kept = [np.full(slots, -1, np.int32), np.zeros((slots, p.dim)), np.zeros((slots, p.dim))]
            n = _keep_particles([host(x).numpy() for x in (p.cell, p.xi, p.u)], kept)
            return {"fields": [host(x) for x in p.V + [p.P]], "loads": None, "vorticity": host(p.vorticity()),
                    "n": n, "cell": kept[0], "xi": kept[1], "u": kept[2]}
        disp = p.elasticity(1.0, 1.0, (1, 2, 4), 3, _body_step(1))
        return {"fields": [host(x) for x in p.reinterpolate(disp)], "loads": None,
                "displacement": [host(x) for x in disp], "vertices": host(p.X + torch.stack(disp, 1))}
    p = _Plain(specs[0], case, fields[0], pseed)
    frozen = [v.clone() for v in p.V]
    for _ in range(case["steps"]):
        p.correct()
        p.move()
        p.check()
        p.project()
        p.old, p.V = p.V, frozen
    return {"fields": torch.cat([host(x) for x in p.old])}
