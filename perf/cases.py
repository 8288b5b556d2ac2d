"""Workloads that stand for what a program has this framework do, through its public
entry points (DgSolver and CavityPool), for timing and for comparing results.

    listed()            the standing cases, as plain dicts
    draw(rng)           one more case of the same ranges
    prepare(case, seed) solver or pool with its mesh, and the initial fields
    run(state)          one pass; returns the fields, histories and diagnostics
    work(case)          bytes and flops one pass cannot do without
    exact(case, seed)   the same outputs from plain torch in 64 bits

Kinds of case:
  "box"     DgSolver on a box mesh: `steps` LSRK45 steps of a resident state.  With
            `blocking`, one DgSolver.step() call after the other, as the reference's
            own driver calls it; otherwise the steps are queued at once.
  "monitor" the loop of a simulation that watches its fields: after every step the
            probes are read, at the end the energy and the largest |E| and |H|.
  "mesh"    DgSolver on a mesh given by its arrays: curved hexahedra (per-node
            geometry) or a sheared box (one full Jacobian per element).
  "pool"    CavityPool: a set of cavities of different orders and sizes, started
            from their pulses, advanced together, their histories (and with
            `states` their fields) read back.

Every field is a set of Gaussian pulses drawn from the seed, as in the benchmark
workloads of this package; the meshes and the mix of a pool belong to the case.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from nekwave_b200 import DgSolver, Mesh
from nekwave_b200.pool import CavityPool

# Carpenter-Kennedy five-stage LSRK45
RK_A = (0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
        -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0)
RK_B = (1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
        1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
        2277821191437.0 / 14882151754819.0)

ON_CHIP = 33_000_000  # bytes of state and register that an SM array's shared memory can hold


def _box(name, N, nel, edges, periodic, c0, steps, precision="fp64", blocking=False):
    return {"name": name, "kind": "box", "N": N, "nx": nel[0], "ny": nel[1], "nz": nel[2],
            "lx": edges[0], "ly": edges[1], "lz": edges[2], "periodic": periodic, "c0": c0,
            "steps": steps, "precision": precision, "blocking": blocking}


def listed():
    return [
        # the reference's call: one blocking step of a small cavity (the TM110 cube of the
        # reference checks, 8000 nodes): launches and the host's wait
        _box("small_blocking_step", 5, (4, 4, 4), (1.0, 1.0, 1.0), 0, 1.0, 1, blocking=True),
        # the same cube's whole run of 200 steps, queued at once
        _box("small_run", 5, (4, 4, 4), (1.0, 1.0, 1.0), 0, 1.0, 200),
        # one request of the serving stream on its own: a mid-size cavity of odd sizes
        # (fits L2), probes read after every step
        {"name": "monitored_cavity", "kind": "monitor", "N": 7, "nx": 9, "ny": 11, "nz": 8,
         "lx": 0.9, "ly": 1.3, "lz": 0.8, "periodic": 0, "c0": 1.0, "steps": 10,
         "precision": "fp64", "probes": 8},
        # the headline: periodic box, 8 points, central flux, 16.8 M nodes
        _box("periodic_box", 8, (32, 32, 32), (1.0, 1.0, 1.0), 7, 0.0, 4),
        # the large PEC cavity, 6 points, upwind, 28.3 M nodes
        _box("large_cavity", 6, (64, 64, 32), (2.0, 2.0, 1.0), 0, 1.0, 4),
        # large serving requests, odd sizes: low and high order
        _box("cavity_low_order", 5, (41, 37, 29), (1.9, 1.6, 1.3), 0, 1.0, 4),
        _box("cavity_high_order", 9, (23, 19, 27), (1.1, 0.9, 1.4), 0, 1.0, 4),
        # the FP32-bulk precision class on the headline box
        _box("periodic_box_fp32", 8, (32, 32, 32), (1.0, 1.0, 1.0), 7, 0.0, 4, "fp32"),
        # a curved mesh handed over as arrays, as the reference's front end does
        {"name": "curved_mesh", "kind": "mesh", "N": 6, "nx": 17, "ny": 15, "nz": 19, "lx": 1.2,
         "ly": 1.0, "lz": 1.4, "periodic": 0, "c0": 1.0, "steps": 4, "precision": "fp64",
         "map": "curved"},
        # 256 uneven cavities advanced together (the batch workload)
        {"name": "batch", "kind": "pool", "count": 256, "mix": 0, "n_lo": 4, "n_hi": 9,
         "el_lo": 2, "el_hi": 12, "steps": 16, "precision": "fp64", "probes": 8,
         "energy_every": 8, "states": False},
        # the server's default precision on 14 cavities of its larger sizes
        {"name": "served_fp32", "kind": "pool", "count": 14, "mix": 3, "n_lo": 4, "n_hi": 9,
         "el_lo": 2, "el_hi": 24, "steps": 20, "precision": "fp32", "probes": 8,
         "energy_every": 10, "states": False},
        # a few small cavities: the pool where launches count
        {"name": "small_batch", "kind": "pool", "count": 16, "mix": 1, "n_lo": 4, "n_hi": 9,
         "el_lo": 2, "el_hi": 5, "steps": 60, "precision": "fp64", "probes": 8,
         "energy_every": 10, "states": True},
    ]


def draw(rng):
    kind = rng.choice(["box", "box", "box", "monitor", "mesh", "pool"])
    precision = "fp32" if rng.random() < 0.25 else "fp64"
    if kind == "pool":
        small = rng.random() < 0.5
        count = int(round(math.exp(rng.uniform(math.log(4), math.log(40 if small else 128)))))
        return {"kind": "pool", "count": count, "mix": rng.randrange(1 << 20), "n_lo": rng.choice([3, 4, 4]),
                "n_hi": rng.choice([8, 9, 9]), "el_lo": 2, "el_hi": rng.randint(3, 6) if small else rng.randint(7, 12),
                "steps": rng.randint(10, 20), "precision": precision, "probes": rng.choice([0, 3, 8]),
                "energy_every": rng.choice([1, 5, 10]), "states": small}
    N = rng.randint(3, 10)
    hi = {"box": 1.5e7, "monitor": 6e5, "mesh": 1.5e6}[kind]
    nodes = math.exp(rng.uniform(math.log(3e3), math.log(hi)))
    mean = (nodes / N ** 3) ** (1.0 / 3.0)
    nel = [max(2, int(round(mean * math.exp(rng.uniform(-0.3, 0.3))))) for _ in range(3)]
    edges = [round(rng.uniform(0.5, 2.0), 3) for _ in range(3)]
    c0 = rng.choice([0.0, 1.0, 1.0])
    base = {"kind": kind, "N": N, "nx": nel[0], "ny": nel[1], "nz": nel[2], "lx": edges[0], "ly": edges[1],
            "lz": edges[2], "c0": c0, "precision": precision}
    if kind == "box":
        return dict(base, periodic=rng.choice([0, 0, 1, 5, 7]), steps=rng.choice([1, 2, 3, 4]),
                    blocking=rng.random() < 0.3)
    if kind == "monitor":
        return dict(base, periodic=rng.choice([0, 0, 7]), steps=rng.randint(5, 12), probes=rng.choice([1, 8]))
    return dict(base, periodic=0, steps=rng.choice([1, 2, 3, 4]), map=rng.choice(["curved", "curved", "sheared"]))


# ---- numerics of the method, from its definition ---------------------------------------


def _gll(N):
    """GLL nodes, weights and differentiation matrix (row: node, column: basis function)."""
    P = np.polynomial.legendre.Legendre.basis(N - 1)
    z = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]])
    dP, ddP = P.deriv(), P.deriv(2)
    for _ in range(3):  # Newton polish of the roots
        z[1:-1] -= dP(z[1:-1]) / ddP(z[1:-1])
    z = 0.5 * (z - z[::-1])
    L = P(z)
    w = 2.0 / (N * (N - 1) * L * L)
    D = np.zeros((N, N))
    for i in range(N):
        for j in range(N):
            if i != j:
                D[i, j] = L[i] / (L[j] * (z[i] - z[j]))
    D[0, 0], D[-1, -1] = -N * (N - 1) / 4.0, N * (N - 1) / 4.0
    return z, w, D


def _dt(case):
    z = _gll(case["N"])[0]
    h = min(case["lx"] / case["nx"], case["ly"] / case["ny"], case["lz"] / case["nz"])
    return (0.25 if case["kind"] == "mesh" else 0.5) * 0.5 * float(np.diff(z).min()) * h


def _coords(case, device):
    """Node coordinates of the box, each [nz, ny, nx, N, N, N]."""
    N, n = case["N"], (case["nx"], case["ny"], case["nz"])
    z = torch.from_numpy(_gll(N)[0]).to(device)
    line = []
    for d, length in enumerate((case["lx"], case["ly"], case["lz"])):
        h = length / n[d]
        line.append((torch.arange(n[d], device=device, dtype=torch.float64)[:, None] + 0.5 * (z + 1.0)) * h)
    full = (n[2], n[1], n[0], N, N, N)
    return (line[0][None, None, :, None, None, :].expand(full), line[1][None, :, None, None, :, None].expand(full),
            line[2][:, None, None, :, None, None].expand(full))


def _pulses(case, seed, k=0):
    """(amplitude, centre, width) of a Gaussian in each of the six components."""
    r = random.Random("%d/%d" % (seed, k))
    edges = (case["lx"], case["ly"], case["lz"])
    return [(r.uniform(0.5, 1.0), *(e * r.uniform(0.25, 0.75) for e in edges),
             r.uniform(0.1, 0.15) * min(edges) + 0.05 * max(edges)) for _ in range(6)]


def _fields(pulses, x):
    """[6, nz, ny, nx, N, N, N] fields of the pulses at the node coordinates x."""
    return torch.stack([a * torch.exp(-((x[0] - p) ** 2 + (x[1] - q) ** 2 + (x[2] - s) ** 2) / (w * w))
                        for a, p, q, s, w in pulses])


def _mapped(case, x):
    """The mesh map of a "mesh" case applied to the box coordinates."""
    L = (case["lx"], case["ly"], case["lz"])
    if case["map"] == "sheared":
        return (x[0] + 0.3 * x[1] + 0.1 * x[2], -0.2 * x[0] + 1.1 * x[1] + 0.05 * x[2],
                0.1 * x[0] + 0.2 * x[1] + 0.9 * x[2])
    s = [torch.sin(math.pi * c / l) for c, l in zip(x, L)]
    bump = 0.06 * min(L) * s[0] * s[1] * s[2]
    return x[0] + bump, x[1] - 0.7 * bump, x[2] + 0.5 * bump


def _along(D, V, axis):
    """Derivative along reference axis 0 (r: last index), 1 (s) or 2 (t)."""
    if axis == 0:
        return V @ D.T
    if axis == 1:
        return D @ V
    N = D.shape[0]
    return (D @ V.reshape(V.shape[:-2] + (N * N,))).reshape(V.shape)


def _metrics(case, X, device):
    """(J, met[3][3]) with met[physical axis][reference axis] = d xi / d x."""
    D = torch.from_numpy(_gll(case["N"])[2]).to(device)
    g = [[_along(D, c.contiguous().reshape(c.shape[:3] + (case["N"],) * 3), a) for a in range(3)] for c in X]
    m = [[g[(c + 1) % 3][(a + 1) % 3] * g[(c + 2) % 3][(a + 2) % 3] -
          g[(c + 1) % 3][(a + 2) % 3] * g[(c + 2) % 3][(a + 1) % 3] for a in range(3)] for c in range(3)]
    J = sum(g[0][a] * m[0][a] for a in range(3))
    return J, [[m[c][a] / J for a in range(3)] for c in range(3)]


# ---- what a program has in hand -----------------------------------------------------------

_FACES = ((1, 0), (0, -1), (1, -1), (0, 0), (2, 0), (2, -1))  # (reference axis, node index) of faces 0..5


def _mesh(case):
    """The case's mesh as a nekwave_b200 Mesh of arrays (box topology, mapped geometry)."""
    N, dev = case["N"], "cuda"
    box = Mesh(N)
    box.createBoxMesh(case["nx"], case["ny"], case["nz"], 0.0, case["lx"], 0.0, case["ly"], 0.0, case["lz"])
    z, w, D = _gll(N)
    X = _mapped(case, _coords(case, dev))
    J, met = _metrics(case, X, dev)
    wd = torch.from_numpy(w).to(dev)
    ww = (wd[:, None] * wd[None, :]).reshape(-1)
    normal, area = [], []
    for axis, at in _FACES:
        # (q, p) order: the face's node axes with the faster one last
        v = torch.stack([met[c][axis].select(5 - axis, at) for c in range(3)]).reshape(3, -1, N * N)
        size = v.norm(dim=0)
        normal.append((1.0 if at else -1.0) * v / size)
        area.append(size * J.select(5 - axis, at).reshape(-1, N * N).abs() * ww)
    normal = torch.stack(normal, 2).reshape(3, -1).cpu().numpy()  # element, face, q, p
    area = torch.stack(area, 1).reshape(-1).cpu().numpy()
    f = box.getFaceArrays()
    flat = lambda v: v.reshape(-1).cpu().numpy()  # noqa: E731
    return Mesh.from_arrays(N, box.getNumElements(), z=z, w=w, D=D.T.reshape(-1).copy(),
                            w3=(w[:, None, None] * w[None, :, None] * w[None, None, :]).reshape(-1), jac=flat(J),
                            met=np.stack([flat(met[c][a]) for c in range(3) for a in range(3)]), vmin=f["vmin"],
                            vplus=f["vplus"], bc=f["bc"], nx=normal[0], ny=normal[1], nz=normal[2], dA=area)


class _View:
    """Device memory of a solver as a tensor's source; the tensor keeps the solver alive."""

    def __init__(self, owner, pointer, shape, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": shape, "strides": strides,
                                         "typestr": "<f8", "version": 3}


def _state_view(state):
    """The solver's current device state as a [6, npts] tensor (two buffers in turn)."""
    pointer = state["solver"].deviceState()[0]
    if pointer not in state["views"]:
        npts, stride = state["npts"], state["stride"]
        view = _View(state["solver"], pointer, (6, npts), (8 * stride, 8))
        state["views"][pointer] = torch.as_tensor(view, device="cuda")
    return state["views"][pointer]


def _cavities(case):
    """The cavities of a pool case: sizes and orders from the case alone."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        n = [r.randint(case["el_lo"], case["el_hi"]) for _ in range(3)]
        c = {"kind": "box", "N": r.randint(case["n_lo"], case["n_hi"]), "nx": n[0], "ny": n[1], "nz": n[2],
             "lx": r.uniform(0.5, 2.0), "ly": r.uniform(0.5, 2.0), "lz": r.uniform(0.5, 2.0), "periodic": 0,
             "c0": 1.0}
        c["points"] = _points(c, case["probes"], r)
        out.append(c)
    return out


def _points(c, count, r):
    return [tuple(e * r.uniform(0.02, 0.98) for e in (c["lx"], c["ly"], c["lz"])) for _ in range(count)]


def _nel(c):
    return c["nx"], c["ny"], c["nz"]


def _npts(c):
    return c["nx"] * c["ny"] * c["nz"] * c["N"] ** 3


def prepare(case, seed):
    lo = (0.0, 0.0, 0.0)
    if case["kind"] == "pool":
        cav = _cavities(case)
        budget = sum(18 * 8 * _npts(c) + 512 * c["nx"] * c["ny"] * c["nz"] for c in cav) * 1.1 + (64 << 20)
        pool = CavityPool(int(budget), max_slots=case["count"], precision=case["precision"])
        slots = [pool.add_box(c["N"], _nel(c), lo, (c["lx"], c["ly"], c["lz"]), c["c0"], _dt(c), case["steps"],
                              probes=c["points"], energy_every=case["energy_every"]) for c in cav]
        return {"case": case, "pool": pool, "slots": slots, "pulses": [_pulses(c, seed, k) for k, c in enumerate(cav)]}
    s = DgSolver(case["precision"])
    if case["kind"] == "mesh":
        s.initialize(_mesh(case), case["c0"])
        u = _fields(_pulses(case, seed), _mapped(case, _coords(case, "cuda")))
        s.uploadState(u.reshape(-1).cpu().numpy())
    else:
        s.initializeBox(case["N"], _nel(case), lo, (case["lx"], case["ly"], case["lz"]), case["c0"],
                        periodic=tuple(bool(case["periodic"] >> d & 1) for d in range(3)))
        s.initPulse(_pulses(case, seed))
    info = s.info()
    state = {"case": case, "solver": s, "dt": _dt(case), "steps": case["steps"], "npts": info["npts"],
             "stride": info["stride"], "views": {}}
    if case["kind"] == "monitor":
        w = _probe_weights(case, _points(case, case["probes"], random.Random(seed)))
        s.probeSetup([e * case["N"] ** 3 for e, _ in w], np.stack([v for _, v in w]))
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "pool":
        pool = state["pool"]
        for slot, pulses in zip(state["slots"], state["pulses"]):
            pool.init_pulse(slot, pulses)
        pool.step(case["steps"])
        got = [pool.results(slot, state=case["states"]) for slot in state["slots"]]
        return {k: np.concatenate([g[k].reshape(-1) for g in got]) for k in got[0] if got[0][k].size}
    s, dt = state["solver"], state["dt"]
    if case["kind"] == "monitor":
        trace = []
        for _ in range(state["steps"]):
            s.steps(dt, 1, sync=False)
            trace.append(s.probeRead())
        return {"energy": s.energy(), "max": list(s.maxNorms()), "probes": np.stack(trace), "state": _state_view(state)}
    if case.get("blocking"):
        for _ in range(state["steps"]):
            s.step(dt)
    else:
        s.steps(dt, state["steps"], sync=False)
    return _state_view(state)


def _work(c, steps, curved=False):
    n, N = _npts(c), c["N"]
    # twelve derivatives and curl combinations a node and component pair, the fluxes of a
    # node's share of face points, the update
    flops = 5.0 * steps * n * (24.0 * N + 24 + 6.0 / N * 40 + 24)
    geometry = n * (72.0 + 6.0 / N * 36.0) if curved else 0.0
    if 96.0 * n + geometry <= ON_CHIP:
        return 96.0 * n + geometry, flops  # state in, state out
    # u read and written every stage; the register written by stages 1-4 and read by 2-5
    return steps * (n * (5 * 96.0 + 4 * 48.0 + 4 * 48.0) + 5 * geometry), flops


def work(case):
    if case["kind"] == "pool":
        parts = [_work(c, case["steps"]) for c in _cavities(case)]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    b, f = _work(case, case["steps"], case.get("map") == "curved")
    return {"bytes": b, "flops": f}


# ---- the same outputs in plain torch ---------------------------------------------------------


def _probe_weights(c, points):
    """(element, N^3 tensor Lagrange weights) of each point."""
    z = _gll(c["N"])[0]
    out = []
    for p in points:
        at, rows = [], []
        for x, n, length in zip(p, _nel(c), (c["lx"], c["ly"], c["lz"])):
            h = length / n
            e = min(n - 1, int(x / h))
            r = 2.0 * (x - e * h) / h - 1.0
            at.append(e)
            rows.append(np.array([np.prod([(r - z[b]) / (z[a] - z[b]) for b in range(c["N"]) if b != a])
                                  for a in range(c["N"])]))
        w = rows[2][:, None, None] * rows[1][None, :, None] * rows[0][None, None, :]
        out.append((at[0] + c["nx"] * (at[1] + c["ny"] * at[2]), w.reshape(-1)))
    return out


class _Plain:
    """The DG scheme of one cavity, written out in torch."""

    def __init__(self, c, device="cuda"):
        self.c, N = c, c["N"]
        z, w, D = _gll(N)
        self.D = torch.from_numpy(D).to(device)
        x = _coords(c, device)
        w1 = torch.from_numpy(w).to(device)
        w3 = w1[:, None, None] * w1[None, :, None] * w1[None, None, :]
        L, n = (c["lx"], c["ly"], c["lz"]), _nel(c)
        if "map" in c:
            self.x = _mapped(c, x)
            J, self.met = _metrics(c, self.x, device)
            self.volume = J * w3
        else:
            self.x = x
            self.met = None
            self.scale = [2.0 * n[d] / L[d] for d in range(3)]
            self.volume = w3 / (self.scale[0] * self.scale[1] * self.scale[2])
        self.faces = []
        for d in range(3):
            for at in (0, -1):
                sign = 1.0 if at else -1.0
                if self.met is None:
                    normal, lift = [sign if a == d else 0.0 for a in range(3)], self.scale[d] / w[0]
                else:
                    v = [self.met[a][d].select(5 - d, at) for a in range(3)]
                    size = torch.sqrt(v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
                    normal, lift = [sign * a / size for a in v], size / w[0]
                self.faces.append((d, at, normal, lift))

    def curl(self, V):
        D = self.D
        if self.met is None:
            g = lambda c, a: self.scale[a] * _along(D, V[c], a)  # noqa: E731
        else:
            ref = [[_along(D, V[c], a) for a in range(3)] for c in range(3)]
            g = lambda c, a: sum(self.met[a][b] * ref[c][b] for b in range(3))  # noqa: E731
        return torch.stack([g(2, 1) - g(1, 2), g(0, 2) - g(2, 0), g(1, 0) - g(0, 1)])

    def rhs(self, U):
        c0 = self.c["c0"]
        out = torch.cat([self.curl(U[3:]), -self.curl(U[:3])])
        for d, at, n, lift in self.faces:
            own = U.select(6 - d, at)
            other = U.select(6 - d, -1 if at == 0 else 0)
            axis = 3 - d  # element axis of (6, nz, ny, nx, ., .)
            jump = torch.roll(other, 1 if at == 0 else -1, axis) - own
            if not self.c["periodic"] >> d & 1:
                wall = jump.select(axis, at)
                mine = own.select(axis, at)
                wall[:3] = -2.0 * mine[:3]
                wall[3:] = 0.0
            cross = lambda v: [n[(a + 1) % 3] * v[(a + 2) % 3] - n[(a + 2) % 3] * v[(a + 1) % 3]  # noqa: E731
                               for a in range(3)]
            nE, nH = cross(jump[:3]), cross(jump[3:])
            nnE, nnH = cross(nE), cross(nH)
            for a in range(3):
                out[a].select(5 - d, at).add_(lift * (0.5 * nH[a] - 0.5 * c0 * nnE[a]))
                out[3 + a].select(5 - d, at).add_(lift * (-0.5 * nE[a] - 0.5 * c0 * nnH[a]))
        return out

    def step(self, U, dt):
        K = torch.zeros_like(U)
        for a, b in zip(RK_A, RK_B):
            K = a * K + dt * self.rhs(U)
            U = U + b * K
        return U

    def energy(self, U):
        return float(0.5 * ((U * U).sum(0) * self.volume).sum())

    def probe(self, U, weights):
        N3 = self.c["N"] ** 3
        E = U.reshape(6, -1, N3)
        return np.stack([(E[:, e] @ torch.from_numpy(w).to(U.device)).cpu().numpy() for e, w in weights])


def exact(case, seed):
    if case["kind"] == "pool":
        parts = {"energy": [], "probes": [], "state": []}
        for k, c in enumerate(_cavities(case)):
            m, weights, dt = _Plain(c), _probe_weights(c, c["points"]), _dt(c)
            U = _fields(_pulses(c, seed, k), m.x)
            for n in range(case["steps"] + 1):
                if n:
                    U = m.step(U, dt)
                recorded = n % case["energy_every"] == 0 or n == case["steps"]
                parts["energy"].append(np.array([m.energy(U) if recorded else np.nan]))
                if weights:
                    parts["probes"].append(m.probe(U, weights).reshape(-1))
            if case["states"]:
                parts["state"].append(U.reshape(-1).cpu().numpy())
        return {k: np.concatenate(v) for k, v in parts.items() if v}
    m, dt = _Plain(case), _dt(case)
    U = _fields(_pulses(case, seed), m.x)
    if case["kind"] != "monitor":
        for _ in range(case["steps"]):
            U = m.step(U, dt)
        return U.reshape(6, -1)
    weights = _probe_weights(case, _points(case, case["probes"], random.Random(seed)))
    trace = []
    for _ in range(case["steps"]):
        U = m.step(U, dt)
        trace.append(m.probe(U, weights))
    size = (U * U).reshape(2, 3, -1).sum(1).amax(1).sqrt()
    return {"energy": m.energy(U), "max": [float(size[0]), float(size[1])], "probes": np.stack(trace),
            "state": U.reshape(6, -1)}
