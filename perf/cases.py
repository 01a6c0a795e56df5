"""The work this framework is used for, as cases that can be timed and compared.

Every case goes through the package's own entry points, as a user's program calls them, over the
grids, materials and motions of the package's workloads (alpineqms_gb300/workloads.py) and tests:

  steps     a run of backward-Euler steps from a saved state, each followed by the H slice that the
            drop-in program dumps (QMSSolver.set_state, step, slices; the three cubes at the end
            when the run saves all fields)
  steady    one magnetostatic solve and its H cubes on a handle that holds the geometry: the next
            direction of a sweep over field directions
  residual  the scaled residual of a caller's own state from the caller's own buffers
            (qms_residual_noalloc)
  requests  whole requests (geometry, steady state, steps, slices) through the serving object
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from alpineqms_gb300 import _lib, workloads
from alpineqms_gb300.serving import NativeServer, SolveRequest
from alpineqms_gb300.solver import PinnedBuffer, QMSSolver, default_desc
from alpineqms_gb300.trajectory import scaled_field

MU0 = 1.25663706e-6
_REQUEST_SIZES = ((48, 48, 48), (64, 64, 64), (64, 48, 32))


def _steps(name, geometry, size, steps, motion="none", precision="mixed", cubes=False):
    return {"name": name, "kind": "steps", "geometry": geometry, "xs": size[0], "ys": size[1], "zs": size[2],
            "steps": steps, "motion": motion, "precision": precision, "cubes": cubes}


def listed():
    return [
        # the smallest grids of the tests: every launch and host wait counts
        _steps("block_16x14x12", "block", (16, 14, 12), 10, cubes=True),
        # a conducting block in a 1 kHz field (workload plain_block_32), whole run of 20 steps
        _steps("block_32", "block", (32, 32, 32), 20, cubes=True),
        # the smallest request of the serving stream: random ellipsoids, AC field
        _steps("ellipsoids_48", "ellipsoids", (48, 48, 48), 8, cubes=True),
        # 24 random inclusions at 500 Hz (workload inclusions_96)
        _steps("ellipsoids_96", "ellipsoids", (96, 96, 96), 6),
        # the largest serving request, saving all fields
        _steps("ellipsoids_128_cubes", "ellipsoids", (128, 128, 128), 4, cubes=True),
        # a plate that starts to move through a static field, odd sizes, harmonic frame motion:
        # another operator every step
        _steps("plate_141x97x53_harmonic", "plate", (141, 97, 53), 8, motion="harmonic"),
        # the same start at constant speed on the largest grid (workload moving_plate_256)
        _steps("plate_256_moving", "plate", (256, 256, 256), 12, motion="constant"),
        # thin steel laminations with one-cell gaps (workload laminated_core, reduced)
        _steps("core_64x64x80", "core", (64, 64, 80), 3, cubes=True),
        # every inner component in FP64
        _steps("ellipsoids_64_fp64", "ellipsoids", (64, 64, 64), 2, precision="fp64"),
        # magnetostatics: one field direction after the other on a ragged grid
        {"name": "steady_157x131x143", "kind": "steady", "xs": 157, "ys": 131, "zs": 143},
        # a check of somebody else's state
        {"name": "residual_192x192x160", "kind": "residual", "xs": 192, "ys": 192, "zs": 160},
        # serving: several requests resident at once, setup and steady state among it
        {"name": "requests_6", "kind": "requests", "count": 6, "steps": 4},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["steady", "residual", "requests"])
    if kind == "steady":
        return {"kind": kind, "xs": _log_int(rng, 24, 160), "ys": _log_int(rng, 24, 160), "zs": _log_int(rng, 24, 160)}
    if kind == "residual":
        return {"kind": kind, "xs": _log_int(rng, 8, 224), "ys": _log_int(rng, 8, 224), "zs": _log_int(rng, 8, 224)}
    if kind == "requests":
        return {"kind": kind, "count": rng.randint(2, 6), "steps": rng.randint(2, 6)}
    geometry = rng.choice(["block", "ellipsoids", "ellipsoids", "plate", "plate", "core"])
    if geometry == "block":
        lo, hi, steps, motion = 10, 48, rng.randint(6, 20), "none"
    elif geometry == "ellipsoids":
        lo, hi, steps, motion = 32, 128, rng.randint(2, 6), "none"
    elif geometry == "plate":
        lo, hi, steps, motion = 32, 224, rng.randint(4, 12), rng.choice(["constant", "constant", "harmonic"])
    else:
        lo, hi, steps, motion = 40, 80, rng.randint(1, 3), "none"
    size = tuple(_log_int(rng, lo, hi) for _ in range(3))
    precision = "fp64" if max(size) <= 72 and rng.random() < 0.2 else "mixed"
    if precision == "fp64":
        steps = min(steps, 3)
    return {k: v for k, v in _steps("", geometry, size, steps, motion, precision, rng.random() < 0.25).items()
            if k != "name"}


# --------------------------------------------------------------------------- inputs
def _block(size, rng):
    """A conducting block in the middle of the grid, 1 kHz field along a tilted axis."""
    geom = np.zeros(size)
    lo = [int(0.31 * s) + int(rng.integers(0, 2)) for s in size]
    n = [max(2, int(0.375 * size[0])), max(2, int(0.375 * size[1])), max(2, int(0.25 * size[2]))]
    geom[lo[0]:lo[0] + n[0], lo[1]:lo[1] + n[1], lo[2]:lo[2] + n[2]] = 1
    mats = [(1, (1.0, 1.0, 1.0), (5.8e7 * rng.uniform(0.6, 1.0),) * 3)]
    B = 1e-3 * np.array([rng.uniform(-0.3, 0.3), rng.uniform(-0.3, 0.3), 1.0])
    return workloads._inputs(size, 1e-3, 1e-5, 1, tuple(B), np.zeros(9), [(0.0, 0.0, 0)] * 3, mats,
                             ("cos", 1000.0, 0.0)), geom.flatten(order="F")


def _plate(size, rng):
    """An aluminium plate across most of the grid in a static field with a gradient along z."""
    xs, ys, zs = size
    geom = np.zeros(size)
    ex, ey, ez = max(4, xs // 9), max(4, ys // 9), max(2, min(10, zs // 8))
    z0 = (zs - ez) // 2 + int(rng.integers(-1, 2))
    geom[ex:xs - ex, ey:ys - ey, z0:z0 + ez] = 1
    g = 0.1 * rng.uniform(0.7, 1.3)
    G = [-0.5 * g, 0.0, 0.0, 0.0, -0.5 * g, 0.0, 0.0, 0.0, g]
    mats = [(1, (1.0, 1.0, 1.0), (3.5e7 * rng.uniform(0.8, 1.0),) * 3)]
    return workloads._inputs(size, 1e-3, 1e-5, 1, (0.0, 0.0, 1e-2 * rng.uniform(0.8, 1.2)), G, [(0.0, 0.0, 0)] * 3,
                             mats, None), geom.flatten(order="F")


def _core(size, rng):
    """Steel laminations, five cells thick with one-cell gaps, in a 60 Hz field."""
    inp, geom = workloads.laminated_core(shape=size, laminations=max(2, (size[2] - 20) // 6))
    m = inp.materials[0]
    m.mu_r = (float(rng.uniform(1000.0, 2000.0)),) * 3
    inp.B = (float(rng.uniform(0.3, 0.5)), float(rng.uniform(-0.1, 0.1)), 0.0)
    return inp, geom


def _workload(case, seed):
    rng = np.random.default_rng(np.random.PCG64(seed))
    size = (case["xs"], case["ys"], case["zs"])
    kind = case.get("geometry", "ellipsoids")
    if kind == "ellipsoids":
        inp, geom = workloads.serving_request(rng, sizes=(size,))
    else:
        inp, geom = {"block": _block, "plate": _plate, "core": _core}[kind](size, rng)
    speed, freq, phase = -10.0 * rng.uniform(0.7, 1.0), rng.uniform(200.0, 1000.0), rng.uniform(0.3, 1.2)
    vel = []
    for n in range(1, case.get("steps", 0) + 1):
        v = {"none": 0.0, "constant": speed,
             "harmonic": -speed * math.sin(2.0 * math.pi * freq * n * inp.dt + phase)}[case.get("motion", "none")]
        vel.append([v, 0.0, 0.0])
    return inp, geom, vel


def _directions(seed):
    rng = np.random.default_rng([int(seed), 7])
    d = rng.standard_normal((3, 3))
    return 5e-3 * d / np.linalg.norm(d, axis=1, keepdims=True)


def _slots(inp, geom):
    """The uint8 material slots and the six-column table of a geometry (slot r = table row r)."""
    lut = np.zeros(int(max(m.mat_id for m in inp.materials)) + 1, np.uint8)
    for r, m in enumerate(inp.materials):
        lut[int(m.mat_id)] = r + 1
    return lut[geom.astype(np.int64)], np.ascontiguousarray(inp.props_table()[:, 1:7])


def _interior(xs, ys, zs):
    """Per block, the [k, j, i] slices of the rows that are not Dirichlet rows."""
    out = []
    for q in range(4):
        b = [slice(2, zs - 1), slice(2, ys - 1), slice(2, xs - 1)]
        if q < 3:
            b[2 - q] = slice(1, (xs, ys, zs)[q] - 1)
        out.append(tuple(b))
    return out


def _residual_inputs(case, seed):
    """A state as an iterative solver meets it: the smooth field of a source plus what is still to be
    removed, and a right-hand side of the operator's own scale on every row."""
    inp, geom, _ = _workload(case, seed)
    slots, rows = _slots(inp, geom)
    xs, ys, zs = case["xs"], case["ys"], case["zs"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    shapes = [(zs + 1, ys + 1, xs), (zs + 1, ys, xs + 1), (zs, ys + 1, xs + 1), (zs + 1, ys + 1, xs + 1)]
    x, b = [], []
    for q, (nk, nj, ni) in enumerate(shapes):
        k, j, i = (torch.linspace(0.0, 1.0, m, dtype=torch.float64, device="cuda") for m in (nk, nj, ni))
        a = torch.rand(3, generator=g, dtype=torch.float64, device="cuda") * 3.0 + 1.0
        f = torch.sin(a[0] * k)[:, None, None] * torch.cos(a[1] * j)[None, :, None] * torch.sin(a[2] * i + q)[None, None]
        noise = torch.randn((2,) + f.shape, generator=g, dtype=torch.float64, device="cuda")
        x.append(1e-4 * (f + 1e-2 * noise[0]))
        b.append(x[q] * (1.0 + 1e-2 * noise[1]))             # Dirichlet rows: nearly met
        # no charge in the V rows: in air their scale is that of 1e-12 S/m
        inner = _interior(xs, ys, zs)[q]
        b[q][inner] = 2e7 * noise[1][inner] if q < 3 else 0.0
    x, b = (torch.cat([t.reshape(-1) for t in parts]) for parts in (x, b))
    return inp, slots, rows, x, b, [-10.0, 2.0, 1.0]


class _Held:
    """What a user's program keeps between calls; gives the handle back with the last reference."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        for name in ("server", "solver", "pinned"):
            held = self.__dict__.get(name)
            if held is not None:
                held.close()


def _solver(inp, geom, case):
    # the plate's runs ask for a quarter of the default tolerance: at the default, the fields of two
    # correct solves of a dozen steps that each start from the one before are up to 6e-10 apart
    tol = 5e-14 if case.get("geometry") == "plate" else None
    s = QMSSolver(default_desc(inp.xs, inp.ys, inp.zs, inp.dx, inp.dy, inp.dz, inp.dt,
                               precision=case.get("precision", "mixed"), tol=tol))
    s.set_geometry_f64(geom, inp.props_table())
    return s


def prepare(case, seed):
    if case["kind"] == "residual":
        inp, slots, rows, x, b, v = _residual_inputs(case, seed)
        fn = _lib.load().qms_residual_noalloc
        fn.restype = ctypes.c_int
        fn.argtypes = [ctypes.c_int] * 3 + [ctypes.c_double] * 4 + [ctypes.c_int, ctypes.POINTER(ctypes.c_double),
                                                                     ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int] + [ctypes.c_void_p] * 5
        return _Held(case=case, fn=fn, inp=inp, slots=torch.from_numpy(slots).cuda(), rows=rows, x=x, b=b,
                     v=_lib.dvec(v), r=torch.empty_like(x), sums=torch.empty(4, dtype=torch.float64, device="cuda"))
    if case["kind"] == "requests":
        rng = np.random.default_rng(np.random.PCG64(seed))
        todo = [workloads.serving_request(rng, sizes=(_REQUEST_SIZES[q % 3],), nt=case["steps"])
                for q in range(case["count"])]
        return _Held(case=case, server=NativeServer(), todo=todo)
    inp, geom, vel = _workload(case, seed)
    solver = _solver(inp, geom, case)
    if case["kind"] == "steady":
        return _Held(case=case, solver=solver, directions=_directions(seed), turn=0)
    B, G = scaled_field(inp.B, inp.G, inp.excitation, 0.0)
    solver.steady([0.0, 0.0, 0.0], B, G)
    pinned = PinnedBuffer(solver.n)
    pinned.array[:] = solver.get_state()
    fields = [scaled_field(inp.B, inp.G, inp.excitation, n * inp.dt) for n in range(1, case["steps"] + 1)]
    return _Held(case=case, solver=solver, pinned=pinned, vel=vel, fields=fields, axis=inp.slice_axis,
                 index=inp.slice_index)


def run(state):
    case = state.case
    if case["kind"] == "residual":
        i = state.inp
        rc = state.fn(i.xs, i.ys, i.zs, i.dx, i.dy, i.dz, i.dt, 1, state.v, state.slots.data_ptr(),
                      state.rows.ctypes.data, state.rows.shape[0], state.x.data_ptr(), state.b.data_ptr(),
                      state.r.data_ptr(), state.sums.data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("qms_residual_noalloc: %d" % rc)
        return {"r": state.r, "sums": state.sums}
    if case["kind"] == "requests":
        ids = [state.server.submit(SolveRequest(inp, geom)) for inp, geom in state.todo]
        done = [state.server.wait(i) for i in ids]
        if any(r.status != "ok" for r in done):
            raise RuntimeError("a request failed: %s" % [r.error for r in done])
        return [np.stack(r.slices) for r in done]
    s = state.solver
    if case["kind"] == "steady":
        B = state.directions[state.turn % len(state.directions)]
        state.turn += 1
        s.steady([0.0, 0.0, 0.0], B, np.zeros(9))
        return s.fields()
    s.set_state(state.pinned.array)
    out = []
    for v, (B, G) in zip(state.vel, state.fields):
        s.step(v, B, G)
        out.append(np.stack([h.ravel(order="F") for h in s.slices(state.axis, state.index)]))
    return {"slices": np.stack(out), "cubes": s.fields() if case["cubes"] else None}


def _unknowns(xs, ys, zs):
    nx, ny, nz = xs + 1, ys + 1, zs + 1
    return xs * ny * nz + nx * ys * nz + nx * ny * zs + nx * ny * nz


def work(case):
    """Per solve: the previous state and one byte of material per cell in, the new state out, and
    one application of the operator (17 couplings in an A row, 37 in a V row); the fields out."""
    if case["kind"] == "requests":
        sizes = [_REQUEST_SIZES[q % 3] for q in range(case["count"])]
        solves, cells = 1 + case["steps"], sum(a * b * c for a, b, c in sizes)
        n = sum(_unknowns(*s) for s in sizes)
        out = sum(24.0 * a * b for a, b, c in sizes)
        return {"bytes": 8.0 * cells + solves * (16.0 * n + cells + out), "flops": solves * 2.0 * 88 * cells}
    xs, ys, zs = case["xs"], case["ys"], case["zs"]
    n, cells = _unknowns(xs, ys, zs), xs * ys * zs
    solve, flops = 16.0 * n + cells, 2.0 * 88 * cells
    if case["kind"] == "residual":
        return {"bytes": 24.0 * n + cells, "flops": flops}
    if case["kind"] == "steady":
        return {"bytes": solve + 24.0 * cells, "flops": flops}
    return {"bytes": case["steps"] * (solve + 24.0 * xs * ys) + 8.0 * n + (24.0 * cells if case["cubes"] else 0.0),
            "flops": case["steps"] * flops}


# --------------------------------------------------------------------------- 64 bits
class _Yee:
    """The Yee-grid A-V system in plain torch, 64 bits: arrays [..., k, j, i], 0-based, i fastest."""

    def __init__(self, inp, geom, device):
        self.xs, self.ys, self.zs = inp.xs, inp.ys, inp.zs
        self.h = (inp.dx, inp.dy, inp.dz)
        self.dt = inp.dt
        slots, rows = _slots(inp, geom)
        cell = torch.from_numpy(slots.reshape(self.zs, self.ys, self.xs).astype(np.int64)).to(device)
        tab = torch.tensor(np.concatenate([[[1.0, 1, 1, 0, 0, 0]], rows]), dtype=torch.float64, device=device)
        nk, nj, ni = self.shape = (self.zs + 1, self.ys + 1, self.xs + 1)
        self.blocks = [(nk, nj, self.xs), (nk, self.ys, ni), (self.zs, nj, ni), (nk, nj, ni)]
        self.n = [a * b * c for a, b, c in self.blocks]
        self.mu, self.sg = [], []
        for a in range(3):                                   # axis x, y, z
            ax = 2 - a
            mu, sg = tab[:, a][cell] * MU0, tab[:, 3 + a][cell]
            f = torch.full(self.shape, MU0, dtype=torch.float64, device=device)
            one, other = mu[1:, 1:, 1:], mu[tuple(slice(0, -1) if d == ax else slice(1, None) for d in range(3))]
            f[1:-1, 1:-1, 1:-1] = 2.0 * one * other / (one + other)
            self.mu.append(f)
            e = torch.zeros(self.shape, dtype=torch.float64, device=device)
            u, v = [d for d in range(3) if d != ax]
            for du in (0, 1):
                for dv in (0, 1):
                    at = [slice(1, None)] * 3
                    at[u] = slice(1, None) if du == 0 else slice(0, -1)
                    at[v] = slice(1, None) if dv == 0 else slice(0, -1)
                    e[1:-1, 1:-1, 1:-1] += 0.25 * sg[tuple(at)]
            self.sg.append(e)
        self.box = _interior(self.xs, self.ys, self.zs)
        self.device = device

    def split(self, x):
        out, at = [], 0
        for n, shape in zip(self.n, self.blocks):
            out.append(x[..., at:at + n].reshape(x.shape[:-1] + shape))
            at += n
        return out

    def join(self, parts):
        return torch.cat([p.reshape(p.shape[:-3] + (-1,)) for p in parts], -1)

    def _at(self, q, arr, d=(0, 0, 0)):
        """arr at every interior row of block q, shifted by d = (x, y, z)."""
        return arr[(...,) + tuple(slice(b.start + d[2 - t], b.stop + d[2 - t]) for t, b in enumerate(self.box[q]))]

    def apply(self, x, v, transient):
        """(M x, diag M)."""
        X = self.split(x)
        y = [p.clone() for p in X]
        diag = [torch.ones(s, dtype=torch.float64, device=self.device) for s in self.blocks]
        h, idt = self.h, (1.0 / self.dt if transient else 0.0)
        e = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]

        def add(*ds):
            return tuple(sum(c) for c in zip(*ds))

        def neg(d):
            return tuple(-c for c in d)

        for a in range(3):
            def S(arr, *ds):
                return self._at(a, arr, add((0, 0, 0), *ds))
            s = S(self.sg[a])
            acc, d = s * idt * S(X[a]), s * idt
            up, um = 1.0 / S(self.mu[a]) / h[a] ** 2, 1.0 / S(self.mu[a], neg(e[a])) / h[a] ** 2
            acc = acc + up * (S(X[a]) - S(X[a], e[a])) + um * (S(X[a]) - S(X[a], neg(e[a])))
            d = d + up + um
            for b in range(3):
                if b == a:
                    continue
                c = 3 - a - b                               # the face normal to a and b
                mp, mm = 1.0 / S(self.mu[c]), 1.0 / S(self.mu[c], neg(e[b]))
                acc = acc + mp / h[b] ** 2 * (S(X[a]) - S(X[a], e[b])) + mm / h[b] ** 2 * (S(X[a]) - S(X[a], neg(e[b])))
                d = d + (mp + mm) / h[b] ** 2
                sv = s * v[b]
                acc = acc + sv / (2 * h[b]) * (S(X[a], neg(e[b])) - S(X[a], e[b]))
                acc = acc + (mm / (h[a] * h[b]) - sv / (2 * h[a])) * (S(X[b], neg(e[b])) - S(X[b], neg(e[b]), e[a]))
                acc = acc + (mp / (h[a] * h[b]) + sv / (2 * h[a])) * (S(X[b], e[a]) - S(X[b]))
            acc = acc + s / h[a] * (S(X[3], e[a]) - S(X[3]))
            self._at(a, y[a])[...] = acc
            self._at(a, diag[a])[...] = d

        def S(arr, *ds):
            return self._at(3, arr, add((0, 0, 0), *ds))
        floor = float(np.float32(1e-12))
        acc, d = 0.0, 0.0
        for a in range(3):
            s0, s1 = S(self.sg[a]), S(self.sg[a], neg(e[a]))
            f0, f1 = s0.clamp_min(floor) / h[a] ** 2, s1.clamp_min(floor) / h[a] ** 2
            acc = acc + f0 * (S(X[3]) - S(X[3], e[a])) + f1 * (S(X[3]) - S(X[3], neg(e[a])))
            d = d + f0 + f1
            acc = acc + idt / h[a] * (s0 * S(X[a]) - s1 * S(X[a], neg(e[a])))
            for b in range(3):                              # div(sigma v x curl A)
                if b == a:
                    continue
                t0, t1 = S(self.sg[b]), S(self.sg[b], neg(e[b]))
                acc = acc + v[b] / (2 * h[a] * h[b]) * (
                    s1 * (S(X[a], neg(e[a]), neg(e[b])) - S(X[a], neg(e[a]), e[b])) + s0 * (S(X[a], e[b]) - S(X[a], neg(e[b]))))
                pair = S(X[a], neg(e[a])) + S(X[a])
                acc = acc + v[a] / (2 * h[b] ** 2) * (
                    t1 * (pair - S(X[a], neg(e[a]), neg(e[b])) - S(X[a], neg(e[b])))
                    + t0 * (pair - S(X[a], neg(e[a]), e[b]) - S(X[a], e[b])))
        self._at(3, y[3])[...] = acc
        self._at(3, diag[3])[...] = d
        return self.join(y), self.join(diag)

    def rhs(self, xprev, v, B, G):
        """Right-hand side: the background field's potential on the Dirichlet rows, sigma A / dt and its
        divergence elsewhere (zero for the steady state, xprev None)."""
        B, G, third = np.asarray(B, float), np.reshape(np.asarray(G, float), (3, 3)), float(np.float32(1.0 / 3.0))
        out = []
        X = self.split(xprev) if xprev is not None else None
        for q, shape in enumerate(self.blocks):
            z, y, x = torch.meshgrid(*[torch.arange(m, dtype=torch.float64, device=self.device) * s
                                       for m, s in zip(shape, self.h[::-1])], indexing="ij")
            p = (x, y, z)
            gr = [sum(G[r][c] * p[c] for c in range(3)) for r in range(3)]
            if q < 3:
                a, c = (q + 1) % 3, (q + 2) % 3
                b = 0.5 * B[a] * p[c] - 0.5 * B[c] * p[a] + third * (gr[a] * p[c] - gr[c] * p[a])
            else:
                b = sum(-((v[(r + 1) % 3] * (B[(r + 2) % 3] + 0.5 * gr[(r + 2) % 3])
                           - v[(r + 2) % 3] * (B[(r + 1) % 3] + 0.5 * gr[(r + 1) % 3])) * p[r]) for r in range(3))
            b = b.clone()
            inner = self._at(q, b)
            if X is None:
                inner[...] = 0.0
            elif q < 3:
                inner[...] = self._at(q, self.sg[q]) / self.dt * self._at(q, X[q])
            else:
                acc = 0.0
                for a in range(3):
                    m = tuple(-1 if t == a else 0 for t in range(3))
                    acc = acc + (self._at(3, self.sg[a]) * self._at(3, X[a])
                                 - self._at(3, self.sg[a], m) * self._at(3, X[a], m)) / (self.dt * self.h[a])
                inner[...] = acc
            out.append(b)
        return self.join(out)

    def field(self, x):
        """H at the cell centres, [k, j, i] per component."""
        A = self.split(x)[:3]
        h, out = self.h, []
        for a in range(3):
            b, c = (a + 1) % 3, (a + 2) % 3

            def diff(arr, t):
                t = 2 - t
                return arr.narrow(t, 1, arr.shape[t] - 1) - arr.narrow(t, 0, arr.shape[t] - 1)
            curl = diff(A[c], b) / h[b] - diff(A[b], c) / h[c]        # on faces normal to a
            w = curl / self.mu[a][tuple(slice(0, m) for m in curl.shape)]
            t = 2 - a
            out.append(0.5 * (w.narrow(t, 0, w.shape[t] - 1) + w.narrow(t, 1, w.shape[t] - 1)))
        return out

    def factor(self, v, transient):
        """The dense matrix, rows scaled by their diagonal, and its LU factors."""
        n = sum(self.n)
        M = torch.empty(n, n, dtype=torch.float64, device=self.device)
        d = None
        for at in range(0, n, 256):
            e = torch.zeros(min(256, n - at), n, dtype=torch.float64, device=self.device)
            e[torch.arange(e.shape[0]), at + torch.arange(e.shape[0])] = 1.0
            y, d = self.apply(e, v, transient)
            M[:, at:at + e.shape[0]] = (y / d).T
        return M, d, torch.linalg.lu_factor(M)

    @staticmethod
    def solve(factor, b):
        M, d, lu = factor
        b = (b / d)[:, None]
        x = torch.linalg.lu_solve(*lu, b)
        for _ in range(4):
            x = x + torch.linalg.lu_solve(*lu, b - M @ x)
        return x[:, 0]


def exact(case, seed):
    """The residual over all sizes; runs of steps on grids that a dense direct solver still takes
    (a larger run has no plain solution in reach of some seconds)."""
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "residual":
        inp, slots, rows, x, b, v = _residual_inputs(case, seed)
        _, geom, _ = _workload(case, seed)
        yee = _Yee(inp, geom, device)
        y, d = yee.apply(x, v, True)
        r, k = (b - y) / d, sum(yee.n[:3])
        return {"r": r, "sums": torch.stack([t.square().sum() for t in (r[:k], r[k:], x[:k], x[k:])])}
    if case["kind"] != "steps" or _unknowns(case["xs"], case["ys"], case["zs"]) > 14000:
        return None
    inp, geom, vel = _workload(case, seed)
    yee = _Yee(inp, geom, device)
    x = yee.solve(yee.factor([0.0] * 3, False), yee.rhs(None, [0.0] * 3, *scaled_field(inp.B, inp.G, inp.excitation, 0.0)))
    k = sum(yee.n[:3])
    x[k:] = 0.0                                              # no potential without motion
    out, factor, last = [], None, None
    for n, v in enumerate(vel):
        if v != last:
            factor, last = yee.factor(v, True), v
        x = yee.solve(factor, yee.rhs(x, v, *scaled_field(inp.B, inp.G, inp.excitation, (n + 1) * inp.dt)))
        H = yee.field(x)
        t = {"x": 2, "y": 1, "z": 0}[inp.slice_axis]
        out.append(torch.stack([f.select(t, inp.slice_index - 1).reshape(-1) for f in H]))
    cubes = [f.permute(2, 1, 0) for f in H] if case["cubes"] else None
    return {"slices": torch.stack(out), "cubes": cubes}
