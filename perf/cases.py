"""The work that users of this framework have it do, as timed cases.

Five kinds of call, each through the public entry points:

* ``step``: one ``FlowSolver.timestep()`` (three SIMPLE passes) on a box in the
  corrected SIMPLE mode with particle sources, the five coupled fields read
  into the program's pinned buffers afterwards;
* ``compat``: the same in the reference's mode with all scalar transports,
  all thirteen fields read;
* ``coupled``: the step of a spray program: particle rows ingested, one
  timestep, the flow state interpolated to the nodes of the particles' cells;
* ``predict`` / ``train``: the learned pressure guess on its own (inference on
  one sample; loss and gradient of a batch);
* ``bicgstab``: the allocation-free solve of one transport system that the
  caller holds in device memory.

A case is a dict of plain values.  ``prepare`` makes what a program holds
before the call (mesh, handle, initial fields, inputs), ``run`` makes one call,
``exact`` restates it in 64 bits with plain torch on the uniform box.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from minicombust_app_b200 import flow, gnn, train_guess
from minicombust_app_b200.workload import gaussian_blobs, noisy_fields

LENGTHS = (0.2, 0.1, 0.1)              # the benchmark's domain
FIELDS = ("U", "V", "W", "P", "TEM")
BLOBS_PER_CELL = 1000 / 4194304        # the benchmark's source density
PASSES = 3                             # SIMPLE passes of one timestep
SOURCE_UNIT = (1.0, 0.0, 0.0, 1.0e3, 1.0e-2)  # momentum x, y, z, energy, mass of a unit source


def _step(name, dims, **options):
    case = {"name": name, "kind": "step", "nx": dims[0], "ny": dims[1], "nz": dims[2], "amg": True, "refined": False,
            "guess": "zero", "rcm": False}
    case.update(options)
    return case


def listed():
    return [
        # the smallest run: a unit test or a tutorial box; launches and host work count
        _step("step_1k_amg", (16, 8, 8)),
        # the drop-in use: the reference's mode, constants and 16,000-cell mesh, all scalars transported
        {"name": "compat_16k_scalars", "kind": "compat", "nx": 40, "ny": 20, "nz": 20},
        # a program that leaves the solver options at their defaults (Jacobi-preconditioned CG)
        _step("step_221k_default", (96, 48, 48), amg=False),
        # refined solves started from the previous correction, on a ragged box
        _step("step_305k_refined_ragged", (101, 67, 45), refined=True, guess="previous"),
        # a spray program: 50,000 particle rows in, three passes, node values out
        {"name": "coupled_65k", "kind": "coupled", "nx": 64, "ny": 32, "nz": 32, "rows": 50000},
        # the half-million-cell configuration with cells in reverse Cuthill-McKee order
        _step("step_524k_rcm", (128, 64, 64), rcm=True),
        # the benchmark box, plain FP64
        _step("step_4m_plain", (256, 128, 128)),
        # the benchmark box with every accelerated option on
        _step("step_4m_learned_refined", (256, 128, 128), refined=True, guess="learned"),
        # inference of the guess network for an outside solver
        {"name": "predict_524k", "kind": "predict", "nx": 128, "ny": 64, "nz": 64, "shuffled": False},
        # one training batch at the training box's size
        {"name": "train_65k_batch8", "kind": "train", "nx": 64, "ny": 32, "nz": 32, "batch": 8},
        # the allocation-free solve inside a host's time loop: small, and at its size limit
        {"name": "bicgstab_3k", "kind": "bicgstab", "nx": 19, "ny": 13, "nz": 12},
        {"name": "bicgstab_262k", "kind": "bicgstab", "nx": 64, "ny": 64, "nz": 64},
    ]


def _box(rng, lo, hi):
    """A box of about 2m x m x m cells, lo <= cells <= hi (log-uniform), ragged."""
    while True:
        cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        m = (cells / 2) ** (1 / 3)
        dims = [max(4, int(round(f * m * rng.uniform(0.75, 1.33)))) for f in (2, 1, 1)]
        if lo <= dims[0] * dims[1] * dims[2] <= hi and dims[0] <= 512:
            return {"nx": dims[0], "ny": dims[1], "nz": dims[2]}


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "compat", "coupled", "predict", "train", "bicgstab"])
    if kind == "step":
        amg = rng.random() < 0.85
        refined = amg and rng.random() < 0.5
        guess = rng.choice(["zero", "previous", "learned"]) if amg else "zero"
        case = _step("", (0, 0, 0), amg=amg, refined=refined, guess=guess, rcm=rng.random() < 0.25)
        del case["name"]
        case.update(_box(rng, 1000, 2000000 if amg else 300000))
        return case
    if kind == "compat":
        return {"kind": kind, **_box(rng, 500, 40000)}
    if kind == "coupled":
        return {"kind": kind, **_box(rng, 2000, 300000), "rows": int(math.exp(rng.uniform(math.log(500), math.log(200000))))}
    if kind == "predict":
        return {"kind": kind, **_box(rng, 2000, 2000000), "shuffled": rng.random() < 0.25}
    if kind == "train":
        return {"kind": kind, **_box(rng, 2000, 140000), "batch": rng.randint(1, 8)}
    return {"kind": kind, "nx": rng.randint(5, 64), "ny": rng.randint(5, 64), "nz": rng.randint(5, 64)}


# ------------------------------------------------------------------- inputs

def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _cells(case):
    return case["nx"] * case["ny"] * case["nz"]


@functools.lru_cache(maxsize=4)
def _mesh(dims, shuffled=False):
    mesh = flow.Mesh.box(*dims, *LENGTHS)
    return mesh.renumbered(mesh.rcm_order()) if shuffled else mesh


def _params(case):
    if case["kind"] == "compat":
        return flow.default_params(flow.MODE_COMPAT)
    if case["kind"] == "coupled":
        return flow.default_params(flow.MODE_SIMPLE, pressure_solver=flow.PSOLVER_PCG_AMG)
    guess = {"zero": flow.GUESS_ZERO, "previous": flow.GUESS_PREVIOUS, "learned": flow.GUESS_LEARNED}[case["guess"]]
    return flow.default_params(
        flow.MODE_SIMPLE, pressure_solver=flow.PSOLVER_PCG_AMG if case["amg"] else flow.PSOLVER_PCG_JACOBI,
        precision=flow.PRECISION_FP32_REFINED if case["refined"] else flow.PRECISION_FP64, initial_guess=guess,
        reorder=flow.REORDER_RCM if case["rcm"] else flow.REORDER_NONE)


def _initial_fields(case, seed):
    return noisy_fields(_cells(case), seed, t0=2000.0 if case["kind"] == "compat" else 1500.0)


def _blob_sources(case, seed):
    return gaussian_blobs(_dims(case), LENGTHS, max(1, round(BLOBS_PER_CELL * _cells(case))), seed)


def _particles(case, seed):
    """Particle rows of a spray cone opening from the inlet: cell ids in arrival order and their source terms."""
    nx, ny, nz = _dims(case)
    rng = np.random.default_rng(seed)
    n = case["rows"]
    x = rng.beta(1.2, 4.0, n)
    spread = 0.05 + 0.3 * x
    y = np.clip(0.5 + spread * rng.standard_normal(n) / 2, 0, 0.999)
    z = np.clip(0.5 + spread * rng.standard_normal(n) / 2, 0, 0.999)
    cells = (x * nx).astype(np.int64) + nx * ((y * ny).astype(np.int64) + ny * (z * nz).astype(np.int64))
    inflow = 1.2 * 50.0 * (LENGTHS[1] / ny) * (LENGTHS[2] / nz)
    size = 1e-3 * inflow * rng.uniform(0.1, 1.0, n)
    terms = size[:, None] * np.array(SOURCE_UNIT)[None, :]
    terms[:, 1:3] = size[:, None] * rng.uniform(-0.2, 0.2, (n, 2))
    return cells.astype(np.uint64), terms


def _spray_cells(case):
    """The cells whose flow state the particle side asks for: the block around the spray."""
    nx, ny, nz = _dims(case)
    keep = lambda n, lo, hi: np.arange(int(lo * n), max(int(lo * n) + 1, int(hi * n)))  # noqa: E731
    z, y, x = np.meshgrid(keep(nz, 0.2, 0.8), keep(ny, 0.2, 0.8), keep(nx, 0.0, 0.7), indexing="ij")
    return (x + nx * (y + ny * z)).reshape(-1).astype(np.uint64)


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _smooth(shape, g):
    """A smooth random field (a coarse random grid, interpolated) of unit variance."""
    coarse = torch.randn((1, 1) + tuple(max(2, s // 8) for s in shape), device="cuda", generator=g)
    f = torch.nn.functional.interpolate(coarse, size=shape, mode="trilinear", align_corners=True).reshape(-1)
    return (f - f.mean()) / f.std()


def _blobs(shape, g):
    """Local sources of a few cells' width (the benchmark's density, at least four) of unit variance and mean zero."""
    n = math.prod(shape)
    f = torch.zeros(n, device="cuda")
    f[torch.randint(0, n, (max(4, round(BLOBS_PER_CELL * n)),), device="cuda", generator=g)] = 1.0
    taps = torch.exp(-0.5 * (torch.arange(-6, 7, device="cuda") / 2.0) ** 2)
    f = f.reshape(1, 1, *shape)
    for axis in range(3):
        kernel, pad = [1, 1, 1], [0, 0, 0]
        kernel[axis], pad[axis] = 13, 6
        f = torch.nn.functional.conv3d(f, taps.reshape(1, 1, *kernel), padding=pad)
    f = f.reshape(-1)
    return (f - f.mean()) / f.std()


def _network_samples(case, seed, count):
    """Records like those of the pressure solves: a right-hand side of mean zero (the divergence of noisy initial
    fields, mass sources of a few cells' width), the matrix diagonal (smaller on the boundary), previous and converged corrections of the
    order of (right-hand side) / (diagonal)."""
    nx, ny, nz = _dims(case)
    shape, g = (nz, ny, nx), _generator(seed)
    faces = torch.full(shape, 6.0, device="cuda")
    for axis in range(3):
        faces.select(axis, 0).sub_(1)
        faces.select(axis, -1).sub_(1)
    out = []
    for _ in range(count):
        noise = torch.randn(nx * ny * nz, device="cuda", generator=g)
        rhs = (noise + 0.02 * _blobs(shape, g)) * 1e-7
        rhs = rhs - rhs.mean()
        diag = 2e-9 * faces.reshape(-1) * (1 + 0.02 * _smooth(shape, g))
        unit = rhs.std() / diag.mean()
        target = unit * _smooth(shape, g)
        prev = 0.3 * unit * _smooth(shape, g)
        out.append(tuple(t.contiguous() for t in (rhs, diag, prev, target)))
    return out


def _transport_system(case, seed):
    """One implicit transport step on a box in the library's row layout: upwind convection along a varying x-velocity
    with cross flow, diffusion, a transient term; unused slots point at their own row."""
    nx, ny, nz = _dims(case)
    n, g = nx * ny * nz, _generator(seed)
    i = torch.arange(n, device="cuda", dtype=torch.int32)
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    has = [z > 0, y > 0, x > 0, x < nx - 1, y < ny - 1, z < nz - 1]
    step = [-nx * ny, -nx, -1, 1, nx, nx * ny]
    along = [0.15, 0.25, 1.5, 0.05, 0.05, 0.05]  # inflow through each side, in units of the cell's content per step
    off = torch.zeros((6, n), device="cuda", dtype=torch.float64)
    col = torch.empty((6, n), device="cuda", dtype=torch.int32)
    for k in range(6):
        value = along[k] * (0.6 + 0.8 * torch.rand(n, device="cuda", dtype=torch.float64, generator=g)) + 0.1
        off[k] = torch.where(has[k], -value, 0.0)
        col[k] = torch.where(has[k], i + step[k], i)
    diag = 1.0 - off.sum(0)
    b = 1500.0 * (1.0 + 0.01 * torch.randn(n, device="cuda", dtype=torch.float64, generator=g))
    return diag, off, col, b


# ------------------------------------------------------------ prepare and run

def _set_fields(solver, values):
    for name, v in values.items():
        a = solver.field(name)
        a[:solver.N] = v
        solver.set_field(name, a)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "compat", "coupled"):
        solver = flow.FlowSolver(_mesh(_dims(case)), params=_params(case))
        _set_fields(solver, _initial_fields(case, seed))
        if kind == "step":
            solver.set_sources(_blob_sources(case, seed))
            if case["guess"] == "learned":
                solver.set_guess_params(train_guess.load_params())
        names = tuple(flow.FIELDS) if kind == "compat" else FIELDS
        state = {"kind": kind, "solver": solver,
                 "out": {n: torch.empty(solver.N + 6, dtype=torch.float64, pin_memory=True) for n in names}}
        if kind == "coupled":
            state["cells"], state["terms"] = _particles(case, seed)
            state["wanted"] = _spray_cells(case)
            # the handle's node tables, made once by a first query
            count = ctypes.c_int64()
            solver.L.mc_flow_interpolate_nodes(solver.h, 1, state["wanted"].ctypes.data, 0, ctypes.byref(count), None,
                                               None)
            torch.cuda.synchronize()
        return state
    if kind in ("predict", "train"):
        net = gnn.GuessNet(seed=0)
        net.set_params(train_guess.load_params())
        graph = net.graph(_mesh(_dims(case), case.get("shuffled", False)))
        state = {"kind": kind, "net": net, "graph": graph,
                 "samples": _network_samples(case, seed, case.get("batch", 1))}
        if kind == "predict":
            state["y"] = torch.empty(_cells(case), device="cuda")
            state["x0"] = torch.empty(_cells(case), device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        return state
    diag, off, col, b = _transport_system(case, seed)
    torch.cuda.synchronize()
    return {"kind": kind, "L": flow.library(), "diag": diag, "off": off, "col": col, "b": b, "x": torch.empty_like(b),
            "iterations": ctypes.c_int()}


def _read_fields(state):
    solver = state["solver"]
    for name, buffer in state["out"].items():
        if solver.L.mc_flow_get_field(solver.h, flow.FIELDS[name], buffer.data_ptr()) != flow.MC_OK:
            raise RuntimeError(f"field {name} cannot be read")
    return state["out"]


def run(state):
    kind = state["kind"]
    if kind in ("step", "compat"):
        state["solver"].timestep()
        return _read_fields(state)
    if kind == "coupled":
        solver = state["solver"]
        solver.ingest_particles(state["cells"], state["terms"])
        solver.timestep()
        ids, values = solver.interpolate_nodes(state["wanted"])
        return {"node_ids": ids.astype(np.int64), "node_values": values, **_read_fields(state)}
    if kind == "predict":
        rhs, diag, prev, _ = state["samples"][0]
        state["net"].predict(state["graph"], rhs, diag, prev, y=state["y"], x0=state["x0"])
        return {"y": state["y"], "x0": state["x0"]}
    if kind == "train":
        loss, grad = state["net"].loss_grad(state["graph"], state["samples"])
        return {"loss": loss, "grad": grad}
    rc = state["L"].mc_solve_bicgstab_noalloc(
        state["b"].numel(), state["diag"].data_ptr(), state["off"].data_ptr(), state["col"].data_ptr(),
        state["b"].data_ptr(), state["x"].data_ptr(), 1e-8, 1000, torch.cuda.current_stream().cuda_stream,
        ctypes.byref(state["iterations"]))
    if rc != flow.MC_OK:
        raise RuntimeError(f"mc_solve_bicgstab_noalloc: status {rc}")
    return state["x"]


# -------------------------------------------------------- work and tolerances

def _faces(case):
    nx, ny, nz = _dims(case)
    return (nx + 1) * ny * nz + nx * (ny + 1) * nz + nx * ny * (nz + 1)


def work(case):
    n, f, kind = _cells(case), _faces(case), case["kind"]
    if kind in ("step", "coupled"):
        # per pass: five fields and the face fluxes in and out, sources, face geometry; the fields copied out once
        per_pass = n * (2 * 5 * 8 + 5 * 8) + f * (2 * 8 + 9 * 8)
        rows = case.get("rows", 0) * 48
        return {"bytes": PASSES * per_pass + 5 * 8 * n + rows, "flops": PASSES * n * 2500.0}
    if kind == "compat":
        per_pass = n * (2 * 13 * 8) + f * (2 * 8 + 9 * 8)
        return {"bytes": PASSES * per_pass + 13 * 8 * n, "flops": PASSES * n * 6000.0}
    if kind == "predict":
        return {"bytes": n * (3 * 4 + 1 + 4 + 8), "flops": n * 4 * 2 * (64 * 32 + 32 * 32 + 6 * 32)}
    if kind == "train":
        return {"bytes": case["batch"] * n * 16, "flops": case["batch"] * 3 * n * 4 * 2 * (64 * 32 + 32 * 32 + 6 * 32)}
    # matrix, right-hand side and solution once; about 20 iterations of two products
    return {"bytes": n * (7 * 8 + 6 * 4 + 2 * 8), "flops": n * 20 * 50.0}


def tolerance(case):
    # about four times the differences measured against exact(), or (compat) between the two cell orders and the
    # 1e-13 its solves stop at
    kind = case["kind"]
    if kind in ("step", "coupled"):
        return {"rel": 2e-6, "max": 2e-5}
    if kind == "compat":
        return {"rel": 1e-10, "max": 4e-9}
    if kind == "predict":
        return {"rel": 1.5e-2, "max": 0.1}
    if kind == "train":
        return {"rel": 3e-2, "max": 0.4}
    return {"rel": 2.5e-8, "max": 1e-7}


# ---------------------------------------------------------------- exact values
#
# On the uniform box every face is orthogonal to the line between its cells, so the SIMPLE pass reduces to the
# formulas below.  Arrays are [nz][ny][nx]; a face direction is (axis of the array, side).

MU, RHO, U_IN, T_REF, DT = 1.8e-5, 1.2, 50.0, 1500.0, 1.0e-5
URF_U, URF_P, URF_T = 0.7, 0.3, 0.95
INLET_MU = MU + RHO * 0.09 * (1.5 * 0.01 * U_IN ** 2) / (0.09 ** 0.75 * (1.5 * 0.01 * U_IN ** 2) ** 1.5)
# boundary sides in slot order: z-min, z-max, x-min (inlet), x-max (outlet), y-min, y-max; (axis, last side?)
SIDES = ((0, 0), (0, 1), (2, 0), (2, 1), (1, 0), (1, 1))
INLET, OUTLET = 2, 3


class _Box:
    def __init__(self, dims):
        nx, ny, nz = dims
        self.shape = (nz, ny, nx)
        self.h = (LENGTHS[2] / nz, LENGTHS[1] / ny, LENGTHS[0] / nx)  # per array axis
        self.vol = self.h[0] * self.h[1] * self.h[2]
        self.area = tuple(self.vol / d for d in self.h)

    def cut(self, t, axis, side):
        return t.select(axis, -1 if side else 0)

    def last_cell(self, side):
        """The cell of a boundary side's last face."""
        axis, hi = SIDES[side]
        at = [-1, -1, -1]
        at[axis] = -1 if hi else 0
        return tuple(at)

    def pairs(self, t, axis):
        n = t.shape[axis]
        return t.narrow(axis, 0, n - 1), t.narrow(axis, 1, n - 1)

    def gradient(self, phi, boundary):
        """Least-squares gradient, [axis]; boundary: the six side values, or None for no difference across sides."""
        out = []
        for axis in range(3):
            h, n = self.h[axis], self.shape[axis]
            lo, hi = self.pairs(phi, axis)
            num, den = torch.zeros_like(phi), torch.zeros_like(phi)
            for part, d in (((0, n - 1), hi - lo), ((1, n - 1), hi - lo)):
                num.narrow(axis, *part).add_(d * h)
                den.narrow(axis, *part).add_(h * h)
            for s, (a, side) in enumerate(SIDES):
                if a != axis:
                    continue
                if boundary is not None:
                    d = boundary[s] - self.cut(phi, axis, side)
                    self.cut(num, axis, side).add_(d * (h / 2 if side else -h / 2))
                self.cut(den, axis, side).add_(h * h / 4)
            out.append(num / den)
        return out


def _apply(diag, off, x):
    """7-point product; off[axis] = (coupling of each cell to its lower neighbour, to its upper one) on the faces."""
    y = diag * x
    for axis in range(3):
        n = x.shape[axis]
        if n < 2:
            continue
        lower, upper = off[axis]
        y.narrow(axis, 1, n - 1).add_(lower * x.narrow(axis, 0, n - 1))
        y.narrow(axis, 0, n - 1).add_(upper * x.narrow(axis, 1, n - 1))
    return y


def _dot(a, b):
    return (a * b).sum()


def _bicgstab(apply, b, rtol=1e-13, limit=400):
    x, r = torch.zeros_like(b), b.clone()
    bb = float(_dot(b, b))
    if bb == 0:
        return x
    r0, p, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
    rho = alpha = omega = torch.ones((), dtype=b.dtype, device=b.device)
    best, at = x, math.inf
    for _ in range(limit):
        rho_new = _dot(r0, r)
        p = r + (rho_new / rho) * (alpha / omega) * (p - omega * v)
        v = apply(p)
        alpha = rho_new / _dot(r0, v)
        s = r - alpha * v
        t = apply(s)
        omega = _dot(t, s) / _dot(t, t)
        x = x + alpha * p + omega * s
        r = s - omega * t
        rho = rho_new
        rr = float(_dot(r, r))
        if not math.isfinite(rr):
            break
        if rr < at:
            best, at = x, rr
        if rr <= rtol * rtol * bb:
            break
    return best


def _cg_mean_free(diag, off, b, rtol=1e-12, limit=8000):
    b = b - b.mean()
    x, r = torch.zeros_like(b), b.clone()
    bb = float(_dot(b, b))
    z = r / diag
    p, rz = z.clone(), _dot(r, z)
    for it in range(limit):
        q = _apply(diag, off, p)
        alpha = rz / _dot(p, q)
        x += alpha * p
        r -= alpha * q
        if it % 16 == 15 and float(_dot(r, r)) <= rtol * rtol * bb:
            break
        z = r / diag
        rz_new = _dot(r, z)
        p = z + (rz_new / rz) * p
        rz = rz_new
    return x - x.mean()


class _Pass:
    """The corrected SIMPLE pass on the uniform box in FP64."""

    def __init__(self, dims, fields, sources):
        self.box = _Box(dims)
        shape = self.box.shape
        as3 = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda").reshape(shape)  # noqa: E731
        self.f = {k: as3(v).clone() for k, v in fields.items()}
        self.src = [as3(sources[:, k]) for k in range(5)]
        inlet_outlet = [U_IN if s in (INLET, OUTLET) else 0.0 for s in range(6)]
        self.bound = {"U": inlet_outlet, "V": [0.0] * 6, "W": [0.0] * 6, "P": [4000.0] * 6, "TEM": [T_REF] * 6}
        self.mass_source = float(self.src[4].sum())
        zero = torch.zeros(shape, dtype=torch.float64, device="cuda")
        self.m = None        # fluxes through internal faces per axis (towards the upper cell)
        self.m_in = self.m_out = None
        g = self.gradients()
        # the first pass's diagonal and fluxes: transient and inlet/outlet parts only
        b = self.box
        AU = zero + RHO * b.vol / DT
        for s in (INLET, OUTLET):
            axis, side = SIDES[s]
            b.cut(AU, axis, side).add_(MU * b.area[axis] / (b.h[axis] / 2))
        self.mass_flux(g, AU)

    def gradients(self):
        f, bd, b = self.f, self.bound, self.box
        return {k: b.gradient(f[k], None if k == "P" else bd[k]) for k in FIELDS}

    def mass_flux(self, g, AU):
        b, f = self.box, self.f
        vel = {2: f["U"], 1: f["V"], 0: f["W"]}
        self.m, self.apv = [], []
        for axis in range(3):
            u0, u1 = b.pairs(vel[axis], axis)
            p0, p1 = b.pairs(f["P"], axis)
            g0, g1 = b.pairs(g["P"][axis], axis)
            a0, a1 = b.pairs(AU, axis)
            apv = 0.5 * RHO * (1 / a0 + 1 / a1) * b.area[axis] * b.vol / b.h[axis]
            self.apv.append(apv)
            self.m.append(RHO * 0.5 * (u0 + u1) * b.area[axis] - apv * ((p1 - p0) - 0.5 * (g0 + g1) * b.h[axis]))
        inlet_area = b.area[2] * torch.ones_like(b.cut(f["U"], 2, 0))
        self.m_in = -RHO * U_IN * inlet_area  # outward
        out = RHO * b.cut(f["U"], 2, 1) * b.area[2]
        out = torch.where(out < 0, 1e-15, out)
        self.m_out = out * ((self.mass_source - self.m_in.sum()) / out.sum())

    def divergence(self):
        """Net outflow of each cell."""
        d = torch.zeros(self.box.shape, dtype=torch.float64, device="cuda")
        for axis in range(3):
            n = d.shape[axis]
            d.narrow(axis, 0, n - 1).add_(self.m[axis])
            d.narrow(axis, 1, n - 1).sub_(self.m[axis])
        self.box.cut(d, 2, 0).add_(self.m_in)
        self.box.cut(d, 2, 1).add_(self.m_out)
        return d

    def couplings(self, visc):
        off = []
        for axis in range(3):
            vis = visc * self.box.area[axis] / self.box.h[axis]
            off.append((-vis - torch.clamp(self.m[axis], min=0), -vis + torch.clamp(self.m[axis], max=0)))
        return off

    @staticmethod
    def row_sums(off, shape):
        s = torch.zeros(shape, dtype=torch.float64, device="cuda")
        for axis in range(3):
            n = shape[axis]
            s.narrow(axis, 1, n - 1).add_(off[axis][0])
            s.narrow(axis, 0, n - 1).add_(off[axis][1])
        return s

    def add_face_sum(self, total, q, axis, weight):
        """total += weight * (mean of q over a cell's two faces of this axis, signed outward), internal faces."""
        q0, q1 = self.box.pairs(q, axis)
        face = 0.5 * weight * (q0 + q1)
        n = total.shape[axis]
        total.narrow(axis, 0, n - 1).add_(face)
        total.narrow(axis, 1, n - 1).sub_(face)

    def momentum(self, g):
        b, f, shape = self.box, self.f, self.box.shape
        names = ("W", "V", "U")  # the component along each array axis
        off = self.couplings(MU)
        ac = torch.zeros(shape, dtype=torch.float64, device="cuda")
        su = [torch.zeros_like(ac) for _ in range(3)]
        new_bound = {k: list(self.bound[k]) for k in "UVW"}
        # deferred viscous stress mu (grad u + grad u^T) . S less the implicit part mu grad u . S
        for axis in range(3):
            for c in range(3):
                self.add_face_sum(su[c], g[names[axis]][c], axis, MU * b.area[axis])
        for s in (INLET, OUTLET):
            axis, side = SIDES[s]
            sign = 1.0 if side else -1.0
            visc = INLET_MU if s == INLET else MU
            vis = visc * b.area[axis] / (b.h[axis] / 2)
            md = self.m_in if s == INLET else torch.where(self.m_out < 0, 1e-15, self.m_out)
            if s == OUTLET:
                self.m_out = md
            coef = -vis + torch.clamp(md, max=0)
            b.cut(ac, axis, side).sub_(coef)
            for c in range(3):
                cell = b.cut(f[names[c]], axis, side)
                uf = (U_IN if names[c] == "U" else 0.0) if s == INLET else cell
                stress = visc * b.area[axis] * sign * b.cut(g[names[axis]][c], axis, side)
                b.cut(su[c], axis, side).add_(stress - coef * uf)
                new_bound[names[c]][s] = (float(uf) if s == INLET else float(f[names[c]][b.last_cell(s)]))
        for s in range(6):
            if s in (INLET, OUTLET):
                continue
            axis, side = SIDES[s]
            coef = MU * b.area[axis] / (b.h[axis] / 2)
            b.cut(ac, axis, side).add_(coef)
            b.cut(su[axis], axis, side).add_(coef * b.cut(f[names[axis]], axis, side))
            for c in range(3):
                new_bound[names[c]][s] = 0.0
        buoyancy = -0.001 * RHO * b.vol * (f["TEM"] - T_REF)
        su[1] = su[1] - 9.81 * buoyancy
        transient = RHO * b.vol / DT
        source = (self.src[2], self.src[1], self.src[0])
        for c in range(3):
            su[c] = su[c] - g["P"][c] * b.vol + transient * f[names[c]] + source[c]
        ac = (ac + transient - self.row_sums(off, shape)) / URF_U
        for c in range(3):
            rhs = su[c] + (1 - URF_U) * ac * f[names[c]]
            f[names[c]] = _bicgstab(lambda v: _apply(ac, off, v), rhs)
        for k in "UVW":
            self.bound[k] = new_bound[k]
        return ac

    def pressure(self, g, AU):
        b, f = self.box, self.f
        self.mass_flux(g, AU)
        off = [(-a, -a) for a in self.apv]
        diag = -self.row_sums(off, b.shape)
        pp = _cg_mean_free(diag, off, self.src[4] - self.divergence())
        gp = b.gradient(pp, None)
        for axis in range(3):
            p0, p1 = b.pairs(pp, axis)
            self.m[axis] = self.m[axis] - self.apv[axis] * (p1 - p0)
        f["P"] = f["P"] + URF_P * pp
        for axis, name in enumerate(("W", "V", "U")):
            f[name] = f[name] - gp[axis] * (b.vol / AU)
        gP = b.gradient(f["P"], None)
        for s in range(6):
            axis, side = SIDES[s]
            at = b.last_cell(s)
            value = float(f["P"][at])
            if s != OUTLET:
                value += float(gP[axis][at]) * (b.h[axis] / 2 if side else -b.h[axis] / 2)
            self.bound["P"][s] = value
        return gP

    def temperature(self, g):
        b, f, shape = self.box, self.f, self.box.shape
        visc = MU / 0.6905
        off = self.couplings(visc)
        at = torch.zeros(shape, dtype=torch.float64, device="cuda")
        # on orthogonal faces the explicit diffusion and its implicit counterpart cancel
        st = torch.zeros_like(at)
        axis, side = SIDES[INLET]
        inlet_visc = (MU + (INLET_MU - MU) / 0.9) / 0.6905
        coef = -inlet_visc * b.area[axis] / (b.h[axis] / 2) + torch.clamp(self.m_in, max=0)
        b.cut(at, axis, side).sub_(coef)
        b.cut(st, axis, side).sub_(coef * T_REF)
        bound = [0.0] * 6
        for s in range(6):
            cell = b.last_cell(s)
            bound[s] = float(f["TEM"][cell])
            if s == INLET:
                bound[s] = T_REF
            elif s == OUTLET:
                bound[s] += float(g["TEM"][2][cell]) * b.h[2] / 2
        transient = RHO * b.vol / DT
        st = st + transient * f["TEM"] + self.src[3]
        at = (at + transient - self.row_sums(off, shape)) / URF_T
        rhs = st + (1 - URF_T) * at * f["TEM"]
        f["TEM"] = _bicgstab(lambda v: _apply(at, off, v), rhs)
        self.bound["TEM"] = bound

    def step(self):
        g = self.gradients()
        AU = self.momentum(g)
        gP = self.pressure(g, AU)
        self.temperature(g)
        return {**g, "P": gP}

    def fields(self):
        return {k: torch.cat([self.f[k].reshape(-1), torch.tensor(self.bound[k], dtype=torch.float64, device="cuda")])
                for k in FIELDS}


def _exact_nodes(p, g, wanted):
    """Node values of the wanted cells: the share of the inlet state for missing cells, then the cells' expansions."""
    nz, ny, nx = p.box.shape
    refs = {"U": U_IN, "V": 0.0, "W": 0.0, "P": 4000.0, "TEM": T_REF}
    count = torch.zeros((nz + 1, ny + 1, nx + 1), dtype=torch.float64, device="cuda")
    values = {k: torch.zeros_like(count) for k in FIELDS}
    flag = torch.zeros(count.shape, dtype=torch.bool, device="cuda")
    want = torch.zeros(nz * ny * nx, dtype=torch.bool, device="cuda")
    want[torch.as_tensor(wanted.astype(np.int64), device="cuda")] = True
    want = want.reshape(nz, ny, nx)
    for dz in (0, 1):
        for dy in (0, 1):
            for dx in (0, 1):
                at = (slice(dz, dz + nz), slice(dy, dy + ny), slice(dx, dx + nx))
                flag[at] |= want
                count[at] += 1
                offset = [(d - 0.5) * h for d, h in zip((dz, dy, dx), p.box.h)]
                for k in FIELDS:
                    values[k][at] += (p.f[k] + sum(g[k][a] * offset[a] for a in range(3))) / 8
    ids = flag.reshape(-1).nonzero().reshape(-1)
    cols = [(values[k] + refs[k] * (8 - count) / 8).reshape(-1)[ids] for k in FIELDS]
    return ids, torch.stack(cols, 1)


def _network(p, sample, shape, edges):
    """The network in FP64 over the box: scaled inputs, four message-passing layers, decoder; (y, unit of the guess)."""
    at = 0

    def take(*size):
        nonlocal at
        at += math.prod(size)
        return p[at - math.prod(size):at].reshape(size)

    rhs, diag, prev, _ = sample
    sb, sd = rhs.square().mean().sqrt(), diag.mean()
    sx = sb / sd
    x = torch.stack([rhs / sb, diag / sd, prev / sx, torch.ones_like(rhs)], 1)
    we, ce = take(32, 4), take(32)
    h = torch.relu(x @ we.T + ce)
    for _ in range(4):
        wg, cg, w1, c1, w2, c2 = take(32, 2), take(32), take(32, 64), take(32), take(32, 32), take(32)
        grid = h.reshape(*shape, 32)
        m = torch.zeros_like(grid)
        for axis in range(3):
            n = shape[axis]
            pad = [0, 0, 0, 0, 0, 0, 0, 0]   # widths of the last grid axis first
            pad[2 * (3 - axis) + 1] = 1
            upper = torch.nn.functional.pad(grid.narrow(axis, 1, n - 1), pad)
            lower = torch.nn.functional.pad(grid.narrow(axis, 0, n - 1), pad[:2 * (3 - axis)] + [1, 0] + pad[8 - 2 * axis:])
            m = m + (wg @ edges[axis] + cg) * (upper + lower)
        u = torch.cat([h, m.reshape(-1, 32)], 1)
        h = h + torch.relu(u @ w1.T + c1) @ w2.T + c2
    wd, cd, wo, co = take(32, 32), take(32), take(32), take(1)
    return torch.relu(h @ wd.T + cd) @ wo + co, sx


def _exact_network(case, samples, parameters, with_gradient):
    box = _Box(_dims(case))
    internal = [(s - 1) * math.prod(box.shape) // s for s in box.shape]
    ratio = [a / h for a, h in zip(box.area, box.h)]
    mean = lambda v: sum(a * c for a, c in zip(v, internal)) / sum(internal)  # noqa: E731
    edges = [torch.tensor([box.area[k] / mean(box.area), ratio[k] / mean(ratio)], dtype=torch.float64, device="cuda")
             for k in range(3)]
    p = torch.tensor(parameters, dtype=torch.float64, device="cuda", requires_grad=with_gradient)
    if not with_gradient:
        y, sx = _network(p, [t.double() for t in samples[0]], box.shape, edges)
        return {"y": y, "x0": y * sx}
    total = 0.0
    for sample in samples:
        sample = [t.double() for t in sample]
        y, sx = _network(p, sample, box.shape, edges)
        d = y - sample[3] / sx
        loss = (d - d.mean()).square().mean() / len(samples)
        loss.backward()
        total += float(loss.detach())
    return {"loss": total, "grad": p.grad.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "compat":
        return None  # the reference's mode carries its quirks (stale pressure system, one-cell correction)
    if kind == "step":
        p = _Pass(_dims(case), _initial_fields(case, seed), _blob_sources(case, seed))
        for _ in range(PASSES):
            p.step()
        return p.fields()
    if kind == "coupled":
        cells, terms = _particles(case, seed)
        sources = np.zeros((_cells(case), 5))
        np.add.at(sources, cells.astype(np.int64), terms)
        p = _Pass(_dims(case), _initial_fields(case, seed), sources)
        for _ in range(PASSES):
            g = p.step()
        ids, values = _exact_nodes(p, g, _spray_cells(case))
        return {"node_ids": ids, "node_values": values, **p.fields()}
    if kind in ("predict", "train"):
        if case.get("shuffled"):
            return None  # the cells' order is the mesh's own; the box case covers the values
        samples = _network_samples(case, seed, case.get("batch", 1))
        return _exact_network(case, samples, train_guess.load_params(), kind == "train")
    diag, off, col, b = _transport_system(case, seed)
    col = col.long()

    def product(x):
        return diag * x + (off * x[col]).sum(0)

    return _bicgstab(product, b)
