"""The workloads this framework is timed on: implicit finite-volume steps of
3-D and 2-D systems, batches of small boxes, and the learned preconditioner's
network, each through the public Python API.

A case is a dict of plain values.  ``path`` names the work:

* ``heat``    time loop of a bounded diffusion box (``timestep``, FP64)
* ``tvd``     time loop of TVD convection-diffusion (``timestep``, FP64)
* ``species`` 2-D, two species, a functor composed of terms, the driver loop
              written out call by call (Build, Solve, CopyTo, halo, old level)
* ``refine``  step with heterogeneous diffusivity, FP32 inner solves
* ``batch``   time loop of many uneven boxes, read back to the host
* ``apply``   one application of the preconditioner network
* ``grad``    loss and weight gradient of the network on a minibatch
* ``learned`` Build and learned-preconditioned solve
* ``host``    time loop of a field that lives in pinned host memory

Sizes are those of the benchmark and of the tests (64^3 diffusion, 128^3 and
256^3 TVD, boxes of 16 to 64 cells a side, networks on 128^3 and 64^3 grids)
and ragged ones in between.
"""
import math

import numpy as np
import torch

import dare_b200 as D

TOL = 1e-10        # relative residual of every solve, as in the benchmark
DEV = "cuda:0"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest calls: a 2-D verification-style run of two species,
        # where launches and host round trips are all there is
        {"name": "species_96x80", "path": "species", "n0": 96, "n1": 80, "limiter": "MINMOD", "steps": 10},
        # the 64^3 diffusion run of ten steps (Gaussian bump and noise)
        {"name": "heat_64", "path": "heat", "n0": 64, "n1": 64, "n2": 64, "steps": 10},
        # a ragged box: odd rows, two periodic directions, walls in the third
        {"name": "tvd_97x61x75", "path": "tvd", "n0": 97, "n1": 61, "n2": 75, "wall": 1, "limiter": "VANALBADA",
         "steps": 2},
        # an ordinary transport step, and the benchmark's headline size
        {"name": "tvd_128", "path": "tvd", "n0": 128, "n1": 128, "n2": 128, "wall": -1, "limiter": "VANLEER",
         "steps": 2},
        {"name": "tvd_256", "path": "tvd", "n0": 256, "n1": 256, "n2": 256, "wall": -1, "limiter": "VANLEER",
         "steps": 1},
        # the largest grid: mixed precision with heterogeneous diffusivity
        {"name": "refine_384", "path": "refine", "n0": 384, "n1": 384, "n2": 384, "steps": 1},
        # batches of independent boxes: the benchmark's sides, and small ragged ones
        {"name": "batch_uneven_256", "path": "batch", "count": 256, "sides": "16,24,32,48,64", "ragged": False,
         "steps": 20},
        {"name": "batch_small_1024", "path": "batch", "count": 1024, "sides": "7,10,13,16,20,25", "ragged": True,
         "steps": 20},
        # the network of a 256^3 system (coarse form, 128^3 convolutions)
        {"name": "apply_256", "path": "apply", "n0": 256, "n1": 256, "n2": 256, "coarse": True},
        # one training minibatch of restricted 128^3 pairs
        {"name": "grad_64x4", "path": "grad", "n0": 64, "n1": 64, "n2": 64, "count": 4},
        # a learned-preconditioned solve at the size the network is trained for
        {"name": "learned_128", "path": "learned", "n0": 128, "n1": 128, "n2": 128},
        # steps of a field kept in host memory (uploads and downloads included)
        {"name": "host_256", "path": "host", "n0": 256, "n1": 256, "n2": 256, "wall": -1, "limiter": "VANLEER",
         "steps": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi, multiple=1):
    """Three sides about one log-uniform size, each within [lo, hi]."""
    base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    out = []
    for _ in range(3):
        s = int(round(base * rng.uniform(0.75, 1.25) / multiple)) * multiple
        out.append(min(hi, max(lo, s)))
    return {"n0": out[0], "n1": out[1], "n2": out[2]}


def draw(rng):
    path = rng.choice(["species", "heat", "tvd", "tvd", "refine", "batch", "apply", "grad", "learned", "host"])
    if path == "species":
        return {"path": path, "n0": _log_int(rng, 24, 400), "n1": _log_int(rng, 24, 400),
                "limiter": rng.choice(["MINMOD", "VANLEER", "VANALBADA", "UPWIND"]), "steps": 10}
    if path == "heat":
        return {"path": path, **_sides(rng, 16, 144), "steps": 10}
    if path == "tvd":
        return {"path": path, **_sides(rng, 24, 256), "wall": rng.choice([-1, -1, 0, 1, 2]),
                "limiter": rng.choice(["VANLEER", "VANLEER", "MINMOD", "VANALBADA", "UPWIND"]), "steps": 1}
    if path == "refine":
        return {"path": path, **_sides(rng, 64, 320), "steps": 1}
    if path == "batch":
        lo = rng.randint(6, 16)
        hi = _log_int(rng, 20, 64)
        sides = sorted({rng.randint(lo, hi) for _ in range(5)})
        count = max(32, min(1024, int(1.6e7 / (sum(s ** 3 for s in sides) / len(sides)))))
        return {"path": path, "count": int(count * rng.uniform(0.3, 1.0)), "sides": ",".join(map(str, sides)),
                "ragged": rng.random() < 0.5, "steps": 20}
    if path == "apply":
        coarse = rng.random() < 0.7
        return {"path": path, **_sides(rng, 32, 256 if coarse else 128, 16 if coarse else 8), "coarse": coarse}
    if path == "grad":
        return {"path": path, **_sides(rng, 16, 64, 8), "count": rng.randint(1, 6)}
    if path == "learned":
        return {"path": path, **_sides(rng, 64, 192, 16)}
    return {"path": "host", **_sides(rng, 48, 240), "wall": -1, "limiter": "VANLEER", "steps": 2}


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _modes(rng, n, offsets, decay=2.0, count=8, kmax=8):
    """Sum of `count` separable periodic modes on the points (i + offset) / n."""
    x = [(torch.arange(n[d], dtype=torch.float64, device=DEV) + offsets[d]) / n[d] for d in range(3)]
    out = torch.zeros(n, dtype=torch.float64, device=DEV)
    for _ in range(count):
        k = rng.integers(1, kmax + 1, size=3)
        ph = rng.uniform(0.0, 2.0 * math.pi, size=3)
        a = float(rng.normal()) / float(np.dot(k, k)) ** (decay / 2.0)
        f = [torch.sin(2.0 * math.pi * float(k[d]) * x[d] + float(ph[d])) for d in range(3)]
        out += a * f[0][:, None, None] * (f[1][:, None] * f[2][None, :])[None]
    return out


def _velocity(rng, n, u_max):
    """Divergence-free face velocities (n + 1 along the normal, the last face
    the first): the discrete curl of an edge-sampled vector potential."""
    dx = [1.0 / s for s in n]
    px, py, pz = (_modes(rng, n, o) for o in ((0.5, 0.0, 0.0), (0.0, 0.5, 0.0), (0.0, 0.0, 0.5)))

    def diff(a, axis):
        return (torch.roll(a, -1, axis) - a) / dx[axis]

    u = [diff(pz, 1) - diff(py, 2), diff(px, 2) - diff(pz, 0), diff(py, 0) - diff(px, 1)]
    scale = u_max / max(float(a.abs().max()) for a in u)
    return [torch.cat([a, a.narrow(d, 0, 1)], dim=d).mul_(scale) for d, a in enumerate(u)]


def _smooth(rng, n):
    f = _modes(rng, n, (0.5, 0.5, 0.5), decay=1.0)
    lo, hi = float(f.min()), float(f.max())
    return (f - lo) / (hi - lo)


def _ghosted(phi, periodic, dim=3):
    """The field with two ghost cells a side, the periodic face ghosts filled."""
    n = list(phi.shape)
    og = [2 if d < dim else 0 for d in range(3)]
    out = torch.zeros([n[d] + 2 * og[d] for d in range(3)], dtype=torch.float64, device=phi.device)
    return _fill(out, phi, n, og, periodic)


def _fill(out, phi, n, og, periodic):
    """Internal cells and periodic face ghosts of a ghosted field."""
    inner = [slice(og[d], og[d] + n[d]) for d in range(3)]
    out[tuple(inner)] = phi
    for d in range(3):
        if og[d] and periodic[d]:
            lo, hi = list(inner), list(inner)
            lo[d], hi[d] = slice(0, 2), slice(2 + n[d], 4 + n[d])
            out[tuple(lo)] = phi.narrow(d, n[d] - 2, 2)
            out[tuple(hi)] = phi.narrow(d, 0, 2)
    return out


def _inputs(case, seed):
    """Everything a case's step needs, as torch tensors and numbers."""
    rng = np.random.default_rng(seed)
    path = case["path"]
    if path == "species":
        n = (case["n0"], case["n1"], 1)
        c = [(torch.arange(s, dtype=torch.float64, device=DEV) + 0.5) / s for s in n[:2]]
        comps = []
        for _ in range(2):      # a disk of each species, smooth background noise
            x0, y0, r0 = rng.uniform(0.35, 0.65), rng.uniform(0.35, 0.65), rng.uniform(0.15, 0.3)
            r = torch.sqrt((c[0][:, None] - x0) ** 2 + (c[1][None, :] - y0) ** 2)
            comps.append(((r < r0).to(torch.float64) + 0.05 * _smooth(rng, n)[:, :, 0])[:, :, None])
        vel = [tuple(float(v) for v in rng.uniform(-1.0, 1.0, size=2)) for _ in range(2)]
        w, e = (float(v) for v in rng.uniform(0.5, 1.0, size=2))
        # x: walls, Dirichlet on one end and zero gradient on the other, the
        # reverse for the second species; y periodic
        bcs = [{1: (1, w), 2: (2, 0.0)}, {1: (2, 0.0), 2: (1, e)}]
        return {"n": n, "dim": 2, "periodic": (0, 1, 0), "dt": 1e-3, "D": 1e-2, "vel": vel, "bcs": bcs,
                "phi": comps, "limiter": case["limiter"]}
    n = (case["n0"], case["n1"], case["n2"])
    nmax = max(n)
    if path == "heat":
        c = [(torch.arange(s, dtype=torch.float64, device=DEV) + 0.5) / s for s in n]
        x0 = rng.uniform(0.4, 0.6, size=3)
        r2 = sum(((c[d] - float(x0[d])) ** 2).reshape([-1 if q == d else 1 for q in range(3)]) for d in range(3))
        gen = torch.Generator(device=DEV).manual_seed(int(seed))
        phi = torch.exp(-r2 / (2.0 * 0.1 ** 2)) + 1e-3 * torch.randn(n, dtype=torch.float64, device=DEV, generator=gen)
        bc = {1: (1, 1.0), 2: (1, 0.0), 3: (2, 0.0), 4: (2, 0.0), 5: (2, 0.0), 6: (2, 0.0)}
        return {"n": n, "dim": 3, "periodic": (0, 0, 0), "dt": 1e-2, "D": 1e-3, "bcs": [bc], "phi": [phi]}
    # convection-diffusion: cell Peclet number 5, CFL 0.5 on the finest direction
    wall = case.get("wall", -1)
    periodic = tuple(0 if d == wall else 1 for d in range(3))
    out = {"n": n, "dim": 3, "periodic": periodic, "limiter": case.get("limiter", "VANLEER"), "bcs": [{}]}
    Dm = 1e-4
    if path == "refine":        # log-normal diffusivity under a 5-cell box filter
        gen = torch.Generator(device=DEV).manual_seed(int(seed))
        Dc = torch.randn(n, dtype=torch.float64, device=DEV, generator=gen).add_(math.log(1e-4)).exp_()
        for axis in range(3):
            acc = torch.zeros_like(Dc)
            for s in range(-2, 3):
                acc += torch.roll(Dc, s, axis)
            Dc = acc.mul_(0.2)
        out["cell_D"] = Dc
        Dm = float(Dc.reshape(-1)[:1 << 20].median())
    out["D"] = Dm
    u_max = 5.0 * Dm * nmax
    out["dt"] = 0.5 / (nmax * u_max)
    out["face_vel"] = _velocity(rng, n, u_max)
    out["phi"] = [_smooth(rng, n)]
    if wall >= 0:
        for d in range(3):      # no flow through the walls
            if d == wall:
                out["face_vel"][d].narrow(d, 0, 1).zero_()
                out["face_vel"][d].narrow(d, n[d], 1).zero_()
        out["bcs"] = [{2 * wall + 1: (1, float(rng.uniform(0.0, 1.0))), 2 * wall + 2: (2, 0.0)}]
    return out


def _boxes(case, seed):
    """Uneven boxes: D log-uniform, one Dirichlet face, zero gradient elsewhere."""
    rng = np.random.default_rng(seed)
    sides = [int(s) for s in case["sides"].split(",")]
    out = []
    for q in range(case["count"]):
        # the sides come round in turn, so that seeds differ in values and not in size
        n = [sides[(q + (q // len(sides)) * d) % len(sides)] if case["ragged"] else sides[q % len(sides)]
             for d in range(3)]
        bc = {f: (2, 0.0) for f in range(1, 7)}
        bc[int(rng.integers(1, 7))] = (1, float(rng.uniform(0.0, 1.0)))
        out.append({"n": tuple(n), "size": (1.0, 1.0, 1.0), "D": float(np.exp(rng.uniform(np.log(1e-5), np.log(1e-2)))),
                    "dt": 1e-2, "bc": bc})
    return out


NET_LAYERS = ((1, 16), (16, 32), (32, 64), (64, 64), (64, 64), (64, 32), (32, 16), (16, 1))   # enc0..3, dec3..0


def _net_weights(seed):
    """Weights of a network in use: unit-gain layers, a small last one."""
    rng = np.random.default_rng(seed)
    parts = []
    for q, (ci, co) in enumerate(NET_LAYERS):
        std = (0.3 if q == 7 else 1.0) / math.sqrt(27.0 * ci)
        parts.append(rng.normal(0.0, std, 27 * ci * co))
    return np.concatenate(parts).astype(np.float32)


def _net_vectors(case, seed, count, n):
    """Residual-like vectors and the errors that belong to them: smooth parts
    and noise of comparable size."""
    rng = np.random.default_rng(seed + 1)
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    r, e = [], []
    for _ in range(count):
        s = _modes(rng, n, (0.5, 0.5, 0.5), decay=1.0)
        s /= s.square().mean().sqrt()
        noise = torch.randn(n, dtype=torch.float64, device=DEV, generator=gen)
        r.append((s + 0.5 * noise).reshape(-1).float())
        e.append((0.8 * s + 0.5 * noise).reshape(-1).float())
    return torch.stack(r), torch.stack(e)


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
class _View:
    """A framework buffer as a torch tensor (zero copy).  The tensor keeps this
    object, and with it the handle that owns the buffer, alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f8", "data": (int(ptr), False),
                                         "version": 3, "strides": None}


def _view(owner, ptr, shape):
    return torch.as_tensor(_View(owner, ptr, shape), device=DEV)


def _solver(**kw):
    p = {"Convergence Tolerance": TOL, "Maximum Iterations": 5000, "tol_relative": 1}
    return D.BiCGStab2(p, **kw)


def prepare(case, seed):
    stream = torch.cuda.Stream()
    ctx = D.Context(0)
    ctx.set_stream(stream.cuda_stream)       # the program's own stream: torch and the framework share it
    st = {"case": case, "ctx": ctx, "stream": stream}
    path = case["path"]
    if path == "batch":
        boxes = _boxes(case, seed)
        bt = D.Batch(ctx, boxes)
        st["solver"] = _solver()
        bt.autotune(st["solver"])
        st["cells"] = [bt.num_cells(q) for q in range(len(boxes))]
        st["out"] = np.empty(sum(st["cells"]))
        st["batch"] = bt
        torch.cuda.synchronize()
        return st
    if path in ("apply", "grad"):
        n = (case["n0"], case["n1"], case["n2"])
        net = D.LearnedPreconditioner(ctx, n, coarse=bool(case.get("coarse", False)))
        net.set_weights(_net_weights(seed))
        st["net"] = net
        r, e = _net_vectors(case, seed, case.get("count", 1), n)
        st.update(r=r, e=e, z=torch.empty_like(r))
        torch.cuda.synchronize()
        return st
    inp = _inputs(case, seed)
    n, dim, periodic, N = inp["n"], inp["dim"], inp["periodic"], len(inp["phi"])
    grid = D.Grid(ctx, n[:dim], None, 2, periodic[:dim])
    field = D.Field(grid, 2, components=N)
    system = D.MatrixSystem(grid, components=N)
    for c, bc in enumerate(inp["bcs"]):
        for face, (kind, value) in bc.items():
            if N > 1:
                system.set_bc(face, kind, value, component=c)
            else:
                system.set_bc(face, kind, value)
    phi0 = torch.stack([_ghosted(p, periodic, dim) for p in inp["phi"]])
    levels = [_view(field, field.device_ptr(q), phi0.shape) for q in range(2)]
    for lev in levels:
        lev.copy_(phi0)
    st.update(grid=grid, field=field, system=system, phi0=phi0, levels=levels)
    if path == "species":
        st["terms"] = [D.Term("DDT", "SET", dt=inp["dt"])] + [
            D.Term("CONVECTION", "ADD", component=c, vel=inp["vel"][c], limiter=inp["limiter"]) for c in range(2)] + [
            D.Term("DIFFUSION", "SUB", D=inp["D"])]
        st["solver"] = _solver()
        torch.cuda.synchronize()
        return st
    kw = {"dt": inp["dt"]}
    if "face_vel" in inp:
        st["vel"] = [D.DeviceArray.from_tensor(t) for t in inp["face_vel"]]
        kw.update(face_vel=tuple(st["vel"]), limiter=inp["limiter"])
    if "cell_D" in inp:
        cell_D = inp["cell_D"].contiguous()
        st["face_D"] = [D.DeviceArray.from_tensor(torch.empty(grid.face_shape(d), dtype=torch.float64, device=DEV))
                        for d in range(3)]
        torch.cuda.synchronize()
        D.face_average(grid, cell_D.data_ptr(), st["face_D"])
        ctx.synchronize()
        kw.update(face_D=tuple(st["face_D"]))
    else:
        kw.update(D=inp["D"])
    st["asm"] = D.Assembly(**kw)
    st["solver"] = _solver(precision="FP32_REFINE" if path == "refine" else "FP64")
    # a time loop needs no true residual at each exit, as in the benchmark
    st["solver"].params.compute_true_residual = 0
    if path == "learned":
        st["net"] = D.LearnedPreconditioner(ctx, n, seed=seed, coarse=True)
        st["x"] = _view(system, system.device_ptr(8), (system.rows,))
    if path == "host":
        st["host"] = torch.empty(phi0.numel(), dtype=torch.float64, pin_memory=True)
        st["host"].copy_(phi0.reshape(-1))
    torch.cuda.synchronize()
    return st


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    path = case["path"]
    if path == "batch":
        bt = st["batch"]
        bt.zero_fields()
        for _ in range(case["steps"]):
            bt.solve(st["solver"])
        at = 0
        for q, m in enumerate(st["cells"]):
            st["out"][at:at + m] = bt.get_field(q)
            at += m
        return {"fields": st["out"]}
    if path == "apply":
        st["net"].apply(st["r"].data_ptr(), st["z"].data_ptr())
        return {"z": st["z"]}
    if path == "grad":
        loss, g = st["net"].loss_grad(st["r"].data_ptr(), st["e"].data_ptr(), case["count"])
        return {"loss": np.float32(loss), "grad": g}      # BF16 activations: not a 64-bit number
    if path == "learned":
        st["system"].build(st["field"], st["asm"])       # the initial guess is the field's
        st["net"].solve(st["system"], st["solver"])
        return {"x": st["x"]}
    if path == "host":          # the field goes on from where the last pass left it
        D.timesteps_host(st["system"], st["field"], st["asm"], st["solver"], case["steps"], st["host"].numpy())
        return {"field": st["host"]}
    system, field, solver = st["system"], st["field"], st["solver"]
    with torch.cuda.stream(st["stream"]):                # from the initial field again
        for lev in st["levels"]:
            lev.copy_(st["phi0"])
    for _ in range(case["steps"]):
        if path == "species":
            system.build(field, st["terms"])
            solver.solve(system)
            system.copy_to(field)
            field.exchange_halo()
            field.copy_to_old()
        else:
            D.timestep(system, field, st["asm"], solver)
    return {"field": st["levels"][0]}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def work(case):
    path = case["path"]
    if path == "batch":
        cells = sum(b["n"][0] * b["n"][1] * b["n"][2] for b in _boxes(case, 0))
        # every box is stepped on the device and read back once; at least two
        # iterations of four 7-point products and the vector updates a step
        return {"bytes": 8.0 * cells * (2 * case["steps"] + 1), "flops": 200.0 * cells * case["steps"]}
    if path == "species":
        cells = case["n0"] * case["n1"] * 2
        return {"bytes": 8.0 * cells * 3 * case["steps"], "flops": 200.0 * cells * case["steps"]}
    cells = float(case["n0"] * case["n1"] * case["n2"])
    if path in ("apply", "grad"):
        net = cells / 8 if case.get("coarse") else cells
        macs = sum(27 * ci * co * net / 8 ** lev for (ci, co), lev in zip(NET_LAYERS, (0, 1, 2, 3, 3, 2, 1, 0)))
        if path == "apply":
            return {"bytes": 8.0 * cells + 4.0 * sum(27 * ci * co for ci, co in NET_LAYERS), "flops": 2.0 * macs}
        # forward, data gradient and weight gradient of each pair
        return {"bytes": case["count"] * 8.0 * cells, "flops": 6.0 * macs * case["count"]}
    arrays = {"heat": 2, "tvd": 5, "host": 7, "refine": 8, "learned": 5}[path]
    steps = case.get("steps", 1)
    return {"bytes": 8.0 * cells * arrays * steps, "flops": 200.0 * cells * steps}


# ---------------------------------------------------------------------------
# exact: the same discretisation solved in 64 bits with plain torch
# ---------------------------------------------------------------------------
def _limiter(kind, r):
    r0 = torch.where(torch.isnan(r), torch.zeros_like(r), r)
    if kind == "UPWIND":
        return torch.zeros_like(r)
    if kind == "MINMOD":
        return r0.clamp(0.0, 1.0)
    if kind == "VANALBADA":
        return (r0 + r0 * r0) / (1.0 + r0 * r0)
    a = r0.abs()                # van Leer
    psi = (r0 + a) / (1.0 + a)
    return torch.where(torch.isinf(r0), torch.where(r0 > 0, 2.0, 0.0).to(r.dtype), psi)


def _rows(inp, ghost, bc, vel=None):
    """Coefficients and right-hand side of one implicit Euler step."""
    n, dim, periodic = inp["n"], inp["dim"], inp["periodic"]
    og = [2 if d < dim else 0 for d in range(3)]
    dx = [1.0 / n[d] for d in range(dim)]
    V = math.prod(dx)

    def cells(shift, d):
        return ghost[tuple(slice(og[q] + (shift if q == d else 0), og[q] + n[q] + (shift if q == d else 0))
                           for q in range(3))]

    phi = cells(0, 0)
    C = torch.full(n, V / inp["dt"], dtype=torch.float64, device=ghost.device)
    rhs = (V / inp["dt"]) * phi
    off = []
    for d in range(dim):
        A = V / dx[d]
        line = [cells(s, d) for s in range(-2, 3)]
        W, E = torch.zeros_like(C), torch.zeros_like(C)
        if vel is not None or "face_vel" in inp:
            if vel is not None:
                faces = [torch.full_like(C, vel[d])] * 2
            else:
                fv = inp["face_vel"][d]
                faces = [fv.narrow(d, 0, n[d]), fv.narrow(d, 1, n[d])]
            flux = []
            for side, v in enumerate(faces):    # upwind value and limited correction of each face
                up = v >= 0.0
                m2, m1, p0, p1, p2 = line
                UU = torch.where(up, m1, p2) if side else torch.where(up, m2, p1)
                U = torch.where(up, p0, p1) if side else torch.where(up, m1, p0)
                Dn = torch.where(up, p1, p0) if side else torch.where(up, p0, m1)
                psi = _limiter(inp["limiter"], (U - UU) / (Dn - U))
                flux.append(-0.5 * psi * (Dn - U) * v)
            lo, hi = faces
            W -= A * lo.clamp(min=0.0)
            E += A * hi.clamp(max=0.0)
            C += A * (hi.clamp(min=0.0) - lo.clamp(max=0.0))
            rhs = rhs + A * (flux[1] - flux[0])
        if "cell_D" in inp:
            Dl = 0.5 * (inp["cell_D"] + torch.roll(inp["cell_D"], 1, d))
            Dh = torch.roll(Dl, -1, d)
        else:
            Dl = Dh = inp["D"]
        W = W - A / dx[d] * Dl
        E = E - A / dx[d] * Dh
        C = C + A / dx[d] * (Dl + Dh)
        if not periodic[d]:
            for face, X, at in ((2 * d + 1, W, 0), (2 * d + 2, E, n[d] - 1)):
                kind, value = bc[face]
                x = X.narrow(d, at, 1)
                if kind == 1:
                    C.narrow(d, at, 1).sub_(x)
                    rhs.narrow(d, at, 1).sub_(2.0 * value * x)
                else:
                    C.narrow(d, at, 1).add_(x)
                x.zero_()
        off.append((W, E))
    return C, off, rhs


def _solve(C, off, rhs, x):
    """Jacobi-preconditioned BiCGStab to the limit of 64 bits."""

    def A(z):
        y = C * z
        for d, (W, E) in enumerate(off):
            y += W * torch.roll(z, 1, d)
            y += E * torch.roll(z, -1, d)
        return y

    def dot(a, b):
        return float((a * b).sum())

    target = 2e-15 * math.sqrt(dot(rhs, rhs))
    best = math.inf
    for _ in range(4):          # restarted from the true residual
        r = rhs - A(x)
        now = math.sqrt(dot(r, r))
        if now <= target or now > 0.5 * best:
            break
        best = now
        rh, p = r.clone(), r.clone()
        rho = dot(rh, r)
        for _ in range(400):
            ph = p / C
            v = A(ph)
            alpha = rho / dot(rh, v)
            s = r - alpha * v
            sh = s / C
            t = A(sh)
            tt = dot(t, t)
            omega = dot(t, s) / tt if tt > 0.0 else 0.0
            x = x + alpha * ph + omega * sh
            r = s - omega * t
            if math.sqrt(dot(r, r)) <= 0.2 * target or omega == 0.0:
                break
            old, rho = rho, dot(rh, r)
            p = r + (rho / old) * (alpha / omega) * (p - omega * v)
    return x


def _exact_boxes(case, seed):
    """Separable boxes: each step solved through the eigenvectors of its three
    one-dimensional operators."""
    out = []
    for box in _boxes(case, seed):
        n, Dc, dt = box["n"], box["D"], box["dt"]
        dx = [box["size"][d] / n[d] for d in range(3)]
        V = math.prod(dx)
        lam, Q, src = [], [], np.zeros(n)
        for d in range(3):
            a = V / dx[d] / dx[d] * Dc
            T = np.diag(np.full(n[d], 2 * a)) - a * (np.eye(n[d], k=1) + np.eye(n[d], k=-1))
            for face, at in ((2 * d + 1, 0), (2 * d + 2, n[d] - 1)):
                kind, value = box["bc"][face]
                T[at, at] += a if kind == 1 else -a
                if kind == 1:
                    where = [slice(None)] * 3
                    where[d] = at
                    src[tuple(where)] += 2.0 * value * a
            w, q = np.linalg.eigh(T)
            lam.append(w)
            Q.append(q)
        tt = V / dt
        den = tt + lam[0][:, None, None] + lam[1][None, :, None] + lam[2][None, None, :]
        fwd = np.einsum("ia,ijk->ajk", Q[0], src)
        fwd = np.einsum("jb,ajk->abk", Q[1], fwd)
        fwd = np.einsum("kc,abk->abc", Q[2], fwd)
        c = np.zeros(n)
        for _ in range(case["steps"]):
            c = (tt * c + fwd) / den
        c = np.einsum("ia,abc->ibc", Q[0], c)
        c = np.einsum("jb,ibc->ijc", Q[1], c)
        out.append(np.einsum("kc,ijc->ijk", Q[2], c).reshape(-1))
    return np.concatenate(out)


def _network(w, u):
    """N(u) = u + U(u) on a batch of volumes, in 64 bits."""
    F = torch.nn.functional
    conv, at = [], 0
    for ci, co in NET_LAYERS:
        # stored as [tap][out][in], the taps over (i, j, k)
        conv.append(w[at:at + 27 * ci * co].reshape(3, 3, 3, co, ci).permute(3, 4, 0, 1, 2))
        at += 27 * ci * co

    def c(q, x):
        return F.conv3d(x, conv[q], padding=1)

    def up(x):
        return x.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)

    e0 = c(0, u)
    e1 = c(1, F.avg_pool3d(e0, 2))
    e2 = c(2, F.avg_pool3d(e1, 2))
    e3 = c(3, F.avg_pool3d(e2, 2))
    s2 = e2 + up(c(4, e3))
    s1 = e1 + up(c(5, s2))
    s0 = e0 + up(c(6, s1))
    return u + c(7, s0)


def exact(case, seed):
    path = case["path"]
    if path == "batch":
        return {"fields": _exact_boxes(case, seed)}
    if path in ("apply", "grad"):
        n = (case["n0"], case["n1"], case["n2"])
        w = torch.from_numpy(_net_weights(seed)).to(DEV).double()
        r, e = _net_vectors(case, seed, case.get("count", 1), n)
        u = r.double().reshape(-1, 1, *n)
        if path == "apply":
            with torch.no_grad():
                if case["coarse"]:
                    v = torch.nn.functional.avg_pool3d(u, 2)
                    c = _network(w, v) - v
                    z = u + c.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4)
                else:
                    z = _network(w, u)
            return {"z": z.reshape(1, -1)}
        w.requires_grad_(True)
        e = e.double().reshape(-1, 1, *n)
        err = (_network(w, u) - e).square().sum(dim=(1, 2, 3, 4)) / e.square().sum(dim=(1, 2, 3, 4))
        loss = err.mean()
        loss.backward()
        return {"loss": np.float32(loss.item()), "grad": w.grad.cpu().numpy()}
    inp = _inputs(case, seed)
    n, dim, periodic = inp["n"], inp["dim"], inp["periodic"]
    og = [2 if d < dim else 0 for d in range(3)]
    ghosts = [_ghosted(p, periodic, dim) for p in inp["phi"]]
    x = None
    for _ in range(case.get("steps", 1)):
        for c, ghost in enumerate(ghosts):
            C, off, rhs = _rows(inp, ghost, inp["bcs"][c], inp["vel"][c] if path == "species" else None)
            x = ghost[tuple(slice(og[d], og[d] + n[d]) for d in range(3))].clone()
            x = _solve(C, off, rhs, x)
            _fill(ghost, x, n, og, periodic)
    if path == "learned":
        return {"x": x.reshape(-1)}
    out = torch.stack(ghosts)
    return {"field": out.cpu().reshape(-1) if path == "host" else out}
