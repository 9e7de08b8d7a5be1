"""The pressure steps whose time is measured: what a user of this library runs, through its public entry points.

``listed()`` holds the fixed cases and ``draw()`` makes more of the same kinds and ranges. The grids, scenes and
tolerances are those of the repository's workloads, tests and benchmark, or generic ones: 1e-8 relative residual on the
benchmark's own workloads, 1e-12 (3D) and 1e-10 (2D) where a step is solved as tightly as NEREUS solves by default.
Fields are N(0, 1) face velocities that vanish on solid faces, as everywhere in this repository.

Kinds:
  step     one Chorin or incremental pressure step of one grid whose fields live on the device
           (nereus_b200_project_device / _device_ex), the grid's layout set once
  host     the same step through PressureSolver.SolvePressure on the caller's numpy arrays
  tanks    one batched step of several free-surface tanks (serving.Batch)
  server   a burst of requests of different shapes through serving.Server
  flip     two consecutive FLIP steps: labels from particles, the new layout, the pressure step
  relabel  FLIP's re-labelling alone
  bc       EnforceVelocityBC and EnforcePressureBC replayed on device fields
"""
import ctypes
import math
import random

import numpy as np
import torch

from nereus_cfd_b200 import capi, serving, workloads
from nereus_cfd_b200.boundary import BoundaryReplay
from nereus_cfd_b200.pressure import MACGrid, PressureSolver

FLUID, SOLID, EMPTY, INFLOW = 0, 1, 2, 3
DEV = "cuda"


def listed():
    return [
        # the smallest step in use: the 2D closed box, bound by launches and their latency
        {"name": "box2d_128", "kind": "step", "dim": 2, "scene": "box", "nx": 128, "ny": 128, "nz": 1,
         "precision": "mixed", "scheme": 0, "tol": 1e-10},
        # a lid-driven cavity's step in the incremental scheme (singular, the previous pressure carried along)
        {"name": "cavity_64_incremental", "kind": "step", "dim": 3, "scene": "box", "nx": 64, "ny": 64, "nz": 64,
         "precision": "mixed", "scheme": 1, "tol": 1e-12},
        # an ordinary grid whose sides are odd and unequal, solved as tightly as NEREUS does by default
        {"name": "sphere_odd_125", "kind": "step", "dim": 3, "scene": "sphere", "nx": 125, "ny": 101, "nz": 117,
         "precision": "mixed", "scheme": 0, "tol": 1e-12},
        # the benchmark's headline step, and the same step in plain FP64 (the largest case)
        {"name": "sphere_256", "kind": "step", "dim": 3, "scene": "sphere", "nx": 256, "ny": 256, "nz": 256,
         "precision": "mixed", "scheme": 0, "tol": 1e-8},
        {"name": "sphere_256_fp64", "kind": "step", "dim": 3, "scene": "sphere", "nx": 256, "ny": 256, "nz": 256,
         "precision": "fp64", "scheme": 0, "tol": 1e-8},
        # the stretched channel past a cylinder, in the precision that reaches 1e-6 in its pressure
        {"name": "cylinder_fp64", "kind": "step", "dim": 3, "scene": "cylinder", "nx": 192, "ny": 128, "nz": 128,
         "precision": "fp64", "scheme": 0, "tol": 1e-8},
        # a NEREUS build's own call: host arrays in, host arrays out
        {"name": "host_64", "kind": "host", "dim": 3, "scene": "sphere", "nx": 64, "ny": 64, "nz": 64,
         "precision": "mixed", "scheme": 0, "tol": 1e-12},
        # a batch of free-surface tanks advanced by one call per step
        {"name": "tanks_16x128", "kind": "tanks", "n": 128, "count": 16, "tol": 1e-8},
        # requests of changing shape, dimension and mask through the server
        {"name": "server_16", "kind": "server", "count": 16, "mix": 5, "tol": 1e-8},
        # FLIP: the labels move with the particles, so every step has a new layout
        {"name": "flip_128", "kind": "flip", "n": 128, "ppc": 8, "tol": 1e-12},
        # FLIP's re-labelling from 30 M particles, the reference's seeding density
        {"name": "relabel_256", "kind": "relabel", "n": 256, "ppc": 8, "stride": 3},
        # the boundary replay of a channel with an inlet, an outlet and a solid sphere
        {"name": "bc_256", "kind": "bc", "n": 256},
    ]


def draw(rng: random.Random):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step2d", "step3d", "step3d", "step3d", "cylinder", "host", "tanks", "server", "flip",
                       "relabel", "bc"])
    if kind == "step2d":
        nx = size(33, 500)
        return {"kind": "step", "dim": 2, "scene": rng.choice(["box", "sphere"]), "nx": nx,
                "ny": max(33, int(nx * rng.uniform(0.5, 1.0))), "nz": 1, "precision": rng.choice(["mixed", "fp64"]),
                "scheme": 0, "tol": 1e-10}
    if kind == "step3d":
        n = size(25, 200)
        n3 = [max(24, int(n * rng.uniform(0.7, 1.0))) for _ in range(3)]
        if rng.random() < 0.5:
            n3[2] += n3[2] % 2
        return {"kind": "step", "dim": 3, "scene": rng.choice(["box", "sphere"]), "nx": n3[0], "ny": n3[1],
                "nz": n3[2], "precision": rng.choice(["mixed", "fp64"]), "scheme": rng.choice([0, 0, 1]),
                "tol": 1e-12}
    if kind == "cylinder":
        return {"kind": "step", "dim": 3, "scene": "cylinder", "nx": 2 * size(32, 96), "ny": size(40, 128),
                "nz": size(40, 128), "precision": "fp64", "scheme": 0, "tol": 1e-8}
    if kind == "host":
        return {"kind": "host", "dim": 3, "scene": rng.choice(["box", "sphere"]), "nx": size(24, 96),
                "ny": size(24, 96), "nz": size(24, 96), "precision": "mixed", "scheme": 0, "tol": 1e-12}
    if kind == "tanks":
        return {"kind": "tanks", "n": 16 * rng.randint(2, 8), "count": rng.randint(2, 16), "tol": 1e-8}
    if kind == "server":
        return {"kind": "server", "count": rng.randint(8, 16), "mix": rng.randint(10, 10000), "tol": 1e-8}
    if kind == "flip":
        return {"kind": "flip", "n": size(32, 128), "ppc": rng.choice([4, 8]), "tol": 1e-12}
    if kind == "relabel":
        return {"kind": "relabel", "n": size(48, 256), "ppc": rng.choice([4, 8]), "stride": rng.choice([3, 7])}
    return {"kind": "bc", "n": size(32, 256)}


# ------------------------------------------------------------------------------------------------------------------
# inputs: geometry on the host as plain arrays, fields on the device from the seed
# ------------------------------------------------------------------------------------------------------------------
def interior_widths(c):
    """Interior cell widths along x, y, z."""
    if c["scene"] == "cylinder":
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        band = max(2, (24 * nx) // 192 // 2 * 2)
        wx = workloads.band_stretched_widths(nx, 2.2, band, 0.5, 1.04)
        return [wx, np.full(ny, 0.41 / ny), np.full(nz, 0.41 / nz)]
    dh = 1.0 / min(c["nx"], c["ny"])
    return [np.full(c["nx"], dh), np.full(c["ny"], dh), np.full(c["nz"], dh)]


def make_grid(c):
    w = interior_widths(c)
    if c["scene"] == "cylinder":
        return workloads.stretched_grid(3, (0.0, 2.2, 0.0, 0.41, 0.0, 0.41), w)
    dh = float(w[0][0])
    ax = [workloads.uniform_axis(0.0, n, dh) for n in (c["nx"], c["ny"])]
    if c["dim"] == 3:
        ax.append(workloads.uniform_axis(0.0, c["nz"], dh))
    else:
        ax.append(workloads.Axis(np.array([dh]), np.array([0.0, dh]), np.array([dh / 2.0])))
    return workloads.Grid(c["dim"], ax, dh, False, (0.0, c["nx"] * dh, 0.0, c["ny"] * dh, 0.0, c["nz"] * dh))


def cell_types(c, a=0.5, b=0.5, dev=DEV):
    """Cell types (Ny, Nx, Nz), ring included: no-slip walls; 'sphere': a solid ball and a p = 0 outlet at x = xmax;
    'cylinder': a solid cylinder along z, an inlet at x = 0 and that outlet; 'tank': liquid where x < a and z < b under
    air; 'inlet': 'sphere' with an inlet at x = 0."""
    w = interior_widths(c)
    xc, yc, zc = [torch.from_numpy(np.cumsum(v) - 0.5 * v).to(dev) for v in w]
    X, Y, Z = xc[None, :, None], yc[:, None, None], zc[None, None, :]
    dim, nx, ny, nz = c["dim"], c["nx"], c["ny"], c["nz"]
    L = [float(v.sum()) for v in w]
    inner = torch.zeros((ny, nx, nz), dtype=torch.uint8, device=dev)
    if c["scene"] in ("sphere", "inlet"):
        d2 = (X - 0.5 * L[0]) ** 2 + (Y - 0.5 * L[1]) ** 2
        d2 = d2 + (Z - 0.5 * L[2]) ** 2 if dim == 3 else d2
        inner[(d2 < (0.15 * min(L[:dim])) ** 2).expand_as(inner)] = SOLID
    elif c["scene"] == "cylinder":
        inner[((X - 0.5) ** 2 + (Y - 0.2) ** 2 < 0.05 ** 2).expand_as(inner)] = SOLID
    elif c["scene"] == "tank":
        inner[~((X < a) & (Z < b)).expand_as(inner)] = EMPTY
    t = torch.full((ny + 2, nx + 2, nz + 2 if dim == 3 else 1), SOLID, dtype=torch.uint8, device=dev)
    if dim == 3:
        t[1:-1, 1:-1, 1:-1] = inner
    else:
        t[1:-1, 1:-1, :] = inner
    if c["scene"] in ("cylinder", "inlet"):
        t[:, 0, :] = INFLOW
    if c["scene"] in ("sphere", "cylinder", "inlet"):
        t[:, -1, :] = EMPTY
    return t


def field_shapes(c):
    Ny, Nx, Nz = c["ny"] + 2, c["nx"] + 2, c["nz"] + 2 if c["dim"] == 3 else 1
    w = (Ny, Nx, Nz + 1) if c["dim"] == 3 else (1,)
    return [(Ny, Nx + 1, Nz), (Ny + 1, Nx, Nz), w, (Ny, Nx, Nz)]


def split_fields(flat, shapes):
    """u, v, w, p as views of one flat array."""
    out, at = [], 0
    for s in shapes:
        n = int(np.prod(s))
        out.append(flat[at:at + n].view(s))
        at += n + (-n) % 32
    return out


def flat_size(shapes):
    return sum(int(np.prod(s)) + (-int(np.prod(s))) % 32 for s in shapes)


def open_faces(t, ax):
    """Faces along array axis ax with no SOLID cell and not the grid's end on either side."""
    pad = torch.full_like(t.narrow(ax, 0, 1), SOLID)
    e = torch.cat([pad, t, pad], ax)
    n = e.shape[ax]
    return (e.narrow(ax, 0, n - 1) != SOLID) & (e.narrow(ax, 1, n - 1) != SOLID)


def fill_velocities(c, t, fields, gen, fp32=False):
    """N(0, 1) on the faces that touch no solid (in a tank: and touch liquid)."""
    for q, ax in enumerate((1, 0, 2)[:c["dim"]]):
        f = fields[q]
        f.normal_(generator=gen)
        if fp32:
            f.copy_(f.float())
        keep = open_faces(t, ax)
        if c["scene"] == "tank":
            pad = torch.full_like(t.narrow(ax, 0, 1), SOLID)
            e = torch.cat([pad, t, pad], ax)
            n = e.shape[ax]
            keep &= (e.narrow(ax, 0, n - 1) == FLUID) | (e.narrow(ax, 1, n - 1) == FLUID)
        f.mul_(keep)


def previous_pressure(c, t, gen):
    """A smooth p^n with a little noise on the unknowns, zero elsewhere (no face prescribes a pressure)."""
    sh = t.shape
    y, x, z = [torch.linspace(0.0, 1.0, n, device=t.device, dtype=torch.float64) for n in sh]
    p = torch.cos(3.0 * x)[None, :, None] * torch.cos(2.0 * y)[:, None, None] + 0.5 * torch.cos(5.0 * z)[None, None, :]
    p = p + 0.05 * torch.randn(sh, generator=gen, device=t.device, dtype=torch.float64)
    return torch.where(unknowns(c, t), p, torch.zeros_like(p)).contiguous()


def unknowns(c, t):
    m = torch.zeros_like(t, dtype=torch.bool)
    s = (slice(1, -1), slice(1, -1), slice(1, -1) if c["dim"] == 3 else slice(None))
    m[s] = t[s] == FLUID
    return m


def generator(seed, dev=DEV):
    g = torch.Generator(device=dev)
    g.manual_seed(1000003 * seed + 17)
    return g


RHO, DT = 1.0, 1e-3


def step_inputs(c, seed, t=None):
    """types, the flat array of u, v, w, p before the step, and p^n (incremental scheme)."""
    gen = generator(seed)
    if t is None:
        t = cell_types(c, c.get("a", 0.5), c.get("b", 0.5))
    shapes = field_shapes(c)
    base = torch.zeros(flat_size(shapes), dtype=torch.float64, device=DEV)
    fill_velocities(c, t, split_fields(base, shapes), gen, fp32=c["scene"] == "tank")
    prev = previous_pressure(c, t, gen) if c.get("scheme") else None
    return t, base, prev


# ------------------------------------------------------------------------------------------------------------------
# the kinds
# ------------------------------------------------------------------------------------------------------------------
def mac_grid(c, g, t):
    types = t.cpu().numpy().reshape(-1)
    none = np.zeros(1)
    return MACGrid(g, types, none, none, none, none, RHO, DT)


def new_solver(c, g, t, stream):
    s = PressureSolver(c["precision"], device=torch.cuda.current_device(), stream=stream.cuda_stream)
    s.InitializePressureSolver(mac_grid(c, g, t))
    return s


def device_step(s, c, fields, prev, compat):
    r = capi.Result()
    ptr = [ctypes.c_void_p(f.data_ptr()) for f in fields]
    if prev is None:
        st = s.lib.nereus_b200_project_device(s.ctx, *ptr, RHO, DT, compat, c["tol"], ctypes.byref(r))
    else:
        st = s.lib.nereus_b200_project_device_ex(s.ctx, *ptr, ctypes.c_void_p(prev.data_ptr()), RHO, DT,
                                                 c["scheme"], compat, 0, c["tol"], ctypes.byref(r))
    capi.check(st)


def prepare_step(c, seed):
    t, base, prev = step_inputs(c, seed)
    stream = torch.cuda.Stream()
    s = new_solver(c, make_grid(c), t, stream)
    work = base.clone()
    torch.cuda.synchronize()
    return {"case": c, "solver": s, "stream": stream, "base": base, "flat": work, "prev": prev,
            "fields": split_fields(work, field_shapes(c)), "compat": int(c["scene"] == "box")}


def run_step(s):
    st = s["stream"]
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        s["flat"].copy_(s["base"])  # this step's intermediate velocities
        device_step(s["solver"], s["case"], s["fields"], s["prev"], s["compat"])
    return s["fields"]


def prepare_host(c, seed):
    t, base, _ = step_inputs(c, seed)
    g = make_grid(c)
    host = base.cpu()
    work = host.clone()
    u, v, w, p = split_fields(work, field_shapes(c))
    m = MACGrid(g, t.cpu().numpy().reshape(-1), u.numpy().reshape(-1), v.numpy().reshape(-1), w.numpy().reshape(-1),
                p.numpy().reshape(-1), RHO, DT)
    s = PressureSolver(c["precision"], device=torch.cuda.current_device())
    s.InitializePressureSolver(m)
    return {"case": c, "solver": s, "grid": m, "base": host, "flat": work, "compat": c["scene"] == "box"}


def run_host(s):
    s["flat"].copy_(s["base"])
    m = s["grid"]
    s["solver"].SolvePressure(m, tol=s["case"]["tol"], needs_compat=s["compat"])
    return [m.u, m.v, m.w, m.p]


def tank_cases(c, seed):
    r = random.Random(7919 * seed + c["n"] + c["count"])
    return [dict(dim=3, scene="tank", nx=c["n"], ny=c["n"], nz=c["n"], a=r.uniform(0.3, 0.7), b=r.uniform(0.3, 0.7),
                 precision="mixed", tol=c["tol"]) for _ in range(c["count"])]


def prepare_tanks(c, seed):
    cases = tank_cases(c, seed)
    shapes = field_shapes(cases[0])
    n = flat_size(shapes)
    base = torch.empty(len(cases) * n, dtype=torch.float64, device=DEV)
    work = torch.empty_like(base)
    stream = torch.cuda.Stream()
    batch = serving.Batch(len(cases), device=torch.cuda.current_device(), stream=stream.cuda_stream)
    g = make_grid(cases[0])
    jobs = []
    for q, k in enumerate(cases):
        t, f, _ = step_inputs(k, 1000 * seed + q)
        base[q * n:(q + 1) * n] = f
        m = mac_grid(k, g, t)
        batch.set_layout(q, m)
        fields = split_fields(work[q * n:(q + 1) * n], shapes)
        jobs.append(serving.Job(m, tol=c["tol"], device_fields=dict(zip("uvwp", fields))))
    torch.cuda.synchronize()
    return {"batch": batch, "jobs": jobs, "items": batch.items(jobs), "stream": stream, "base": base, "flat": work}


def run_tanks(s):
    st = s["stream"]
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        s["flat"].copy_(s["base"])
        s["batch"].project(s["jobs"], items=s["items"], allow=(capi.NB_OK,))
    return [j.device_fields[k] for j in s["jobs"] for k in "uvwp"]


def request_cases(c):
    """The shapes of a burst: mostly 3D, sides over a range, the three masks, a few 2D ones."""
    r = random.Random(c["mix"])
    out = []
    for _ in range(c["count"]):
        three = r.random() < 0.7
        n = int(math.exp(r.uniform(math.log(32), math.log(96)))) if three else \
            int(math.exp(r.uniform(math.log(64), math.log(400))))
        scene = r.choice(["box", "sphere", "tank"] if three else ["box", "sphere"])
        out.append(dict(dim=3 if three else 2, scene=scene, nx=n, ny=n, nz=n if three else 1, a=r.uniform(0.3, 0.7),
                        b=r.uniform(0.3, 0.7), precision="mixed", tol=c["tol"]))
    return out


def prepare_server(c, seed):
    cases = request_cases(c)
    sizes = [flat_size(field_shapes(k)) for k in cases]
    base = torch.empty(sum(sizes), dtype=torch.float64, device=DEV)
    work = torch.empty_like(base)
    jobs, at = [], 0
    for q, k in enumerate(cases):
        t, f, _ = step_inputs(k, 1000 * seed + q)
        base[at:at + sizes[q]] = f
        fields = split_fields(work[at:at + sizes[q]], field_shapes(k))
        at += sizes[q]
        jobs.append(serving.Job(mac_grid(k, make_grid(k), t), tol=c["tol"], needs_compat=k["scene"] == "box",
                                device_fields=dict(zip("uvwp", fields))))
    srv = serving.Server(devices=(torch.cuda.current_device(),), slots_per_device=4)
    torch.cuda.synchronize()
    return {"server": srv, "jobs": jobs, "base": base, "flat": work}


def run_server(s):
    s["flat"].copy_(s["base"])
    torch.cuda.current_stream().synchronize()  # the fields' writers finish before the submissions
    tickets = [s["server"].submit(j) for j in s["jobs"]]
    for q in tickets:
        capi.check(s["server"].wait(q))
    return [j.device_fields[k] for j in s["jobs"] for k in "uvwp"]


def particles(n, ppc, seed, step, stride=3):
    """ppc particles in every liquid cell of an n^3 tank but 3% of the cells, cell by cell, as rows of `stride`
    doubles (7: the reference's Particle, x at the second). The surface is a wave that moves with ``step``."""
    gen = generator(seed + 7 * step)
    dh = 1.0 / n
    xc = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) * dh
    top = 0.5 + 0.08 * torch.sin(2.0 * math.pi * (xc + 0.05 * step + 0.01 * (seed % 10)))
    liquid = (xc[None, None, :] < top[None, :, None]).expand(n, n, n)  # (y, x, z)
    cells = torch.nonzero(liquid)
    keep = torch.rand(cells.shape[0], device=DEV, generator=gen, dtype=torch.float64) >= 0.03
    cells = cells[keep].repeat_interleave(ppc, dim=0)
    rows = torch.rand(cells.shape[0], stride, device=DEV, generator=gen, dtype=torch.float64)
    at = 1 if stride == 7 else 0
    for q, ax in enumerate((1, 0, 2)):  # x from column j, y from row i, z from k
        rows[:, at + q] = (rows[:, at + q] + cells[:, ax]) * dh
    return rows


def relabel_state(n, rows):
    lib = capi.load()
    N = n + 2
    c = dict(dim=3, scene="tank", nx=n, ny=n, nz=n)
    return {"lib": lib, "N": N, "dh": 1.0 / n, "rows": rows, "types": cell_types(c, 2.0, 0.5).reshape(-1),
            "scratch": torch.zeros(lib.nereus_b200_update_fluid_cells_scratch_bytes(3, N, N, N) // 4 + 1,
                                   dtype=torch.int32, device=DEV),
            "skipped": torch.zeros(1, dtype=torch.int64, device=DEV)}


def relabel(s, rows, stream):
    n, stride = rows.shape
    at = rows.data_ptr() + (8 if stride == 7 else 0)
    N, dh = s["N"], s["dh"]
    capi.check(s["lib"].nereus_b200_update_fluid_cells_device(
        torch.cuda.current_device(), 3, N, N, N, -dh, -dh, -dh, dh, ctypes.c_void_p(at), ctypes.c_void_p(at + 8),
        ctypes.c_void_p(at + 16), n, stride, ctypes.c_void_p(s["types"].data_ptr()),
        ctypes.c_void_p(s["scratch"].data_ptr()), 4 * s["scratch"].numel(), ctypes.c_void_p(s["skipped"].data_ptr()),
        ctypes.c_void_p(stream.cuda_stream)))


def prepare_relabel(c, seed):
    s = relabel_state(c["n"], particles(c["n"], c["ppc"], seed, 0, c["stride"]))
    torch.cuda.synchronize()
    return s


def run_relabel(s):
    relabel(s, s["rows"], torch.cuda.current_stream())
    return [s["types"], s["skipped"]]


def flip_case(c):
    return dict(dim=3, scene="tank", nx=c["n"], ny=c["n"], nz=c["n"], precision="mixed", tol=c["tol"])


def labels_of(rows, n):
    """The labels of a tank's particles in plain torch: the cells that hold one, then the in-place pass (a cell with
    five liquid neighbours fills, the lower neighbours counting as the pass left them)."""
    N = n + 2
    inner = slice(1, -1)
    fixed = torch.full((N, N, N), SOLID, dtype=torch.uint8, device=rows.device)
    fixed[inner, inner, inner] = EMPTY
    idx = (rows[:, :3] * n).floor().long() + 1
    mark = torch.zeros((N, N, N), dtype=torch.int32, device=rows.device)
    mark[idx[:, 1], idx[:, 0], idx[:, 2]] = 1
    mark[fixed == SOLID] = 0
    last = mark
    while True:
        up = sum(torch.roll(mark, -1, ax) for ax in range(3))
        low = sum(torch.roll(last, 1, ax) for ax in range(3))
        new = torch.where((fixed == EMPTY) & ((mark > 0) | (up + low >= 5)), 1, 0).to(torch.int32)
        if torch.equal(new, last):
            break
        last = new
    fixed[last > 0] = FLUID
    return fixed


def flip_fields(c, seed, step, t):
    return step_inputs(flip_case(c), 100 * seed + step, t)[1]


def prepare_flip(c, seed):
    k = flip_case(c)
    rows = [particles(c["n"], c["ppc"], seed, step) for step in range(2)]
    bases = [flip_fields(c, seed, step, labels_of(rows[step], c["n"])) for step in range(2)]
    s = relabel_state(c["n"], None)
    s["clouds"], s["bases"], s["case"] = rows, bases, k
    s["flats"] = [b.clone() for b in bases]
    s["fields"] = [split_fields(f, field_shapes(k)) for f in s["flats"]]
    s["labels"] = [torch.empty_like(s["types"]) for _ in range(2)]
    s["host"] = torch.empty(s["types"].numel(), dtype=torch.uint8, pin_memory=True)
    s["stream"] = torch.cuda.Stream()
    g = make_grid(k)
    s["solver"] = new_solver(k, g, s["types"], s["stream"])
    none = np.zeros(1)
    s["grid"] = MACGrid(g, s["host"].numpy(), none, none, none, none, RHO, DT)
    torch.cuda.synchronize()
    return s


def run_flip(s):
    st = s["stream"]
    st.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(st):
        for step in range(2):
            relabel(s, s["clouds"][step], st)
            s["labels"][step].copy_(s["types"])
            s["host"].copy_(s["types"], non_blocking=True)
            s["flats"][step].copy_(s["bases"][step])
            st.synchronize()  # the new labels are on the host
            s["solver"].EnsureSystem(s["grid"])
            device_step(s["solver"], s["case"], s["fields"][step], None, 0)
    return s["labels"] + [f for q in s["fields"] for f in q]


def boundary_lists(c):
    """A channel's boundary lists: solid faces, prescribed inlet faces, the outlet's copies, and the pressure ring
    (y, x, then z faces)."""
    t = cell_types(c, dev="cpu")
    Ny, Nx, Nz = t.shape
    i32 = lambda x: np.ascontiguousarray(x, dtype=np.int32).reshape(-1)
    shapes = field_shapes(c)
    idx = [np.arange(int(np.prod(s)), dtype=np.int64).reshape(s) for s in shapes]
    out = {}
    for q, ax in enumerate((1, 0, 2)):
        out["solid%d" % q] = i32(idx[q].reshape(-1)[~open_faces(t, ax).numpy().reshape(-1)])
    inlet = [idx[0][1:-1, :2, 1:-1], idx[1][1:-1, 0, 1:-1], idx[2][1:-1, 0, 1:-1]]
    out["presc_comp"] = i32(np.concatenate([np.full(v.size, q) for q, v in enumerate(inlet)]))
    out["presc_index"] = i32(np.concatenate([v.reshape(-1) for v in inlet]))
    dst = [idx[0][1:-1, Nx, 1:-1], idx[1][1:-1, Nx - 1, 1:-1], idx[2][1:-1, Nx - 1, 1:-1]]
    src = [idx[0][1:-1, Nx - 1, 1:-1], idx[1][1:-1, Nx - 2, 1:-1], idx[2][1:-1, Nx - 2, 1:-1]]
    out["copy_comp"] = i32(np.concatenate([np.full(v.size, q) for q, v in enumerate(dst)]))
    out["copy_dst"] = i32(np.concatenate([v.reshape(-1) for v in dst]))
    out["copy_src"] = i32(np.concatenate([v.reshape(-1) for v in src]))
    cell = idx[3]
    rd, rs = [], []
    for ax in (0, 1, 2):
        for lo, inn in ((0, 1), (cell.shape[ax] - 1, cell.shape[ax] - 2)):
            rd.append(cell.take(lo, axis=ax).reshape(-1))
            rs.append(cell.take(inn, axis=ax).reshape(-1))
    rd, rs = np.concatenate(rd), np.concatenate(rs)
    out["ring_dst"], out["ring_src"] = i32(rd), i32(rs)
    out["ring_kind"] = i32(np.where(t.numpy().reshape(-1)[rd] == EMPTY, 0, 2))
    for k in ("inlet_comp", "inlet_index", "inlet_area", "inlet_sign", "outflow_comp", "outflow_index",
              "outflow_outer", "outflow_area", "outflow_sign"):
        out[k] = np.zeros(0)
    return out


def bc_case(c):
    return dict(dim=3, scene="inlet", nx=c["n"], ny=c["n"], nz=c["n"])


def prepare_bc(c, seed):
    k = bc_case(c)
    lists = boundary_lists(k)
    N = c["n"] + 2
    gen = generator(seed)
    shapes = field_shapes(k)
    flat = torch.randn(flat_size(shapes), generator=gen, dtype=torch.float64, device=DEV)
    presc = torch.randn(lists["presc_comp"].size, generator=gen, dtype=torch.float64, device=DEV)
    torch.cuda.synchronize()
    return {"replay": BoundaryReplay(lists, 3, N, N, N, device=torch.cuda.current_device()), "presc": presc,
            "fields": split_fields(flat, shapes)}


def run_bc(s):
    st = torch.cuda.current_stream()
    u, v, w, p = s["fields"]
    s["replay"].EnforceVelocityBC(u, v, w, s["presc"], st)
    s["replay"].EnforcePressureBC(p, None, st)
    return s["fields"]


PREPARE = {"step": prepare_step, "host": prepare_host, "tanks": prepare_tanks, "server": prepare_server,
           "flip": prepare_flip, "relabel": prepare_relabel, "bc": prepare_bc}
RUN = {"step": run_step, "host": run_host, "tanks": run_tanks, "server": run_server, "flip": run_flip,
       "relabel": run_relabel, "bc": run_bc}


def prepare(case, seed):
    return dict(PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return RUN[state["kind"]](state)


# ------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------
def step_work(c):
    fields = sum(int(np.prod(s)) for s in field_shapes(c)) * 8
    cells = int(np.prod(field_shapes(c)[3]))
    extra = 8 * cells if c.get("scheme") else 0
    # velocities in, all four fields out, the labels; divergence and gradient, and one sweep of the operator
    return 2 * fields + extra + cells, 40 * cells


def work(case):
    k = case["kind"]
    if k in ("step", "host"):
        b, f = step_work(case)
    elif k == "tanks":
        b, f = [case["count"] * x for x in step_work(tank_cases(case, 0)[0])]
    elif k == "server":
        per = [step_work(q) for q in request_cases(case)]
        b, f = sum(x for x, _ in per), sum(x for _, x in per)
    elif k == "flip":
        n = case["n"]
        b, f = step_work(flip_case(case))
        b, f = 2 * (b + 24 * case["ppc"] * n ** 3 // 2 + n ** 3), 2 * f
    elif k == "relabel":
        n = case["n"]
        b, f = 24 * case["ppc"] * n ** 3 // 2 + 2 * (n + 2) ** 3, 0
    else:
        n = case["n"]
        lists = 12 * n * n + 2 * 4 * n * n * 4
        b, f = 12 * lists, 0
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------------------------------------------------------
# the exact outputs: plain torch in 64 bits
# ------------------------------------------------------------------------------------------------------------------
class System:
    """The finite-volume pressure system of a grid: sum over faces of c (p_neighbour - p) = rho/dt * net outflow on
    the fluid cells; c is area over the centres' distance, doubled toward a Dirichlet ring cell (half a cell away), no
    flux at solid and inlet faces. Solved by CG, preconditioned by the inverse of the same operator on the box around
    the fluid (a sum of one-dimensional operators, through their eigenvectors)."""

    def __init__(self, c, t):
        self.c, self.t = c, t
        dim = c["dim"]
        self.axes = (1, 0, 2)[:dim]  # array axes of x, y, z
        w = interior_widths(c)
        self.w = [torch.from_numpy(np.concatenate([v[:1], v, v[-1:]])).to(t.device) for v in w][:dim]
        self.unk = unknowns(c, t)
        self.n = int(self.unk.sum())
        fluid = self.unk
        self.coef = []  # per axis, the coupling of cells m and m + 1 (zero where there is none)
        self.diag = torch.zeros(t.shape, dtype=torch.float64, device=t.device)
        dirichlet = t == EMPTY
        any_dir = False
        for q, ax in enumerate(self.axes):
            n = t.shape[ax]
            gap = 0.5 * (self.w[q][1:] + self.w[q][:-1])
            area = torch.ones([1, 1, 1], dtype=torch.float64, device=t.device)
            for r, bx in enumerate(self.axes):
                if r != q:
                    area = area * self.w[r].view([-1 if a == bx else 1 for a in range(3)])
            cf = area / gap.view([-1 if a == ax else 1 for a in range(3)])
            lo, hi = fluid.narrow(ax, 0, n - 1), fluid.narrow(ax, 1, n - 1)
            dlo, dhi = dirichlet.narrow(ax, 0, n - 1), dirichlet.narrow(ax, 1, n - 1)
            ring = torch.ones(n - 1, dtype=torch.float64, device=t.device)
            ring[0] = ring[-1] = 2.0
            ring = ring.view([-1 if a == ax else 1 for a in range(3)])
            both = cf * (lo & hi)
            self.coef.append(both)
            d = self.diag
            d.narrow(ax, 0, n - 1).add_(both + cf * ring * (lo & dhi))
            d.narrow(ax, 1, n - 1).add_(both + cf * ring * (hi & dlo))
            any_dir = any_dir or bool(((lo & dhi) | (hi & dlo)).any())
        self.singular = not any_dir
        self._box()

    def _box(self):
        t = self.t
        nz = torch.nonzero(self.unk)
        lo, hi = nz.min(0).values.tolist(), nz.max(0).values.tolist()
        self.box = tuple(slice(a, b + 1) for a, b in zip(lo, hi))
        self.vec, vals = [], []
        for q, ax in enumerate(self.axes):
            a, b, n = lo[ax], hi[ax], t.shape[ax]
            w = self.w[q]
            gap = 0.5 * (w[1:] + w[:-1])
            m = b - a + 1
            K = torch.zeros(m, m, dtype=torch.float64, device=t.device)
            g = 1.0 / gap[a:b]
            r = torch.arange(m - 1, device=t.device)
            K[r, r + 1] = K[r + 1, r] = -g
            K[r, r] += g
            K[r + 1, r + 1] += g
            for end, cell in ((0, a - 1), (m - 1, b + 1)):
                plane, inner = t.select(ax, cell), self.unk.select(ax, a if end == 0 else b)
                if bool(((plane == EMPTY) & inner).any()):
                    K[end, end] += (2.0 if cell in (0, n - 1) else 1.0) / gap[b if end else a - 1]
            s = w[a:b + 1].sqrt()
            lam, V = torch.linalg.eigh(K / (s[:, None] * s[None, :]))
            self.vec.append(V / s[:, None])
            vals.append(lam.view([-1 if d == ax else 1 for d in range(3)]))
        total = sum(vals)
        floor = 1e-10 * float(total.max())
        self.inv = torch.where(total > floor, 1.0 / total.clamp(min=floor), torch.zeros_like(total))

    def apply(self, x):
        """minus the operator: positive semi-definite."""
        y = self.diag * x
        for q, ax in enumerate(self.axes):
            n = x.shape[ax]
            y.narrow(ax, 0, n - 1).sub_(self.coef[q] * x.narrow(ax, 1, n - 1))
            y.narrow(ax, 1, n - 1).sub_(self.coef[q] * x.narrow(ax, 0, n - 1))
        return y

    def precondition(self, r):
        b = r[self.box]
        for q, ax in enumerate(self.axes):
            b = torch.tensordot(b, self.vec[q], dims=([ax], [0])).movedim(-1, ax)
        b = b * self.inv
        for q, ax in enumerate(self.axes):
            b = torch.tensordot(b, self.vec[q], dims=([ax], [1])).movedim(-1, ax)
        z = torch.zeros_like(r)
        z[self.box] = b
        return self.centre(z * self.unk)

    def centre(self, x):
        return torch.where(self.unk, x - x.sum() / self.n, x) if self.singular else x

    def solve(self, b):
        x = torch.zeros_like(b)
        b = self.centre(b)
        bn = float(b.norm())
        if bn == 0.0:
            return x
        for _ in range(4):  # CG, restarted from the true residual until that stops falling
            r = self.centre(b - self.apply(x))
            rn = float(r.norm())
            if rn <= 2e-15 * bn:
                break
            z = self.precondition(r)
            p, rz = z.clone(), float((r * z).sum())
            dx = torch.zeros_like(x)
            for _ in range(400):
                q = self.apply(p)
                a = rz / float((p * q).sum())
                dx.add_(p, alpha=a)
                r.sub_(q, alpha=a)
                if float(r.norm()) <= 1e-7 * rn:
                    break
                z = self.precondition(r)
                new = float((r * z).sum())
                p.mul_(new / rz).add_(z)
                rz = new
            x = x + dx
        return self.centre(x)

    def area(self, q):
        a = torch.ones([1, 1, 1], dtype=torch.float64, device=self.t.device)
        for r, bx in enumerate(self.axes):
            if r != q:
                a = a * self.w[r].view([-1 if d == bx else 1 for d in range(3)])
        return a

    def net_outflow(self, fields):
        s = torch.zeros(self.t.shape, dtype=torch.float64, device=self.t.device)
        for q, ax in enumerate(self.axes):
            f, n = fields[q], self.t.shape[ax]
            s += (f.narrow(ax, 1, n) - f.narrow(ax, 0, n)) * self.area(q)
        return s * self.unk

    def ring(self, p):
        for ax in (0, 1, 2)[:self.c["dim"]]:
            n = p.shape[ax]
            for at, src in ((0, 1), (n - 1, n - 2)):
                empty = self.t.select(ax, at) == EMPTY
                p.select(ax, at).copy_(torch.where(empty, torch.zeros_like(p.select(ax, src)), p.select(ax, src)))

    def project(self, fields, p):
        """u -= dt/rho grad p on the faces between two cells that are not solid, inside the ring along the others."""
        t, dim = self.t, self.c["dim"]
        for q, ax in enumerate(self.axes):
            n = t.shape[ax]
            gap = (0.5 * (self.w[q][1:] + self.w[q][:-1])).view([-1 if a == ax else 1 for a in range(3)])
            grad = (p.narrow(ax, 1, n - 1) - p.narrow(ax, 0, n - 1)) / gap
            for face, cell in ((0, 0), (n - 2, n - 1)):
                two = t.select(ax, cell) == EMPTY
                grad.select(ax, face).mul_(torch.where(two, 2.0, 1.0))
            grad *= (t.narrow(ax, 0, n - 1) != SOLID) & (t.narrow(ax, 1, n - 1) != SOLID)
            inside = tuple(slice(None) if a == ax or (a == 2 and dim == 2) else slice(1, -1) for a in range(3))
            fields[q].narrow(ax, 1, n - 1)[inside] -= (DT / RHO) * grad[inside]


def exact_step(c, t, base, prev):
    flat = base.clone()
    fields = split_fields(flat, field_shapes(c))
    S = System(c, t)
    x = S.solve(-(RHO / DT) * S.net_outflow(fields))
    p = fields[3]
    p[S.unk] = x[S.unk]
    S.ring(p)
    S.project(fields, p)
    if prev is not None:
        p[S.unk] = S.centre(torch.where(S.unk, prev + x, torch.zeros_like(x)))[S.unk]
        S.ring(p)
    return fields


def exact(case, seed):
    k = case["kind"]
    if k in ("step", "host"):
        out = exact_step(case, *step_inputs(case, seed))
        return [f.reshape(-1).cpu().numpy() for f in out] if k == "host" else out
    if k == "tanks":
        per = [exact_step(q, *step_inputs(q, 1000 * seed + m)) for m, q in enumerate(tank_cases(case, seed))]
        return [f for q in per for f in q]
    if k == "server":
        per = [exact_step(q, *step_inputs(q, 1000 * seed + m)) for m, q in enumerate(request_cases(case))]
        return [f for q in per for f in q]
    if k == "flip":
        labels, fields = [], []
        for step in range(2):
            t = labels_of(particles(case["n"], case["ppc"], seed, step), case["n"])
            labels.append(None)
            fields += exact_step(flip_case(case), t, flip_fields(case, seed, step, t), None)
        return labels + fields
    return None
