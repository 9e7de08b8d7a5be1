"""The server on the B200 (nereus_b200_server_* through nereus_cfd_b200.serving): a mix of different requests run
concurrently (several slots on one device) gives each request exactly what it gives alone through
nereus_b200_project / _ex; admission by the memory budget; the statistics."""
import numpy as np
import pytest

from conftest import load_golden, scheme_golden_names
from nereus_cfd_b200 import capi, serving
from nereus_cfd_b200 import workloads as W
from nereus_cfd_b200.pressure import MACGrid, PressureSolver

pytestmark = pytest.mark.gpu


def mix():
    cases = [W.sphere_outlet_3d(24, seed=40), W.flip_tank_3d(20, seed=41), W.flip_tank_3d(20, seed=42),
             W.closed_box_2d(48, seed=43), W.stretched_cylinder_3d(24, 16, 16, seed=44),
             W.sphere_outlet_3d(16, seed=45), W.pressure_outlet_3d(14, seed=46), W.flip_tank_3d(32, seed=47)]
    jobs = [serving.job_from_case(c, tol=1e-9) for c in cases]
    # one incremental request from its fixture
    name = [n for n in scheme_golden_names() if n.startswith("incremental_")][0]
    case, meta, z = load_golden(name)
    m = MACGrid(case.grid, z["types"].copy(), z["u"].copy(), z["v"].copy(), z["w"].copy(), z["p_in"].copy(),
                meta["rho"], meta["dt"])
    jobs.append(serving.Job(m, tol=1e-9, needs_compat=meta["needs_compat"], scheme=capi.SCHEME_INCREMENTAL,
                            p_prev=z["p_prev"].copy()))
    return jobs


def alone(job, precision):
    m = job.grid
    s = PressureSolver(precision)
    s.InitializePressureSolver(m, job.scheme)
    ant = None
    if job.p_prev is not None:
        ant = MACGrid(m.grid, m.types, m.u, m.v, m.w, job.p_prev, m.rho, m.dt)
    r = s.SolvePressure(m, tol=job.tol, needs_compat=job.needs_compat, grid_ant=ant)
    s.DestroyPressureSolver()
    return r


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_mix_equals_alone(nb, precision):
    served = mix()
    ref = mix()
    with serving.Server(slots_per_device=4, precision=precision) as srv:
        st = serving.serve(served, srv)
    assert st["completed"] == len(served) and st["failed"] == 0
    assert st["p50_ms"] <= st["p99_ms"] and st["solves_per_s"] > 0
    for a, b in zip(served, ref):
        r = alone(b, precision)
        assert a.status == capi.NB_OK and r.status == capi.NB_OK
        assert a.result["iters_inner"] == r.iters_inner
        for f in ("p", "u", "v", "w"):
            assert np.array_equal(getattr(a.grid, f), getattr(b.grid, f)), f


def test_device_fields_equal_host_fields(nb):
    host = mix()
    dev = [serving.to_device(j) for j in mix()]
    with serving.Server(slots_per_device=4) as srv:
        serving.serve(host, srv)
    with serving.Server(slots_per_device=4) as srv:
        serving.serve(dev, srv)
    for a, b in zip(host, dev):
        serving.fetch(b)
        assert a.status == b.status == capi.NB_OK
        assert a.result["iters_inner"] == b.result["iters_inner"]
        for f in ("p", "u", "v", "w"):
            assert np.array_equal(getattr(a.grid, f), getattr(b.grid, f)), f


def slab(dim, n, stretched=False):
    """A grid of n interior cells a side, its cell widths along x growing from the middle when stretched."""
    if stretched:
        w = [W.band_stretched_widths(n[0], 2.2, max(2, n[0] // 8 // 2 * 2), 0.5, 1.04)]
        w += [np.full(m, 0.41 / m) for m in n[1:]]
        g = W.stretched_grid(dim, (0.0, 2.2, 0.0, 0.41, 0.0, 0.41), w)
    else:
        h = 1.0 / min(n[:2])
        g = W.uniform_grid(dim, (0.0, n[0] * h, 0.0, n[1] * h, 0.0, n[-1] * h), min(n[:2]))
    return W.Case("slab", g, W.walls_scene(dim, outlet_face=1), 3)


# stretched 3D grids in FP64 (whose levels keep their diagonals) of both parities of Nz, a thin one whose padded rows are
# 1.6 times its cells, a 2D one
@pytest.mark.parametrize("dim,n,stretched,precision", [
    (3, (384, 192, 192), True, "fp64"), (3, (400, 200, 151), True, "fp64"), (3, (200, 200, 251), False, "fp64"),
    (3, (1000, 1100, 8), False, "fp64"), (3, (1000, 1100, 8), False, "mixed"), (3, (240, 240, 240), False, "mixed"),
    (3, (384, 192, 192), True, "mixed"), (2, (3000, 3000), False, "fp64"), (2, (3000, 3000), False, "mixed")])
def test_request_bytes_cover_what_a_solve_takes(nb, dim, n, stretched, precision):
    """The admission estimate against the device memory a context holds after a step on host fields."""
    import torch

    g = slab(dim, n, stretched).grid
    types = capi.label_cells(g, W.walls_scene(dim, outlet_face=1))
    fields = [np.zeros(k) for k in (g.Ny * (g.Nx + 1) * g.Nz, (g.Ny + 1) * g.Nx * g.Nz,
                                    g.Ny * g.Nx * (g.Nz + 1) if dim == 3 else 1, g.cells)]
    fields[0][:] = np.random.default_rng(1).normal(size=fields[0].size)
    for warm in (True, False):  # the kernels' code is loaded by a first, small solve
        h = slab(dim, (24, 24, 16)[:dim], stretched).grid if warm else g
        t = capi.label_cells(h, W.walls_scene(dim, outlet_face=1)) if warm else types
        f = [np.zeros(k) for k in (h.Ny * (h.Nx + 1) * h.Nz, (h.Ny + 1) * h.Nx * h.Nz,
                                   h.Ny * h.Nx * (h.Nz + 1) if dim == 3 else 1, h.cells)] if warm else fields
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        s = PressureSolver(precision, max_iters=3, max_outer=1)
        s.SolvePressure(MACGrid(h, t, *f), tol=1e-8)
        used = free - torch.cuda.mem_get_info()[0]
        s.DestroyPressureSolver()
    prec = capi.PRECISION_FP64 if precision == "fp64" else capi.PRECISION_MIXED
    assert used <= serving.request_bytes(serving.Job(MACGrid(g, types, *fields)), prec)


def test_admission_budget(nb):
    job = mix()[0]
    with serving.Server(hbm_budget_gb=0.01) as srv:
        with pytest.raises(capi.NBError) as e:
            srv.submit(job)
        assert e.value.status == capi.NB_BAD_INPUT
    need = serving.request_bytes(job) / 1e9
    # a budget for one request at a time: all still complete, one after another
    jobs = mix()[:4]
    with serving.Server(hbm_budget_gb=max(serving.request_bytes(j) for j in jobs) / 1e9 * 1.01,
                        slots_per_device=4) as srv:
        st = serving.serve(jobs, srv)
    assert need > 0 and st["completed"] == 4


def test_poll_and_bad_requests(nb):
    job = mix()[0]
    with serving.Server() as srv:
        t = srv.submit(job)
        st = srv.poll(t)
        assert st in (capi.NB_BUSY, capi.NB_OK)
        assert srv.wait(t, 60.0) == capi.NB_OK
        assert srv.poll(t) == capi.NB_OK
        res = capi.Result()
        assert srv.lib.nereus_b200_poll(srv.srv, 987654321, None) == capi.NB_BAD_INPUT
        bad = serving.Job(job.grid, scheme=capi.SCHEME_INCREMENTAL)  # no previous pressure
        with pytest.raises(capi.NBError):
            srv.submit(bad)
