"""Parity at the sizes the benchmark configurations name, through the C ABI.

* The 2D 128^2 closed box (all-Neumann, compatibility on) at its own tolerance 1e-10, against the reference's Eigen-CG
  solution at 1e-12 (tests/golden/closed_box_2d_128.npz): mean-free pressure within 1e-6 relative L2.
* The 3D sphere-outlet workload at 208^3, whose first coarse levels (106^3 = 1,191,016 and 55^3 = 166,375 cells) lie above
  the 2^17 cells from which the colour-split restriction runs one thread per four coarse cells, as they do on the 256^3
  headline grid, and whose next one lies below:
  - the two restriction kernels (one thread per coarse cell, one per four) give the same bits through a whole mixed
    solve, and so does the default choice between them;
  - the mixed and the plain FP64 solves to 1e-8 against the reference's own solve of the same system
    (oracle/_ref/ref_harness, AMGCL SA+SPAI0 CG, run on this host): relative residual <= 1e-8, pressure within 1e-6
    relative L2 of the reference's solve at 1e-12, and max |div u| within 10x of the reference's at 1e-8, driven the
    way tests/suite_pressure.cpp:104-141 drives the reference.
* A 2D box of 4608^2 cells, whose sums run over more blocks than a solver keeps room for at least, against numpy's sums.
"""
import os

import numpy as np
import pytest

from conftest import load_golden
from nereus_cfd_b200 import capi, workloads as W
from nereus_cfd_b200.pressure import MACGrid, PressureSolver
from oracle import refcase

pytestmark = pytest.mark.gpu
SIZE = 208


def mean_free_err(x, xr, singular):
    if singular:
        x, xr = x - x.mean(), xr - xr.mean()
    return float(np.linalg.norm(x - xr) / max(np.linalg.norm(xr), 1e-300))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_closed_box_128_at_its_own_tolerance(nb, precision):
    case, meta, z = load_golden("closed_box_2d_128")
    assert case.tol == 1e-10 and meta["needs_compat"] and meta["singular"]
    m = MACGrid(case.grid, z["types"].copy(), z["u"].copy(), z["v"].copy(), z["w"].copy(), z["p_in"].copy(),
                meta["rho"], meta["dt"])
    s = PressureSolver(precision)
    r = s.SolvePressure(m, tol=case.tol, needs_compat=True)
    assert r.status == capi.NB_OK and r.rel_res <= case.tol, r.as_dict()
    idp = z["idp"]
    x = m.p[idp >= 0][np.argsort(idp[idp >= 0])]
    assert mean_free_err(x, z["x"], True) <= 1e-6
    s.DestroyPressureSolver()


@pytest.fixture(scope="module")
def big():
    case = W.sphere_outlet_3d(SIZE, seed=2)
    types = capi.label_cells(case.grid, case.scene)
    u, v, w = W.face_velocities(case.grid, types, case.seed)
    return case, types, u, v, w


def solve(big, precision, tol=1e-8, **opts):
    case, types, u, v, w = big
    m = MACGrid.from_case(case, types, u.copy(), v.copy(), w.copy())
    s = PressureSolver(precision, **opts)
    r = s.SolvePressure(m, tol=tol)
    mask = s.IDP() >= 0
    s.DestroyPressureSolver()
    return r, m, mask


def test_quad_and_per_cell_restriction_agree(nb, big):
    r1, m1, _ = solve(big, "mixed", transfer_kernels=1)
    r2, m2, _ = solve(big, "mixed", transfer_kernels=2)
    r0, m0, _ = solve(big, "mixed")
    for r in (r1, r2, r0):
        assert r.status == capi.NB_OK and r.rel_res <= 1e-8, r.as_dict()
    assert (r1.iters_inner, r1.iters_outer) == (r2.iters_inner, r2.iters_outer)
    assert np.array_equal(m1.p, m2.p), np.abs(m1.p - m2.p).max()
    assert np.array_equal(m1.u, m2.u) and np.array_equal(m1.v, m2.v) and np.array_equal(m1.w, m2.w)
    # the default runs one kernel on the larger levels and the other on the smaller
    assert np.array_equal(m0.p, m2.p)


@pytest.fixture(scope="module")
def reference(big):
    if not refcase.available():
        pytest.skip("oracle/_ref/ref_harness is not built")
    case, types, u, v, w = big
    threads = os.cpu_count() or 1
    run = lambda tol: refcase.run(case, u, v, w, label_mode=1, types=types, solver=refcase.SOLVER_AMG, tol=tol,
                                  threads=threads, timeout=1800, lean=True)
    return run(1e-12), run(1e-8)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_headline_size_against_reference(nb, big, reference, precision):
    r12, r8 = reference
    assert r12.rel_res <= 1e-11 and r8.rel_res <= 1e-8
    r, m, mask = solve(big, precision)
    assert r.status == capi.NB_OK and r.rel_res <= 1e-8, r.as_dict()
    assert r.n == r12.n and r.singular == int(r12.singular)
    err = mean_free_err(m.p[mask], r12.p[mask], r12.singular)
    assert err <= 1e-6, err
    # the cells off the unknowns (solid, outlet ring, copied walls) as the reference leaves them, to the solution's
    # tolerance for the copies
    scale = np.abs(r12.p).max()
    assert np.abs(m.p[~mask] - r12.p[~mask]).max() <= 1e-6 * scale
    assert r.max_div <= 10.0 * r8.max_div, (r.max_div, r8.max_div)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_sums_over_more_blocks_than_the_least_room(nb, precision):
    """A 2D box of 4608^2 cells, whose grid-wide sums run over 82,944 blocks where a solver keeps room for 65,536 at least:
    the count of unknowns, the reported residual and divergence against numpy's. The residual's own rounding is of the
    order of 8 (products and sums per cell) times 2^-53 of |A| |p| / |b|; after a few iterations on this box |A| |p| is
    below 1e3 |b|, so the two agree to 1e-12 of |b|, and rel_res is far above that."""
    n, rho, dt = 4608, 1.0, 1e-3
    assert capi.load().nereus_b200_sum_blocks(2, n + 2, n + 2, 1) == 144 * 576
    g = W.uniform_grid(2, (0.0, 1.0, 0.0, 1.0, 0.0, 1.0), n)
    types = capi.label_cells(g, W.walls_scene(2))
    rng = np.random.default_rng(12)
    u, v = np.zeros((n + 2, n + 3)), np.zeros((n + 3, n + 2))
    u[1:-1, 2:-2] = rng.normal(size=(n, n - 1))
    v[2:-2, 1:-1] = rng.normal(size=(n - 1, n))
    m = MACGrid(g, types, u.reshape(-1).copy(), v.reshape(-1).copy(), np.zeros(1), np.zeros(g.cells), rho, dt)
    s = PressureSolver(precision, max_iters=3, max_outer=1)
    r = s.SolvePressure(m, tol=1e-10)
    s.DestroyPressureSolver()
    assert r.status == capi.NB_NOT_CONVERGED and r.n == n * n

    def divergence(u, v):
        return (u[1:-1, 2:-1] - u[1:-1, 1:-2]) / g.dh + (v[2:-1, 1:-1] - v[1:-2, 1:-1]) / g.dh

    b = rho / dt * divergence(u, v)
    p = np.pad(m.p.reshape(n + 2, n + 2)[1:-1, 1:-1], 1, mode="edge")
    inner = p[1:-1, 1:-1]
    lap = ((p[2:, 1:-1] - inner) + (p[:-2, 1:-1] - inner) + (p[1:-1, 2:] - inner) + (p[1:-1, :-2] - inner)) / g.dh ** 2
    rel = np.linalg.norm(b - lap) / np.linalg.norm(b)
    assert rel > 1e-6 and abs(r.rel_res - rel) <= 1e-12
    after = np.abs(divergence(m.u.reshape(u.shape), m.v.reshape(v.shape))).max()
    assert abs(r.max_div - after) <= 1e-12 * after
