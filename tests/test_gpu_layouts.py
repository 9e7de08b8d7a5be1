"""A context reused across layouts gives what a fresh context gives, through the C ABI: a uniform grid of the same
sizes at another cell width (the hierarchy keeps its shape and captured iterations; the spacing tables and the
matrix scale are replaced) and a 2D grid after it, in both precisions, bit for bit."""
import copy

import numpy as np
import pytest

from nereus_cfd_b200 import serving, workloads as W
from nereus_cfd_b200.pressure import PressureSolver

pytestmark = pytest.mark.gpu


def sphere_box(L, n, seed):
    g = W.uniform_grid(3, (0.0, L, 0.0, L, 0.0, L), n)
    sph = W.Region(W.REGION_SOLID, W.PRIM_SPHERE, (0.5 * L, 0.5 * L, 0.5 * L), radius=0.15 * L)
    return W.Case("sphere_box_%g_%d" % (L, n), g, W.walls_scene(3, outlet_face=1, regions=[sph]), seed)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_rescaled_uniform_layout_equals_fresh(nb, precision):
    jobs = [serving.job_from_case(sphere_box(L, 24, s), tol=1e-9) for L, s in ((1.0, 5), (2.5, 6), (0.3, 7))]
    jobs.append(serving.job_from_case(W.closed_box_2d(40, seed=8), tol=1e-9))
    reused = PressureSolver(precision)
    for j in jobs:
        a, b = copy.deepcopy(j), copy.deepcopy(j)
        ra = reused.SolvePressure(a.grid, tol=j.tol, needs_compat=j.needs_compat)
        fresh = PressureSolver(precision)
        rb = fresh.SolvePressure(b.grid, tol=j.tol, needs_compat=j.needs_compat)
        fresh.DestroyPressureSolver()
        assert ra.status == rb.status == 0 and ra.rel_res <= j.tol
        assert (ra.iters_inner, ra.iters_outer, ra.rel_res) == (rb.iters_inner, rb.iters_outer, rb.rel_res)
        for f in ("p", "u", "v", "w"):
            assert np.array_equal(getattr(a.grid, f), getattr(b.grid, f)), f
    reused.DestroyPressureSolver()


def disc_channel(nx, ny, at, seed, L=1.0):
    """A 2D channel with an outlet around a solid disc whose centre is ``at`` (in units of L)."""
    g = W.uniform_grid(2, (0.0, nx * L / ny, 0.0, L, 0.0, L), ny)
    disc = W.Region(W.REGION_SOLID, W.PRIM_SPHERE, (at[0] * L, at[1] * L, 0.0), radius=0.12 * L)
    return W.Case("disc_%d_%d" % (nx, ny), g, W.walls_scene(2, outlet_face=1, regions=[disc]), seed)


def solve_both(reused, case, precision, tol=1e-9):
    """The same step on the reused solver and on a fresh one: the same report, the same bits."""
    j = serving.job_from_case(case, tol=tol)
    a, b = copy.deepcopy(j), copy.deepcopy(j)
    ra = reused.SolvePressure(a.grid, tol=tol)
    fresh = PressureSolver(precision)
    rb = fresh.SolvePressure(b.grid, tol=tol)
    fresh.DestroyPressureSolver()
    assert ra.status == rb.status == 0 and ra.rel_res <= tol
    assert (ra.iters_inner, ra.iters_outer, ra.rel_res) == (rb.iters_inner, rb.iters_outer, rb.rel_res)
    for f in ("p", "u", "v"):
        assert np.array_equal(getattr(a.grid, f), getattr(b.grid, f)), f


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_2d_moved_labels_equal_fresh(nb, precision):
    """A 2D grid solved until its iterations are captured, then with moved labels and with another cell width, all of
    one shape and one singularity: each solve gives what a fresh context gives. Smaller shapes before it leave holes in
    the context's memory, so that an array given back and taken again on a layout change would lie elsewhere."""
    reused = PressureSolver(precision)
    for nx, ny in ((40, 40), (64, 48), (90, 57)):
        solve_both(reused, disc_channel(nx, ny, (0.4, 0.5), 11), precision)
    for n, (at, L) in enumerate((((0.40, 0.50), 1.0), ((0.40, 0.50), 1.0), ((0.40, 0.50), 1.0), ((0.45, 0.52), 1.0),
                                 ((0.62, 0.40), 1.0), ((0.62, 0.40), 2.5), ((0.30, 0.55), 2.5), ((0.30, 0.55), 2.5))):
        solve_both(reused, disc_channel(150, 130, at, 20 + n, L), precision)
    reused.DestroyPressureSolver()
