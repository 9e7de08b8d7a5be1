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


# (interior x, y, z), stretched; where the memory ends: at the layout, or at the step's copies of host fields
@pytest.mark.parametrize("at", ["layout", "fields"])
@pytest.mark.parametrize("n,stretched,precision", [((320, 160, 161), True, "fp64"), ((240, 240, 239), False, "fp64"),
                                                   ((900, 1000, 9), False, "mixed")])
def test_without_room_for_the_split_layout(nb, n, stretched, precision, at):
    """A grid whose colour-split layout does not fit the device's free memory while the grid layout does, as it did before
    the split layout was these grids' default: it is solved by the grid layout's kernels (those of pair_kernels = 1), bit
    for bit."""
    import torch

    if stretched:
        case = W.stretched_cylinder_3d(*n)
    else:
        h = 1.0 / min(n[:2])
        g = W.uniform_grid(3, (0.0, n[0] * h, 0.0, n[1] * h, 0.0, n[2] * h), min(n[:2]))
        case = W.Case("box", g, W.walls_scene(3, outlet_face=1), 3)
    job = serving.job_from_case(case, tol=1e-6)

    def free():
        return torch.cuda.mem_get_info()[0]

    def run(family, room=None):
        """The step's fields, and the memory that the layout and the whole context take. room: the free bytes there are
        for the layout, or for all of it."""
        torch.cuda.empty_cache()
        j, hog = copy.deepcopy(job), None
        if room is not None:
            hog = torch.empty(free() - room, dtype=torch.uint8, device="cuda")
        start = free()
        s = PressureSolver(precision, pair_kernels=family, max_iters=4, max_outer=1)
        s.InitializePressureSolver(j.grid)
        layout = start - free()
        if at == "layout":
            del hog
            torch.cuda.empty_cache()
        s.SolvePressure(j.grid, tol=j.tol)
        whole = start - free()
        s.DestroyPressureSolver()
        return j.grid, layout, whole

    run(2)  # loads the kernels' code
    run(1)
    expect, *lean = run(1)
    _, *split = run(2)
    q = 0 if at == "layout" else 1
    assert split[q] - lean[q] > 64 << 20
    try:
        got, _, _ = run(2, (lean[q] + split[q]) // 2)
    finally:
        torch.cuda.empty_cache()  # the memory that was held back
    for f in ("p", "u", "v", "w"):
        assert np.array_equal(getattr(got, f), getattr(expect, f)), f
