"""The three FP32 kernel families of the mixed-precision inner solve against each other and the reference.

pair_kernels = 0 (per-cell kernels), 1 (cell pairs in the grid layout), 2 (the colour-split layout, the default):
the same V-cycle up to FP32 rounding, so every family meets the parity bars of the solve (relative residual <= the
tolerance, mean-free pressure within 1e-6 rel-L2 of the reference's solution), and on grids deep enough for several
colour-split levels the split solution agrees with the cell-pair one to the solve's tolerance.
"""
import numpy as np
import pytest

from conftest import golden_names, load_golden
from nereus_cfd_b200 import capi, workloads as W
from nereus_cfd_b200.pressure import MACGrid, PressureSolver

pytestmark = pytest.mark.gpu
FAMILIES = [0, 1, 2]
NAMES_3D = [n for n in golden_names() if "_3d_" in n]


def mac_from_golden(case, meta, z):
    return MACGrid(case.grid, z["types"].copy(), z["u"].copy(), z["v"].copy(), z["w"].copy(), z["p_in"].copy(),
                   meta["rho"], meta["dt"])


@pytest.mark.parametrize("family", FAMILIES)
@pytest.mark.parametrize("name", NAMES_3D)
def test_family_against_reference(nb, name, family):
    case, meta, z = load_golden(name)
    s = PressureSolver("mixed", pair_kernels=family)
    m = mac_from_golden(case, meta, z)
    r = s.SolvePressure(m, tol=meta["tol"], needs_compat=meta["needs_compat"])
    assert r.status == capi.NB_OK, r.as_dict()
    assert r.rel_res <= meta["tol"]
    if meta["n"]:
        idp = z["idp"]
        x = m.p[idp >= 0][np.argsort(idp[idp >= 0])]
        xr = z["x"]
        if meta["singular"]:
            x, xr = x - x.mean(), xr - xr.mean()
        assert np.linalg.norm(x - xr) / max(np.linalg.norm(xr), 1e-300) <= 1e-6
    s.DestroyPressureSolver()


def closed_box_3d(n):
    g = W.uniform_grid(3, (0.0, 1.0, 0.0, 1.0, 0.0, 1.0), n)
    sph = W.Region(W.REGION_SOLID, W.PRIM_SPHERE, (0.4, 0.5, 0.6), radius=0.2)
    return W.Case("closed_box_3d_%d" % n, g, W.walls_scene(3, regions=[sph]), 9, needs_compat=True, tol=1e-9)


CASES = {
    "sphere_outlet_48": lambda: W.sphere_outlet_3d(48),
    "flip_tank_40": lambda: W.flip_tank_3d(40),
    "stretched_cylinder_48x32x32": lambda: W.stretched_cylinder_3d(48, 32, 32),
    "closed_box_40": lambda: closed_box_3d(40),
    # 30 x 36 x 26 interior cells: odd coarse sizes along x and z (15, 13), rows padded to the split's multiple of 4
    "sphere_outlet_30x36x26": lambda: W.Case(
        "sphere_outlet_30x36x26", W.uniform_grid(3, (0.0, 1.0, 0.0, 1.2, 0.0, 26.0 / 30.0), 30),
        W.sphere_outlet_3d(8).scene, 2),
}


def solve(case, family, tol):
    g = case.grid
    types = capi.label_cells(g, case.scene)
    u, v, w = W.face_velocities(g, types, case.seed, case.velocity_rule, case.fp32_velocity)
    m = MACGrid(g, types.copy(), u.copy(), v.copy(), w.copy(), np.zeros(g.cells), case.rho, case.dt)
    s = PressureSolver("mixed", pair_kernels=family)
    r = s.SolvePressure(m, tol=tol, needs_compat=case.needs_compat)
    s.DestroyPressureSolver()
    return r, m, types


@pytest.mark.parametrize("name", sorted(CASES))
def test_split_agrees_with_pairs(nb, name):
    case = CASES[name]()
    tol = 1e-9
    r2, m2, types = solve(case, 2, tol)
    r1, m1, _ = solve(case, 1, tol)
    assert r2.status == capi.NB_OK and r1.status == capi.NB_OK
    assert r2.rel_res <= tol and r1.rel_res <= tol
    assert r2.levels >= 3
    unk = np.zeros(case.grid.shape, dtype=bool)
    unk[1:-1, 1:-1, 1:-1] = (types.reshape(case.grid.shape) == W.FLUID)[1:-1, 1:-1, 1:-1]
    unk = unk.reshape(-1)
    p1, p2 = m1.p[unk], m2.p[unk]
    if r1.singular:
        p1, p2 = p1 - p1.mean(), p2 - p2.mean()
    assert np.linalg.norm(p2 - p1) / max(np.linalg.norm(p1), 1e-300) <= 1e-6
    # the same preconditioner up to FP32 rounding: about the same iterations
    assert abs(r2.iters_inner - r1.iters_inner) <= 2 + r1.iters_inner // 5, (r2.iters_inner, r1.iters_inner)


def test_split_repeat_is_bit_identical(nb):
    case = W.sphere_outlet_3d(32)
    _, a, _ = solve(case, 2, 1e-10)
    _, b, _ = solve(case, 2, 1e-10)
    assert np.array_equal(a.p, b.p) and np.array_equal(a.u, b.u)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_device_loop_equals_host_loop(nb, precision):
    """The CG loop as one graph with a device-side WHILE condition (use_graphs = 2), one graph per iteration
    (use_graphs = 1) and plain launches iteration by iteration from the host (use_graphs = 0) run the same kernels in
    the same order: the same iterations and the same bits."""
    case = W.sphere_outlet_3d(40)
    g = case.grid
    types = capi.label_cells(g, case.scene)
    u, v, w = W.face_velocities(g, types, case.seed, case.velocity_rule, case.fp32_velocity)
    out = []
    for graphs in (2, 1, 0):
        m = MACGrid(g, types.copy(), u.copy(), v.copy(), w.copy(), np.zeros(g.cells), case.rho, case.dt)
        s = PressureSolver(precision, use_graphs=graphs)
        r = s.SolvePressure(m, tol=1e-9)
        assert r.status == capi.NB_OK and r.rel_res <= 1e-9
        # a second solve on the same context replays the loop built by the first
        m2 = MACGrid(g, types.copy(), u.copy(), v.copy(), w.copy(), np.zeros(g.cells), case.rho, case.dt)
        r2 = s.SolvePressure(m2, tol=1e-9)
        s.DestroyPressureSolver()
        assert np.array_equal(m.p, m2.p) and r.iters_inner == r2.iters_inner
        out.append((r.iters_inner, r.iters_outer, m.p, m.u))
    for o in out[1:]:
        assert out[0][:2] == o[:2]
        assert np.array_equal(out[0][2], o[2]) and np.array_equal(out[0][3], o[3])


def test_device_loop_stops_at_the_iteration_cap(nb):
    case = W.sphere_outlet_3d(32)
    g = case.grid
    types = capi.label_cells(g, case.scene)
    u, v, w = W.face_velocities(g, types, case.seed, case.velocity_rule, case.fp32_velocity)
    m = MACGrid(g, types.copy(), u.copy(), v.copy(), w.copy(), np.zeros(g.cells), case.rho, case.dt)
    s = PressureSolver("fp64", max_iters=2, max_outer=1)
    r = s.SolvePressure(m, tol=1e-12)
    s.DestroyPressureSolver()
    assert r.status == capi.NB_NOT_CONVERGED
    assert r.iters_inner == 2


@pytest.mark.parametrize("name", ["closed_box_2d", "stretched_cylinder_3d", "flip_tank_3d"])
def test_device_refinement_loop_equals_host_loop(nb, name):
    """The mixed solve as one graph (use_graphs = 2: the refinement passes in a WHILE node around the CG loop's WHILE
    node) and the refinement loop on the host (use_graphs = 1): the same passes, iterations and bits, on a singular
    2D box (compatibility on), a stretched 3D channel and a free-surface tank."""
    case = {"closed_box_2d": lambda: W.closed_box_2d(48, seed=3),
            "stretched_cylinder_3d": lambda: W.stretched_cylinder_3d(24, 16, 16, seed=4),
            "flip_tank_3d": lambda: W.flip_tank_3d(30, seed=5)}[name]()
    g = case.grid
    types = capi.label_cells(g, case.scene)
    u, v, w = W.face_velocities(g, types, case.seed, case.velocity_rule, case.fp32_velocity)
    out = []
    for graphs in (2, 1):
        s = PressureSolver("mixed", use_graphs=graphs)
        for rep in range(2):
            m = MACGrid(g, types.copy(), u.copy(), v.copy(), w.copy(), np.zeros(g.cells), case.rho, case.dt)
            r = s.SolvePressure(m, tol=1e-10, needs_compat=case.needs_compat)
            assert r.status == capi.NB_OK and r.rel_res <= 1e-10
            out.append((r.iters_inner, r.iters_outer, r.rel_res, m.p, m.u, m.v))
        s.DestroyPressureSolver()
    for o in out[1:]:
        assert out[0][:3] == o[:3]
        for a, b in zip(out[0][3:], o[3:]):
            assert np.array_equal(a, b)


def test_device_refinement_loop_limits(nb):
    """The device-side refinement loop stops at max_outer passes with NOT_CONVERGED, and a zero right-hand side needs
    no pass at all."""
    case = W.sphere_outlet_3d(24, seed=6)
    g = case.grid
    types = capi.label_cells(g, case.scene)
    u, v, w = W.face_velocities(g, types, case.seed, case.velocity_rule, case.fp32_velocity)
    s = PressureSolver("mixed", max_outer=1)
    m = MACGrid(g, types.copy(), u.copy(), v.copy(), w.copy(), np.zeros(g.cells), case.rho, case.dt)
    r = s.SolvePressure(m, tol=1e-14)
    assert r.status == capi.NB_NOT_CONVERGED and r.iters_outer == 1 and r.rel_res > 1e-14
    z = MACGrid(g, types.copy(), np.zeros_like(u), np.zeros_like(v), np.zeros_like(w), np.zeros(g.cells), case.rho,
                case.dt)
    r0 = s.SolvePressure(z, tol=1e-8)
    s.DestroyPressureSolver()
    assert r0.status == capi.NB_OK and r0.iters_outer == 0 and r0.iters_inner == 0 and r0.rel_res == 0.0
    assert not np.any(z.p[types == W.FLUID])


def sphere_case(size, closed):
    """A box of cubic cells of the given interior size around a solid sphere, closed or with an outlet."""
    nx, ny, nz = size
    h = 1.0 / min(nx, ny)
    g = W.uniform_grid(3, (0.0, nx * h, 0.0, ny * h, 0.0, nz * h), min(nx, ny))
    assert (g.Nx, g.Ny, g.Nz) == (nx + 2, ny + 2, nz + 2)
    sph = W.Region(W.REGION_SOLID, W.PRIM_SPHERE, (0.5 * nx * h, 0.5 * ny * h, 0.5 * nz * h), radius=0.2 * min(size) * h)
    case = W.Case("sphere", g, W.walls_scene(3, outlet_face=None if closed else 1, regions=[sph]), 31,
                  needs_compat=closed)
    return case, capi.label_cells(g, case.scene)


def solve_family(case, types, family, precision, closed, tol=1e-12, **options):
    g = case.grid
    u, v, w = W.face_velocities(g, types, case.seed)
    m = MACGrid(g, types.copy(), u, v, w, np.zeros(g.cells), case.rho, case.dt)
    s = PressureSolver(precision, pair_kernels=family, **dict({"tail_cells": 512}, **options))
    r = s.SolvePressure(m, tol=tol, needs_compat=closed)
    assert r.status == capi.NB_OK and r.rel_res <= tol, r.as_dict()
    s.DestroyPressureSolver()
    return m


# FP64: (interior x, y, z), outlet or closed; row lengths around the 16-byte quads and their padding, one tile and
# several, the smallest grid with a split level above the coarse end and its neighbours
FP64_SIZES = [(12, 12, 12), (14, 13, 16), (16, 16, 14), (30, 36, 26), (33, 40, 48), (64, 20, 34)]


# sweeps: small levels run one launch per leg with one sweep, and a launch per operation with two
@pytest.mark.parametrize("sweeps", [1, 2])
@pytest.mark.parametrize("closed", [False, True])
@pytest.mark.parametrize("size", FP64_SIZES)
def test_fp64_split_agrees_with_per_cell_kernels(nb, size, closed, sweeps):
    """The plain FP64 form on the colour-split layout against its per-cell kernels (pair_kernels = 0), both to 1e-12.
    Each solution is within cond * 1e-12 of the exact one; cond <= 5 N^2 on N cells along the longest side (the lowest
    mode a quarter wave), so the two agree within 1e-11 N^2."""
    case, types = sphere_case(size, closed)
    a, b = [solve_family(case, types, family, "fp64", closed, pre_sweeps=sweeps, post_sweeps=sweeps)
            for family in (2, 0)]
    bar = 1e-11 * max(size) ** 2
    for x, y in ((a.p, b.p), (a.u, b.u), (a.v, b.v), (a.w, b.w)):
        assert np.linalg.norm(x - y) <= bar * np.linalg.norm(y)


# Nz odd: the last cell of a row has no pair, and one colour's rows hold a cell less. (interior x, y, z), row lengths
# around the quads and their padding; the last two have odd levels below an even one and above the coarse end
ODD_SIZES = [(12, 12, 9), (16, 13, 15), (17, 15, 17), (24, 31, 33), (33, 40, 47), (20, 20, 38), (28, 36, 50)]


@pytest.mark.parametrize("sweeps", [1, 2])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("size", ODD_SIZES)
def test_odd_rows_agree_with_per_cell_kernels(nb, size, precision, sweeps):
    """The colour-split layout on grids and levels of odd Nz against the per-cell kernels, closed and with an outlet,
    all to 1e-12 (the bar of test_fp64_split_agrees_with_per_cell_kernels)."""
    for closed in (False, True):
        case, types = sphere_case(size, closed)
        a, b = [solve_family(case, types, family, precision, closed, pre_sweeps=sweeps, post_sweeps=sweeps)
                for family in (2, 0)]
        bar = 1e-11 * max(size) ** 2
        for x, y in ((a.p, b.p), (a.u, b.u), (a.v, b.v), (a.w, b.w)):
            assert np.linalg.norm(x - y) <= bar * np.linalg.norm(y)


# (interior x, y, z): fine rows around the restriction's quads of coarse cells (2 doubles, 4 floats) and a last quad that is
# partly past the row, Nz even and odd, one coarse split level and several
RESTRICT_SIZES = FP64_SIZES + ODD_SIZES + [(40, 24, 18), (26, 22, 70)]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("size", RESTRICT_SIZES)
def test_restriction_by_quads_equals_per_cell(nb, size, precision):
    """The restriction of colour-split levels with one thread per coarse cell (transfer_kernels = 1) and with one per quad
    of them (2): the same sums in the same order, so whole solves agree bit for bit. Two sweeps, because with one a launch
    per leg takes levels of these sizes."""
    for closed in (False, True):
        case, types = sphere_case(size, closed)
        a, b = [solve_family(case, types, 2, precision, closed, tol=1e-10, pre_sweeps=2, post_sweeps=2,
                             transfer_kernels=mode) for mode in (1, 2)]
        for f in ("p", "u", "v", "w"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("groups", [1, 0])
@pytest.mark.parametrize("size", [(24, 16, 16), (32, 17, 15), (48, 32, 33), (64, 24, 40), (97, 30, 21)])
def test_stretched_restriction_by_quads_equals_per_cell(nb, size, groups):
    """The same on stretched FP64 grids, x groups on and off."""
    case = W.stretched_cylinder_3d(*size)
    types = capi.label_cells(case.grid, case.scene)
    a, b = [solve_family(case, types, 2, "fp64", False, tol=1e-10, x_groups=groups, transfer_kernels=mode)
            for mode in (1, 2)]
    for f in ("p", "u", "v", "w"):
        assert np.array_equal(getattr(a, f), getattr(b, f)), f


# stretched FP64: (interior x, y, z) of the cylinder channel; Nz even and odd, one level above the coarse end and
# several, x groups on and off
@pytest.mark.parametrize("groups", [1, 0])
@pytest.mark.parametrize("size", [(24, 16, 16), (32, 17, 15), (48, 32, 33), (64, 24, 40)])
def test_stretched_fp64_agrees_with_per_cell_kernels(nb, size, groups):
    """The stretched FP64 sweeps of the colour-split layout against the per-cell kernels. Both solve to 1e-12, so the
    pressures agree within 2 cond(A) 1e-12, with cond(A) from the assembled matrix's extreme eigenvalues."""
    import scipy.sparse as sp
    import scipy.sparse.linalg as sl

    case = W.stretched_cylinder_3d(*size)
    types = capi.label_cells(case.grid, case.scene)
    a, b = [solve_family(case, types, family, "fp64", False, x_groups=groups) for family in (2, 0)]
    s = PressureSolver("fp64")
    s.InitializePressureSolver(b)
    rowptr, col, val, _ = s.ExportMatrix()
    s.DestroyPressureSolver()
    A = -sp.csr_matrix((val, col, rowptr))
    top = sl.eigsh(A, k=1, which="LA", return_eigenvectors=False, tol=1e-3)[0]
    low = sl.eigsh(A.tocsc(), k=1, sigma=0.0, return_eigenvectors=False)[0]
    bar = 2.0 * top / low * 1e-12
    idp = types.reshape(-1) == W.FLUID
    assert np.linalg.norm((a.p - b.p)[idp]) <= bar * np.linalg.norm(b.p[idp])


# 2D: (interior x, y) around the 32 x 16 cells a block of the legs owns; one level above the coarse end and several
@pytest.mark.parametrize("sweeps", [1, 2, 3])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("size", [(20, 20), (31, 33), (32, 48), (33, 65), (64, 50), (97, 80)])
def test_2d_legs_agree_with_per_cell_kernels(nb, size, precision, sweeps):
    """2D levels with a launch per leg (pair_kernels = 2 and up to two sweeps) against a launch per operation, closed and
    with an outlet, all to 1e-12 (the bar of test_fp64_split_agrees_with_per_cell_kernels)."""
    nx, ny = size
    h = 1.0 / min(size)
    g = W.uniform_grid(2, (0.0, nx * h, 0.0, ny * h, 0.0, 1.0), min(size))
    assert (g.Nx, g.Ny) == (nx + 2, ny + 2)
    disc = W.Region(W.REGION_SOLID, W.PRIM_CYLINDER, (0.4 * nx * h, 0.5 * ny * h, 0.0), radius=0.2)
    for closed in (False, True):
        case = W.Case("disc", g, W.walls_scene(2, outlet_face=None if closed else 1, regions=[disc]), 37,
                      needs_compat=closed)
        types = capi.label_cells(g, case.scene)
        a, b = [solve_family(case, types, family, precision, closed, pre_sweeps=sweeps, post_sweeps=sweeps,
                             tail_cells=128) for family in (2, 0)]
        bar = 1e-11 * max(size) ** 2
        for x, y in ((a.p, b.p), (a.u, b.u), (a.v, b.v)):
            assert np.linalg.norm(x - y) <= bar * np.linalg.norm(y)


@pytest.mark.parametrize("sweeps", [1, 2, 3])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("size", [(40, 24), (65, 33)])
def test_2d_stretched_legs_agree_with_per_cell_kernels(nb, size, precision, sweeps):
    """The same on the stretched channel; each solution within cond(A) 1e-11 of the exact one."""
    import scipy.sparse as sp
    import scipy.sparse.linalg as sl

    case = W.channel_2d_stretched(*size)
    types = capi.label_cells(case.grid, case.scene)
    a, b = [solve_family(case, types, family, precision, False, tol=1e-11, stretched_sweeps=sweeps, tail_cells=128)
            for family in (2, 0)]
    s = PressureSolver("fp64")
    s.InitializePressureSolver(b)
    rowptr, col, val, _ = s.ExportMatrix()
    s.DestroyPressureSolver()
    A = -sp.csr_matrix((val, col, rowptr))
    top = sl.eigsh(A, k=1, which="LA", return_eigenvectors=False, tol=1e-3)[0]
    low = sl.eigsh(A.tocsc(), k=1, sigma=0.0, return_eigenvectors=False)[0]
    assert np.linalg.norm(a.p - b.p) <= 2.0 * top / low * 1e-11 * np.linalg.norm(b.p)


@pytest.mark.parametrize("shape", [(3, 3, 3), (5, 4, 7), (9, 12, 6), (2, 5, 4), (5, 2, 4), (6, 5, 2), (7, 6, 1), (3, 2, 1)])
def test_pressure_ring_replay(nb, shape):
    """EnforcePressureBC's passes (y, x, then z faces; EMPTY 0, PRESSURE kept, any other ring cell copies inward) on
    random ring labels: on a grid without unknowns the step only replays the ring. Exact; the last shapes have sides
    without interior cells."""
    Ny, Nx, Nz = shape
    dim = 2 if Nz == 1 else 3
    rng = np.random.default_rng(Ny * 100 + Nx * 10 + Nz)
    axis = lambda n: W.Axis(np.full(n, 0.1), 0.1 * np.arange(n + 1), 0.1 * np.arange(n) + 0.05)
    g = W.Grid(dim, [axis(Nx), axis(Ny), axis(Nz)], 0.1, False, (0.0, 1.0) * 3)
    types = rng.choice([W.SOLID, W.EMPTY, W.INFLOW, W.PRESSURE, W.OUTFLOW], size=shape).astype(np.uint8)
    p = rng.standard_normal(shape)
    expect = p.copy()
    for _ in range(2):  # at the start of the step and after the (empty) solve
        for ax in range(dim if dim == 2 else 3):
            n = shape[ax]
            for at, src in ((0, 1), (n - 1, n - 2)):
                t, d, s = types.take(at, ax), expect.take(at, ax), expect.take(src, ax)
                face = np.where(t == W.EMPTY, 0.0, np.where(t == W.PRESSURE, d, s))
                expect[tuple(at if a == ax else slice(None) for a in range(3))] = face
    zeros = lambda s: np.zeros(int(np.prod(s)))
    m = MACGrid(g, types.reshape(-1).copy(), zeros(g.u_shape()), zeros(g.v_shape()), zeros(g.w_shape()),
                p.reshape(-1).copy(), 1.0, 1e-3)
    s = PressureSolver("mixed")
    s.InitializePressureSolver(m)
    assert s.SystemSize() == 0
    s.SolvePressure(m, tol=1e-8)
    s.DestroyPressureSolver()
    assert np.array_equal(m.p.reshape(shape), expect)


# (interior x, y, z): Nz odd and even, both with rows that the colour-split layout pads
@pytest.mark.parametrize("sweeps", [1, 2])
@pytest.mark.parametrize("form", ["mixed_odd", "mixed_even", "fp64_odd", "fp64_even", "fp64_stretched"])
def test_an_overflowed_solve_leaves_nothing_behind(nb, form, sweeps):
    """A step whose solve overflows (NOT_CONVERGED, no finite pressure), then an ordinary one on the same solver: what a
    fresh solver gives, bit for bit. The mixed form overflows in FP32 from velocities of 1e60. The FP64 form's products
    have to pass 1.8e308 where |b|^2 stays below: on cells of 1e6 the solver's units scale b by 1e12; on the stretched
    grid of thin cells r.z is above r.r (an eigenvalue of the operator is at most twice its diagonal, here below 0.4)."""
    precision, shape = form.split("_")
    dh = 1.0 if precision == "mixed" else 1e6
    if shape == "stretched":
        case = W.stretched_cylinder_3d(24, 16, 17)
    else:
        n = (20, 18, 17 if shape == "odd" else 18)
        g = W.uniform_grid(3, (0.0, n[0] * dh, 0.0, n[1] * dh, 0.0, n[2] * dh), 18)
        assert (g.Nx, g.Ny, g.Nz) == (n[0] + 2, n[1] + 2, n[2] + 2)
        case = W.Case("box", g, W.walls_scene(3, outlet_face=1), 41)
    g, types = case.grid, capi.label_cells(case.grid, case.scene)
    assert 2 * ((((g.Nz + 1) // 2) + 3) // 4 * 4) >= g.Nz + 2
    u, v, w = W.face_velocities(g, types, case.seed)

    def step(s, scale):
        m = MACGrid(g, types.copy(), scale * u, scale * v, scale * w, np.zeros(g.cells), case.rho, case.dt)
        return s.SolvePressure(m, tol=1e-9), m

    options = dict(pre_sweeps=sweeps, post_sweeps=sweeps, stretched_sweeps=sweeps)
    fresh = PressureSolver(precision, **options)
    r0, m0 = step(fresh, 1.0)
    assert r0.status == capi.NB_OK and r0.levels >= 2
    fresh.DestroyPressureSolver()
    s = PressureSolver(precision, **options)
    big = 1e60 if precision == "mixed" else (1.2e154 if shape == "stretched" else 1e147) / r0.b_norm
    for _ in range(2):
        r, m = step(s, big)
        assert r.status == capi.NB_NOT_CONVERGED and np.isfinite(r.b_norm) and not np.all(np.isfinite(m.p))
        for _ in range(2):
            r, m = step(s, 1.0)
            assert (r.status, r.iters_inner, r.rel_res) == (r0.status, r0.iters_inner, r0.rel_res)
            for a, b in ((m.p, m0.p), (m.u, m0.u), (m.v, m0.v), (m.w, m0.w)):
                assert np.array_equal(a, b)
    s.DestroyPressureSolver()
