"""The single-block coarse end (nb_tail.cu) against the same levels run by their own launches (tail_cells = 0): the same
V-cycle up to rounding, so both solves meet the tolerance and agree to it."""
import numpy as np
import pytest

from nereus_cfd_b200 import capi, workloads as W
from nereus_cfd_b200.pressure import MACGrid, PressureSolver

pytestmark = pytest.mark.gpu


def solve(case, precision, tail_cells, tol):
    g = case.grid
    types = capi.label_cells(g, case.scene)
    u, v, w = W.face_velocities(g, types, case.seed)
    m = MACGrid(g, types, u, v, w, np.zeros(g.cells), case.rho, case.dt)
    s = PressureSolver(precision, tail_cells=tail_cells)
    r = s.SolvePressure(m, tol=tol, needs_compat=case.needs_compat)
    assert r.status == capi.NB_OK and r.rel_res <= tol, r.as_dict()
    s.DestroyPressureSolver()
    return m.p


CASES = {"box_2d": lambda: W.closed_box_2d(67), "outlet_2d": lambda: W.cavity_outlet_2d(64),
         "channel_2d": lambda: W.channel_2d_stretched(48, 24), "sphere_3d": lambda: W.sphere_outlet_3d(35),
         "cylinder_3d": lambda: W.stretched_cylinder_3d(48, 20, 20)}


# 64: the coarsest level alone, although it has more cells; 256: warp-sized levels; 2048 (the default) and 5000: up to,
# and more than, an unknown of each colour per thread
@pytest.mark.parametrize("tail_cells", [64, 256, 2048, 5000])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_tail_agrees_with_its_levels_own_launches(nb, name, precision, tail_cells):
    """Both solutions are within cond * tol of the exact one. With tol = 1e-11 and cond <= 5 N^2 on the uniform grids
    (N <= 67 cells along a side, the lowest mode a quarter wave) that is 2.3e-7 each; the channels' cells grow 1.04 per
    cell over a length of five heights, N = 48 and cond below 50 N^2: 1.2e-6."""
    case = CASES[name]()
    a, b = solve(case, precision, tail_cells, 1e-11), solve(case, precision, 0, 1e-11)
    bar = 2.4e-6 if "channel" in name or "cylinder" in name else 4.6e-7
    assert np.linalg.norm(a - b) <= bar * np.linalg.norm(b)
