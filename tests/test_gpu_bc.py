"""The boundary-condition replay on the B200 (nereus_b200_bc_*) against the reference's own EnforceVelocityBC and
EnforcePressureBC (tests/golden/bc_*.npz: the lists its MAC::BuildBoundaryLists made, the values its boundary
functions gave, and the fields before and after): bit for bit, ApplyOutflowFlux included; without boundary
functions against the oracle's replay; and replayed from a CUDA graph."""
import numpy as np
import pytest

from conftest import bc_golden_names, load_golden
from nereus_cfd_b200.boundary import BoundaryReplay
from oracle import cpu

pytestmark = pytest.mark.gpu
NAMES = bc_golden_names()


def _setup(name):
    import torch

    case, meta, z = load_golden(name)
    g = case.grid
    nz = g.Nz if g.dim == 3 else 1
    bc = BoundaryReplay(dict(z), g.dim, g.Nx, g.Ny, nz)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to("cuda")
    fields = [d(z["u_in"]), d(z["v_in"]), d(z["w_in"]) if g.dim == 3 else None, d(z["p_in"])]
    return case, z, bc, fields, d


def _host(fields):
    return [f.cpu().numpy() if f is not None else np.zeros(0) for f in fields]


@pytest.mark.parametrize("name", NAMES)
def test_replay_matches_reference(nb, name):
    import torch

    case, z, bc, (u, v, w, p), d = _setup(name)
    bc.EnforceVelocityBC(u, v, w, d(z["presc_value"]) if len(z["presc_value"]) else None)
    bc.EnforcePressureBC(p, d(z["ring_value"]) if len(z["ring_value"]) else None)
    torch.cuda.synchronize()
    hu, hv, hw, hp = _host([u, v, w, p])
    assert np.array_equal(hu, z["u_out"])
    assert np.array_equal(hv, z["v_out"])
    assert np.array_equal(hw, z["w_out"])
    assert np.array_equal(hp, z["p_out"])
    lv, lp = bc.levels()
    assert 1 <= lv <= 16 and 1 <= lp <= 16
    bc.close()


@pytest.mark.parametrize("name", NAMES)
def test_replay_without_boundary_functions_matches_oracle(nb, name):
    """No boundary velocity function: the prescribed entries stay unwritten; no pressure function: 0 there."""
    import torch

    case, z, bc, (u, v, w, p), d = _setup(name)
    bc.EnforceVelocityBC(u, v, w, None)
    bc.EnforcePressureBC(p, None)
    torch.cuda.synchronize()
    lists = dict(z)
    lists["ring_value"] = np.zeros_like(z["ring_value"])
    ru, rv, rw, rp = cpu.bc_replay(lists, z["u_in"], z["v_in"], z["w_in"], z["p_in"], with_velocity_function=False)
    hu, hv, hw, hp = _host([u, v, w, p])
    assert np.array_equal(hu, ru) and np.array_equal(hv, rv) and np.array_equal(hp, rp)
    assert np.array_equal(hw, rw)
    bc.close()


def test_replay_in_a_cuda_graph(nb):
    import torch

    name = [n for n in NAMES if "channel" in n][0]
    case, z, bc, (u, v, w, p), d = _setup(name)
    pv, rv = d(z["presc_value"]), d(z["ring_value"])
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        bc.EnforceVelocityBC(u, v, w, pv, stream=s)
        bc.EnforcePressureBC(p, rv, stream=s)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        bc.EnforceVelocityBC(u, v, w, pv, stream=s)
        bc.EnforcePressureBC(p, rv, stream=s)
    rng = np.random.default_rng(5)
    for _ in range(2):
        ins = [rng.normal(size=len(z[k])) for k in ("u_in", "v_in", "w_in", "p_in")]
        for t, a in zip((u, v, w, p), ins):
            t.copy_(torch.from_numpy(a))
        graph.replay()
        torch.cuda.synchronize()
        ref = cpu.bc_replay(dict(z), *ins)
        for got, want in zip(_host([u, v, w, p]), ref):
            assert np.array_equal(got, want)
    del graph
    bc.close()


def random_lists(seed, n=7, dense=False):
    """Lists on an n^3 grid that no scene would make: repeated destinations, chains of copies, sources written before and
    after they are read (dense: most programs then do not resolve into independent writes), rows and single entries."""
    rng = np.random.default_rng(seed)
    sizes = [n * n * (n + 1)] * 3
    pick = lambda size, count: rng.integers(0, size, count)
    z = {}
    for c in range(3):
        z["solid%d" % c] = np.concatenate([np.arange(5, 5 + rng.integers(1, 300)), pick(sizes[c], 20)]) % sizes[c]
    m = 400 if dense else 60
    comp = np.sort(rng.integers(0, 3, m))
    z["presc_comp"], z["presc_index"] = comp, pick(sizes[0], m)
    z["presc_value"] = rng.normal(size=m)
    comp = np.repeat(np.arange(3), m)
    z["copy_comp"] = comp
    if dense:
        z["copy_dst"], z["copy_src"] = pick(sizes[0], 3 * m), pick(sizes[0], 3 * m)
    else:  # from a block no copy writes, or along a chain of entries copied just before
        z["copy_dst"] = np.tile(np.arange(100, 100 + m), 3)
        z["copy_src"] = np.where(rng.random(3 * m) < 0.5, 300 + pick(40, 3 * m), np.maximum(z["copy_dst"] - 1, 100))
        z["copy_src"][::m] = 350
    r = 500 if dense else 120
    z["ring_dst"] = pick(n ** 3, r) if dense else np.arange(0, 2 * r, 2)
    z["ring_kind"], z["ring_value"] = rng.integers(0, 3, r), rng.normal(size=r)
    z["ring_src"] = pick(n ** 3, r) if dense else 2 * pick(60, r) + 1
    for k in ("inlet_comp", "inlet_index", "inlet_area", "inlet_sign", "outflow_comp", "outflow_index", "outflow_outer",
              "outflow_area", "outflow_sign"):
        z[k] = np.zeros(0)
    return z


@pytest.mark.parametrize("values", [True, False])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("seed", range(6))
def test_random_programs_match_the_serial_replay(nb, seed, dense, values):
    import torch

    n = 7
    z = random_lists(seed, n, dense)
    rng = np.random.default_rng(100 + seed)
    ins = [rng.normal(size=n * n * (n + 1)) for _ in range(3)] + [rng.normal(size=n ** 3)]
    bc = BoundaryReplay(z, 3, n, n, n)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to("cuda")
    fields = [d(a) for a in ins]
    bc.EnforceVelocityBC(*fields[:3], d(z["presc_value"]) if values else None)
    bc.EnforcePressureBC(fields[3], d(z["ring_value"]) if values else None)
    torch.cuda.synchronize()
    lists = dict(z)
    if not values:
        lists["ring_value"] = np.zeros_like(z["ring_value"])
    ref = cpu.bc_replay(lists, *ins, with_velocity_function=values)
    for got, want in zip(_host(fields), ref):
        assert np.array_equal(got, want)
    bc.close()
