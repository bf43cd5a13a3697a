"""The corrections without the non-orthogonal flux correction (meshes whose
cell centres all lie on their faces' normal lines, found at creation) and the
short form of a face's unit normal, against the CPU oracle, which always
evaluates the general expressions: an axis-aligned box takes the short forms, a
box with displaced cell centres the general ones."""
import numpy as np
import pytest

from checkers import SIMPLE, Oracle, noisy_initial_fields, oracle_mesh, oracle_params
from minicombust_app_b200 import flow

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("psolver", [flow.PSOLVER_PCG_JACOBI, flow.PSOLVER_PCG_AMG], ids=["jacobi", "amg"])
@pytest.mark.parametrize("reorder", [flow.REORDER_NONE, flow.REORDER_RCM], ids=["natural", "rcm"])
def test_box_matches_oracle(gpu, psolver, reorder):
    dims, lengths = (14, 9, 7), (2.0, 1.3, 0.9)  # rounding of these coordinates reaches the 3e-16 threshold
    p = flow.default_params(flow.MODE_SIMPLE, u_rtol=1e-13, p_rtol=1e-13, pressure_solver=psolver, reorder=reorder)
    s = flow.FlowSolver(flow.Mesh.box(*dims, *lengths), params=p)
    o = Oracle(oracle_mesh(*dims, *lengths), oracle_params(SIMPLE, u_rtol=1e-13, p_rtol=1e-13))
    for name, vals in noisy_initial_fields(s.N, {"U": 50.0, "V": 0.0, "W": 0.0, "P": 4000.0, "TEM": 1500.0}, 2).items():
        for h in (s, o):
            a = h.field(name)
            a[:s.N] = vals
            h.set_field(name, a)
    for _ in range(3):
        s.simple_iteration()
        o.step()
    for name in ("U", "V", "W", "P", "TEM"):
        a, b = s.field(name), o.field(name)
        assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max(), name


@pytest.mark.parametrize("psolver", [flow.PSOLVER_PCG_JACOBI, flow.PSOLVER_PCG_AMG], ids=["jacobi", "amg"])
@pytest.mark.parametrize("reorder", [flow.REORDER_NONE, flow.REORDER_RCM], ids=["natural", "rcm"])
def test_displaced_centres_match_oracle(gpu, psolver, reorder):
    """Displaced centres make the flux correction non-zero, so a second corrector
    has a right-hand side: fields against the oracle, and the box, whose
    second corrector has none, beside it."""
    dims, lengths = (12, 8, 8), (0.2, 0.1, 0.1)
    shift = np.random.default_rng(0).uniform(-1, 1, (12 * 8 * 8, 3)) * 5e-4
    for displaced in (True, False):
        mesh, om = flow.Mesh.box(*dims, *lengths), oracle_mesh(*dims, *lengths)
        if displaced:
            mesh.cell_centers += shift
            om.cell_centers += shift
        s = flow.FlowSolver(mesh, params=flow.default_params(flow.MODE_SIMPLE, pressure_solver=psolver, reorder=reorder,
                                                             u_rtol=1e-13, p_rtol=1e-13))
        o = Oracle(om, oracle_params(SIMPLE, u_rtol=1e-13, p_rtol=1e-13))
        for name, vals in noisy_initial_fields(s.N, {"U": 50.0, "V": 0.0, "W": 0.0, "P": 4000.0, "TEM": 1500.0},
                                               3).items():
            for h in (s, o):
                a = h.field(name)
                a[:s.N] = vals
                h.set_field(name, a)
        for _ in range(3):
            s.simple_iteration()
            o.step()
            assert (s.last_stats.pressure_iters_total > s.last_stats.pressure_iters_first) == displaced
        for name in ("U", "V", "W", "P", "TEM"):
            a, b = s.field(name), o.field(name)
            assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max(), (displaced, name)
        s.close()


@pytest.mark.parametrize("cell", [0, -1], ids=["first", "last"])
def test_one_displaced_centre_is_found(gpu, cell):
    """The check at creation sees every cell, the last ones uploaded too."""
    mesh = flow.Mesh.box(96, 40, 40, 0.2, 0.1, 0.1)
    mesh.cell_centers[cell] += 2e-4
    for _ in range(3):
        s = flow.FlowSolver(mesh, params=flow.default_params(flow.MODE_SIMPLE, pressure_solver=flow.PSOLVER_PCG_AMG,
                                                             p_rtol=1e-12))
        for name, vals in noisy_initial_fields(s.N, {"U": 50.0, "V": 0.0, "W": 0.0, "P": 4000.0, "TEM": 1500.0},
                                               3).items():
            a = s.field(name)
            a[:s.N] = vals
            s.set_field(name, a)
        s.simple_iteration()
        assert s.last_stats.pressure_iters_total > s.last_stats.pressure_iters_first
        s.close()
