"""The FP64 x-line sweeps (momentum, temperature and scalar solves on boxes
whose cells run x-fastest) against the CPU oracle, whose solves are BiCGStab:
line lengths at the edges of the 32-cell scan chunks, meshes of a few lines,
handles that renumber their cells, and flows across the lines: slow sweeps, and
with a long time step ones too slow to go on with, where BiCGStab takes over.

Solves run to 1e-12 on both sides; fields agree to 1e-9 of their maximum, the
parity gate of the other whole-pass tests (the transient term bounds the
matrices' condition, so 1e-12 residuals leave errors far below it).
"""
import numpy as np
import pytest

from checkers import SIMPLE, Oracle, noisy_initial_fields, oracle_mesh, oracle_params
from minicombust_app_b200 import flow

pytestmark = pytest.mark.gpu

BASE = {"U": 50.0, "V": 0.0, "W": 0.0, "P": 4000.0, "TEM": 1500.0}


def run_both(dims, passes=2, base=BASE, counts=None, **kw):
    lengths = (0.2, 0.1, 0.1)
    p = flow.default_params(flow.MODE_SIMPLE, **{"u_rtol": 1e-12, "p_rtol": 1e-12, **kw})
    solver = flow.FlowSolver(flow.Mesh.box(*dims, *lengths), params=p)
    okw = {"u_rtol": 1e-12, "p_rtol": 1e-12}
    okw.update({k: kw[k] for k in ("delta", "urf_momentum") if k in kw})
    orc = Oracle(oracle_mesh(*dims, *lengths), oracle_params(SIMPLE, scalars=p.transport_scalars, **okw))
    for name, vals in noisy_initial_fields(solver.N, base, 1).items():
        for s in (solver, orc):
            a = s.field(name)
            a[:solver.N] = vals
            s.set_field(name, a)
    solver.set_timing(counts is not None)
    for _ in range(passes):
        solver.simple_iteration()
        orc.step()
    if counts is not None:
        counts.update({k: n for k, (_, n) in solver.kernel_times().items()})
    for name in BASE:
        a, b = solver.field(name), orc.field(name)
        assert np.abs(a - b).max() <= 1e-9 * np.abs(b).max(), (dims, name)
    st = solver.last_stats
    solver.close()
    return st


@pytest.mark.parametrize("dims", [(2, 3, 3), (31, 3, 2), (32, 2, 5), (33, 5, 3), (257, 2, 2), (513, 2, 2),
                                  (1024, 2, 2)])
def test_sweeps_match_oracle(gpu, dims):
    st = run_both(dims)
    # a sweep gains about three decades on this flow: 1e-12 within one batch
    assert 1 <= max(st.momentum_iters) <= 12 and 1 <= st.temperature_iters <= 12


@pytest.mark.parametrize("dims", [(2, 1, 1), (33, 1, 1), (1000, 1, 1), (1, 33, 1)])
@pytest.mark.parametrize("reorder", [0, 1], ids=["natural", "rcm"])
def test_single_lines_match_oracle(gpu, dims, reorder):
    """A mesh of one line: renumbering reverses it, so that its rows are stored
    by direction although the handle's own order has no x-lines."""
    run_both(dims, reorder=reorder, transport_scalars=1)


@pytest.mark.parametrize("dims", [(2, 3, 3), (32, 2, 5), (33, 5, 3), (257, 2, 2), (18, 17, 9)])
def test_renumbered_sweeps_match_oracle(gpu, dims):
    st = run_both(dims, reorder=1, transport_scalars=1)
    assert 1 <= max(st.momentum_iters) <= 12 and 1 <= st.temperature_iters <= 12


def test_scalars_by_sweeps_match_oracle(gpu):
    run_both((33, 6, 5), transport_scalars=1)


@pytest.mark.parametrize("precision", [flow.PRECISION_FP64, flow.PRECISION_FP32_REFINED], ids=["fp64", "refined"])
@pytest.mark.parametrize("urf", [0.7, 1.0])
def test_slow_sweeps_are_kept(gpu, precision, urf):
    """A sweep takes off less than half of the residual here, the first ones a tenth,
    and some 60 sweeps still cost a fraction of BiCGStab's iterations."""
    n = {}
    st = run_both((24, 32, 16), passes=1, base={**BASE, "U": 1.0, "V": 80.0}, delta=1e-3, counts=n,
                  pressure_solver=flow.PSOLVER_PCG_AMG, precision=precision, urf_momentum=urf)
    assert max(st.momentum_iters) > 20 and st.temperature_iters > 20
    assert n["line_sweep3_64"] >= max(st.momentum_iters) and n["line_sweep1_64"] >= st.temperature_iters
    assert all(n[k] == 0 for k in n if k.startswith("bicg"))


def test_refined_sweeps_whatever_max_iters(gpu):
    """With FP32 refinement max_iters bounds the inner solves, not the sweeps."""
    n = {}
    st = run_both((24, 12, 10), counts=n, max_iters=20, pressure_solver=flow.PSOLVER_PCG_AMG,
                  precision=flow.PRECISION_FP32_REFINED)
    assert n["line_sweep3_64"] > 0 and n["line_sweep1_64"] > 0
    assert all(n[k] == 0 for k in n if k.startswith("bicg"))
    assert 1 <= max(st.momentum_iters) <= 12 and 1 <= st.temperature_iters <= 12


def test_sweeps_within_max_iters(gpu):
    """A temperature solve that needs some 200 sweeps or iterations, bounded at 100."""
    s = flow.FlowSolver(flow.Mesh.box(24, 32, 16, 0.2, 0.1, 0.1),
                        params=flow.default_params(flow.MODE_SIMPLE, delta=1e-2, max_iters=100,
                                                   pressure_solver=flow.PSOLVER_PCG_AMG))
    for name, vals in noisy_initial_fields(s.N, {**BASE, "U": 1.0, "V": 80.0}, 1).items():
        a = s.field(name)
        a[:s.N] = vals
        s.set_field(name, a)
    s.set_timing(True)
    assert s.simple_iteration(check=False) == flow.MC_ERR_NOT_CONVERGED
    assert 0 < s.kernel_times()["line_sweep1_64"][1] <= 100 and s.last_stats.temperature_iters <= 100
    assert max(s.last_stats.momentum_iters) <= 100
    s.close()


def test_long_step_cross_flow_matches_oracle(gpu):
    run_both((12, 24, 6), passes=1, base={**BASE, "U": 1.0, "V": 80.0}, delta=1e-2)


def test_stalled_sweeps_fall_back_to_bicgstab(gpu):
    """The sweeps' true residual cannot reach 1e-17 ||b||, the recursive one of
    BiCGStab can: the stall is seen within three batches."""
    n = {}
    run_both((12, 24, 6), passes=1, counts=n, u_rtol=1e-17)
    assert n["bicg3_init"] == 1 and n["bicg1_team"] == 1
    assert 0 < n["line_sweep3_64"] <= 18 and 0 < n["line_sweep1_64"] <= 18
