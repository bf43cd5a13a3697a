"""V-cycle halves as one kernel per level (MC_AMG_TILES=2: every box level of the
hierarchy) against the per-sweep kernels (0): the same operator in another
order of evaluation.  Boxes at the edges of the tiles (26 x 10 cells, even plane
counts) and of the levels' halving: one cell over or under, odd sizes, two cells.

The pressure solve stops at 1e-2 of its right-hand side, so a V-cycle that
differed anywhere would change the fields by about 1e-2 of the correction: more
than 1e-5 of the pressure here.  Rounding leaves 1e-9 of each field (FP64) and,
with the FP32 V-cycle inside, 1e-6.
"""
import os

import numpy as np
import pytest

from minicombust_app_b200 import flow
from minicombust_app_b200.workload import noisy_fields

pytestmark = pytest.mark.gpu

FIELDS = ("U", "V", "W", "P", "TEM")


def run(dims, tiles, **kw):
    saved = os.environ.get("MC_AMG_TILES"), os.environ.get("MC_AMG_HALF")
    os.environ.update(MC_AMG_TILES=tiles, MC_AMG_HALF="0")
    try:
        s = flow.FlowSolver(flow.Mesh.box(*dims, 0.2, 0.1, 0.1),
                            params=flow.default_params(flow.MODE_SIMPLE, pressure_solver=flow.PSOLVER_PCG_AMG,
                                                       p_rtol=1e-2, **kw))
    finally:
        for k, v in zip(("MC_AMG_TILES", "MC_AMG_HALF"), saved):
            os.environ.pop(k, None) if v is None else os.environ.update({k: v})
    for name, vals in noisy_fields(s.N, seed=3).items():
        a = s.field(name)
        a[:s.N] = vals
        s.set_field(name, a)
    its, before = [], s.launch_count()
    for _ in range(2):
        s.simple_iteration()
        its.append(s.last_stats.as_dict()["pressure_iters_total"])
    launches = s.launch_count() - before
    fields = {n: s.field(n) for n in FIELDS}
    s.close()
    return fields, its, launches


@pytest.mark.parametrize("dims", [(26, 10, 8), (27, 11, 7), (52, 20, 9), (53, 21, 33), (25, 9, 31), (2, 30, 40),
                                  (104, 2, 20), (40, 40, 2), (40, 41, 3), (79, 31, 65)])
@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32"])
def test_tiles_match_sweeps(gpu, dims, fp32):
    kw = dict(precision=flow.PRECISION_FP32_REFINED) if fp32 else {}
    tiles, its_t, n_t = run(dims, "2", **kw)
    sweeps, its_s, n_s = run(dims, "0", **kw)
    assert its_t == its_s
    # two kernels a level instead of six (FP32, paired sweeps) or eight; a
    # small box may have no level above the single-block ones
    assert n_t <= n_s and (n_t < n_s or np.prod(dims) < 8192)
    for n in FIELDS:
        rel = np.abs(tiles[n] - sweeps[n]).max() / np.abs(sweeps[n]).max()
        assert rel <= (1e-6 if fp32 else 1e-9), (n, rel)


def test_rule_takes_tiles_at_a_large_box(gpu):
    """At 256 x 128 x 128 the default rule tiles levels 0 and 1: two kernels instead
    of eight on each, in every V-cycle (one per iteration and one before the first)."""
    rule, its_r, n_r = run((256, 128, 128), "1")
    sweeps, its_s, n_s = run((256, 128, 128), "0")
    assert its_r == its_s
    assert n_s - n_r >= sum(2 * 6 * (n + 1) for n in its_r)
    for n in FIELDS:
        assert np.abs(rule[n] - sweeps[n]).max() <= 1e-9 * np.abs(sweeps[n]).max(), n


@pytest.mark.parametrize("dims,tiled", [((128, 64, 64), True), ((80, 116, 141), False), ((200, 101, 97), False)])
def test_rule_by_steps_per_row_and_size(gpu, dims, tiled):
    """FP64: up to 2.9 cell steps per row, up to 3.35 below 650,000 cells (here 3.32,
    3.19 and 3.13, the last two slower with tiles)."""
    _, its, n_rule = run(dims, "1")
    _, _, n_sweeps = run(dims, "0")
    assert (n_sweeps - n_rule >= sum(6 * (n + 1) for n in its)) if tiled else n_rule == n_sweeps
