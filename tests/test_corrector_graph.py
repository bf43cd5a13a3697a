"""The first pressure corrector of a pass as one device graph: bit for bit the
host-driven pass, and what it reports and leaves behind when a solve in it, or
the guess before it, breaks down."""
import os
import subprocess
import sys

import numpy as np
import pytest

from minicombust_app_b200 import flow
from minicombust_app_b200.workload import noisy_fields

pytestmark = pytest.mark.gpu


ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def pressure_status(scale):
    """Status of the pressure stage of a pass with velocities of 50 x scale; a
    stage that reports a non-finite solve has corrected nothing."""
    s = flow.FlowSolver(flow.Mesh.box(16, 12, 8, 0.2, 0.1, 0.1),
                        params=flow.default_params(flow.MODE_SIMPLE, pressure_solver=flow.PSOLVER_PCG_AMG,
                                                   precision=flow.PRECISION_FP32_REFINED))
    for name, vals in noisy_fields(s.N, seed=3).items():
        a = s.field(name)
        a[:s.N] = vals * (scale if name in "UVW" else 1.0)
        s.set_field(name, a)
    s.stage("gradients")
    s.stage("momentum")
    before = {n: s.field(n)[:s.N] for n in ("U", "V", "W", "P")}
    status = flow.MC_OK
    try:
        s.stage("pressure")
    except flow.FlowError as e:
        status = e.status
    same = all(np.array_equal(s.field(n)[:s.N], a) for n, a in before.items())
    assert same == (status == flow.MC_ERR_NONFINITE)
    s.close()
    return status


def test_inner_fp32_breakdown_is_reported(gpu):
    """Velocities whose flow imbalance exceeds FP32's range (but not FP64's) break
    the inner FP32 solve down while the FP64 refinement around it stays finite."""
    assert pressure_status(1.0) == flow.MC_OK
    assert pressure_status(1e45) == flow.MC_ERR_NONFINITE


PASSES = r"""
import os, sys
sys.path.insert(0, os.environ["MC_ROOT"])
import numpy as np
from minicombust_app_b200 import flow, train_guess
from minicombust_app_b200.workload import noisy_fields
out = {}
for precision in (flow.PRECISION_FP64, flow.PRECISION_FP32_REFINED):
    for guess in (flow.GUESS_ZERO, flow.GUESS_PREVIOUS, flow.GUESS_LEARNED):
        for displaced in (0, 1):
            mesh = flow.Mesh.box(20, 12, 11, 0.2, 0.1, 0.1)
            if displaced:  # a second corrector with a right-hand side
                mesh.cell_centers += np.random.default_rng(0).uniform(-1, 1, mesh.cell_centers.shape) * 5e-4
            s = flow.FlowSolver(mesh, params=flow.default_params(
                flow.MODE_SIMPLE, pressure_solver=flow.PSOLVER_PCG_AMG, precision=precision, initial_guess=guess))
            if guess == flow.GUESS_LEARNED:
                s.set_guess_params(train_guess.load_params())
            for name, vals in noisy_fields(s.N, seed=3).items():
                a = s.field(name)
                a[:s.N] = vals
                s.set_field(name, a)
            for _ in range(4):
                s.simple_iteration()
                st = s.last_stats.as_dict()
            key = f"{precision}_{guess}_{displaced}_"
            for n in ("U", "V", "W", "P", "TEM"):
                out[key + n] = s.field(n)
            for n in ("pressure_solves", "pressure_iters_total", "pressure_iters_first"):
                out[key + n] = np.array(st[n])
            s.close()
np.savez(sys.argv[1], **out)
"""


def test_graph_and_host_driven_passes_agree_bit_for_bit(gpu, tmp_path):
    out = []
    for loops in ("1", "0"):
        path = str(tmp_path / f"loops{loops}.npz")
        env = dict(os.environ, MC_ROOT=ROOT, MC_LOOP_GRAPHS=loops)
        r = subprocess.run([sys.executable, "-c", PASSES, path], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, loops + r.stdout + r.stderr
        out.append(np.load(path))
    assert len(out[0].files) == 96
    for k in out[0].files:
        assert np.array_equal(out[0][k], out[1][k]), k


CHILD = r"""
import os, sys
sys.path.insert(0, os.environ["MC_ROOT"])
import numpy as np
from minicombust_app_b200 import flow, train_guess
for precision in (flow.PRECISION_FP64, flow.PRECISION_FP32_REFINED):
    s = train_guess.make_solver(16, 3, guess=flow.GUESS_LEARNED, precision=precision, params=train_guess.load_params())
    assert s.simple_iteration() == flow.MC_OK
    os.environ["MC_GNN_WAIT_POLLS"] = "0"
    s.stage("gradients")
    s.stage("momentum")
    before = {n: s.field(n)[:s.N] for n in ("U", "V", "W", "P")}
    try:
        s.stage("pressure")
        raise SystemExit("no error")
    except flow.FlowError as e:
        assert e.status == flow.MC_ERR_TIMEOUT, e
    del os.environ["MC_GNN_WAIT_POLLS"]
    for n, a in before.items():
        assert np.array_equal(s.field(n)[:s.N], a), n
    assert s.simple_iteration() == flow.MC_OK
    s.close()
print("uncorrected ok")
"""


def test_failed_guess_leaves_the_fields_uncorrected(gpu):
    """A learned guess whose layer kernel gave up is an error of the pressure stage
    found before its corrections, on the graph as on the host-driven path."""
    for loops in ("1", "0"):
        env = dict(os.environ, MC_ROOT=ROOT, MC_GNN_LAYER="umma", MC_LOOP_GRAPHS=loops)
        env.pop("MC_GNN_WAIT_POLLS", None)
        r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, loops + r.stdout + r.stderr
        assert "uncorrected ok" in r.stdout
