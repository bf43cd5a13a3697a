"""Krylov solves run as one kernel by a team of blocks (cluster up to 16 x 1024
rows, then a cooperative grid; one row per thread up to 256 rows a block, then
two), at the edges of the team's forms: BiCGStab through the allocation-free entry point, its
true residual checked in FP64 on the CPU, and the Jacobi-preconditioned
pressure solve against the AMG-preconditioned one (the per-kernel solvers) on
the same passes.

Tolerances: BiCGStab stops on its recursive residual at 1e-10 ||b||, which
stays within rounding of the true one on these diagonally dominant systems
(checked at 2e-10).  Pressure solves run to 1e-12 of ||b||; two solutions then
differ by at most 2e-12 times the condition number (below 1e4 at these sizes)
relative to the correction, itself a small part of the fields: 1e-9.
"""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from minicombust_app_b200 import flow
from minicombust_app_b200.workload import noisy_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 129, 1025, 2047, 2048, 4096, 4097, 9000, 16384, 16385, 151553, 262144])
def test_bicgstab_team(gpu, n):
    import torch
    rng = np.random.default_rng(n)
    idx = np.arange(n)
    off, col = np.zeros((6, n)), np.tile(idx.astype(np.int32), (6, 1))
    for k, d in enumerate((-700, -13, -1, 1, 13, 700)):
        ok = (idx + d >= 0) & (idx + d < n)
        off[k, ok] = -(0.2 + rng.random(int(ok.sum())))
        col[k, ok] = (idx[ok] + d).astype(np.int32)
    diag = 1.02 * np.abs(off).sum(axis=0) + 0.5
    b = rng.standard_normal(n)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (diag, off, col, b)]
    L = flow.library()
    for _ in range(2):  # the second call finds the first one's scratch
        x = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
        its = ctypes.c_int(-1)
        torch.cuda.synchronize()
        rc = L.mc_solve_bicgstab_noalloc(n, *(t.data_ptr() for t in dev), x.data_ptr(), 1e-10, 500, None,
                                         ctypes.byref(its))
        assert rc == flow.MC_OK and its.value > 0
        got = x.cpu().numpy()
        res = b - diag * got - sum(off[k] * got[col[k]] for k in range(6))
        assert np.linalg.norm(res) <= 2e-10 * np.linalg.norm(b)
    rc = L.mc_solve_bicgstab_noalloc(n, *(t.data_ptr() for t in dev), x.data_ptr(), 1e-14, 1, None, None)
    assert rc == (flow.MC_OK if n == 1 else flow.MC_ERR_NOT_CONVERGED)


@pytest.mark.parametrize("dims,reorder", [((8, 4, 4), 0), ((17, 11, 11), 0), ((32, 32, 16), 0), ((33, 25, 20), 0),
                                          ((33, 25, 20), 1), ((80, 44, 43), 0), ((80, 44, 44), 0)])
def test_pcg_team_matches_amg(gpu, dims, reorder):
    out = []
    for psolver in (flow.PSOLVER_PCG_JACOBI, flow.PSOLVER_PCG_AMG):
        s = flow.FlowSolver(flow.Mesh.box(*dims, 0.2, 0.1, 0.1),
                            params=flow.default_params(flow.MODE_SIMPLE, pressure_solver=psolver, reorder=reorder,
                                                       u_rtol=1e-12, p_rtol=1e-12))
        for name, vals in noisy_fields(s.N, 5).items():
            a = s.field(name)
            a[:s.N] = vals
            s.set_field(name, a)
        for _ in range(2):
            s.simple_iteration()
        assert s.last_stats.pressure_rel_residual_first <= 1e-12
        out.append({n: s.field(n) for n in ("U", "V", "W", "P", "TEM")})
        s.close()
    for n, a in out[0].items():
        assert np.abs(a - out[1][n]).max() <= 1e-9 * np.abs(a).max(), n


@pytest.mark.parametrize("dims,team", [((17, 11, 11), True), ((80, 44, 43), True), ((80, 60, 63), True),
                                       ((80, 64, 60), False)])
def test_kernel_counts_name_the_solver_that_ran(gpu, dims, team):
    """A cluster, the grid up to 2,048 rows per SM, the per-kernel solver above."""
    s = flow.FlowSolver(flow.Mesh.box(*dims, 0.2, 0.1, 0.1), params=flow.default_params(flow.MODE_SIMPLE))
    for name, vals in noisy_fields(s.N, 5).items():
        a = s.field(name)
        a[:s.N] = vals
        s.set_field(name, a)
    s.set_timing(True)
    s.simple_iteration()
    n = {k: c for k, (_, c) in s.kernel_times().items()}
    assert (n["pcg_team"] > 0) == team and (n["pcg_iter1_spmv"] > 0) == (not team)
    s.close()


def test_handles_of_two_sizes_in_two_threads(gpu):
    """Two systems that run the same team kernel with different amounts of shared
    memory: each pass is made by the team, with the bits of a pass made alone."""
    import threading
    boxes = ((50, 30, 30), (90, 50, 48))

    def passes(dims, out):
        s = flow.FlowSolver(flow.Mesh.box(*dims, 0.2, 0.1, 0.1), params=flow.default_params(flow.MODE_SIMPLE))
        for name, vals in noisy_fields(s.N, 5).items():
            a = s.field(name)
            a[:s.N] = vals
            s.set_field(name, a)
        s.set_timing(True)
        for _ in range(12):
            s.simple_iteration()
        n = {k: c for k, (_, c) in s.kernel_times().items()}
        out[dims] = {f: s.field(f) for f in ("U", "P", "TEM")}, n["pcg_team"], n["pcg_iter1_spmv"]
        s.close()

    alone, together = {}, {}
    for dims in boxes:
        passes(dims, alone)
    threads = [threading.Thread(target=passes, args=(dims, together)) for dims in boxes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for dims in boxes:
        assert together[dims][1] == alone[dims][1] > 0 and together[dims][2] == alone[dims][2] == 0
        for f, a in alone[dims][0].items():
            assert np.array_equal(together[dims][0][f], a), (dims, f)


CHILD = r"""
import ctypes, os, sys
sys.path.insert(0, os.environ["MC_ROOT"])
import numpy as np
import torch
from minicombust_app_b200 import flow
from minicombust_app_b200.workload import noisy_fields
L = flow.library()
n = 40000
idx = np.arange(n, dtype=np.int32)
off, col = np.zeros((6, n)), np.tile(idx, (6, 1))
off[0, 1:], col[0, 1:] = -1.0, idx[:-1]
dev = [torch.from_numpy(a).cuda() for a in (np.full(n, 2.0), off, col, np.ones(n))]
x = torch.zeros(n, dtype=torch.float64, device="cuda")
def solve():
    torch.cuda.synchronize()
    return L.mc_solve_bicgstab_noalloc(n, *(t.data_ptr() for t in dev), x.data_ptr(), 1e-10, 200, None, None)
s = flow.FlowSolver(flow.Mesh.box(40, 30, 30, 0.2, 0.1, 0.1), params=flow.default_params(flow.MODE_SIMPLE, max_iters=49))
s1 = flow.FlowSolver(flow.Mesh.box(40, 30, 30, 0.2, 0.1, 0.1), params=flow.default_params(flow.MODE_SIMPLE))
for h in (s, s1):
    for name, vals in noisy_fields(h.N, 5).items():
        a = h.field(name)
        a[:h.N] = vals
        h.set_field(name, a)
    h.stage("gradients")
    h.stage("momentum")
def stage(h, name):
    try:
        h.stage(name)
    except flow.FlowError as e:
        return e.status
    return flow.MC_OK
before = s1.field("P")
os.environ["MC_TEAM_WAIT_POLLS"] = "0"
for _ in range(3):
    assert solve() == flow.MC_ERR_TIMEOUT
assert stage(s1, "pressure") == flow.MC_ERR_TIMEOUT
assert np.array_equal(before[:s1.N], s1.field("P")[:s1.N])
assert stage(s, "temperature") == flow.MC_ERR_TIMEOUT  # 49 iterations: BiCGStab, not sweeps
del os.environ["MC_TEAM_WAIT_POLLS"]
for _ in range(2):
    assert solve() == flow.MC_OK
    want = np.zeros(n)
    for k in range(60):  # x_i = (1 + x_{i-1}) / 2
        want = (1.0 + np.concatenate([[0.0], want[:-1]])) / 2
    assert np.abs(x.cpu().numpy() - want).max() <= 1e-8
    assert stage(s1, "pressure") == flow.MC_OK
    assert stage(s, "temperature") in (flow.MC_OK, flow.MC_ERR_NOT_CONVERGED)
print("team timeout ok")
"""


def test_wait_that_runs_out_is_reported_and_recovers(gpu):
    """With a bound of no polls a block that is not the last to arrive gives up at its
    first barrier; the last one waits for none and cannot know.  (These sizes
    take the grid form, so the per-kernel solvers did not run either.)"""
    env = dict(os.environ, MC_ROOT=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    env.pop("MC_TEAM_WAIT_POLLS", None)
    r = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "team timeout ok" in r.stdout
