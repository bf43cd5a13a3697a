"""The first pressure corrector of a pass as one device graph: what it reports
when a solve in it breaks down."""
import numpy as np
import pytest

from minicombust_app_b200 import flow
from minicombust_app_b200.workload import noisy_fields

pytestmark = pytest.mark.gpu


def pressure_status(scale):
    """Status of the pressure stage of a pass with velocities of 50 x scale."""
    s = flow.FlowSolver(flow.Mesh.box(16, 12, 8, 0.2, 0.1, 0.1),
                        params=flow.default_params(flow.MODE_SIMPLE, pressure_solver=flow.PSOLVER_PCG_AMG,
                                                   precision=flow.PRECISION_FP32_REFINED))
    for name, vals in noisy_fields(s.N, seed=3).items():
        a = s.field(name)
        a[:s.N] = vals * (scale if name in "UVW" else 1.0)
        s.set_field(name, a)
    s.stage("gradients")
    s.stage("momentum")
    status = flow.MC_OK
    try:
        s.stage("pressure")
    except flow.FlowError as e:
        status = e.status
    s.close()
    return status


def test_inner_fp32_breakdown_is_reported(gpu):
    """Velocities whose flow imbalance exceeds FP32's range (but not FP64's) break
    the inner FP32 solve down while the FP64 refinement around it stays finite."""
    assert pressure_status(1.0) == flow.MC_OK
    assert pressure_status(1e45) == flow.MC_ERR_NONFINITE
