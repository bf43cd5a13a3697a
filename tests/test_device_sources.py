"""Sources set once from device memory and kept over several passes: their
total mass source must outlive a pass (it shared its word with the largest
pressure diagonal, which the refined AMG path forms in every pass)."""
import numpy as np
import pytest

from minicombust_app_b200 import flow
from minicombust_app_b200.workload import gaussian_blobs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [flow.PRECISION_FP64, flow.PRECISION_FP32_REFINED], ids=["fp64", "refined"])
def test_device_sources_kept_over_passes(gpu, precision):
    import torch
    dims, lengths = (24, 12, 12), (0.2, 0.1, 0.1)
    src = gaussian_blobs(dims, lengths, 4, 1, rel_amplitude=0.05)
    out = []
    for device in (False, True):
        s = flow.FlowSolver(flow.Mesh.box(*dims, *lengths),
                            params=flow.default_params(flow.MODE_SIMPLE, pressure_solver=flow.PSOLVER_PCG_AMG,
                                                       precision=precision, u_rtol=1e-12, p_rtol=1e-12))
        if device:
            t = torch.from_numpy(np.ascontiguousarray(src.T)).cuda()
            torch.cuda.synchronize()
            s.set_sources_device(t.data_ptr())
        else:
            s.set_sources(src)
        for _ in range(3):
            s.simple_iteration()
        out.append({n: s.field(n) for n in ("U", "V", "W", "P", "TEM")})
        s.close()
    # the two totals are summed in different orders: last bits only
    for n, a in out[0].items():
        assert np.abs(a - out[1][n]).max() <= 1e-9 * np.abs(a).max(), n
