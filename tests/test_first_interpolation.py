"""The first node interpolation of a handle: the node tables are set up on the
default stream, and the call's kernels must not start before they are there
(too few nodes were counted where they did)."""
import numpy as np
import pytest

from minicombust_app_b200 import flow

pytestmark = pytest.mark.gpu


def test_first_call_counts_every_node(gpu):
    dims = (64, 32, 32)
    mesh = flow.Mesh.box(*dims, 0.2, 0.1, 0.1)
    cells = np.arange(mesh.n_cells, dtype=np.uint64)
    for _ in range(6):
        s = flow.FlowSolver(mesh, params=flow.default_params(flow.MODE_SIMPLE))
        s.stage("gradients")
        ids, vals = s.interpolate_nodes(cells)
        assert len(ids) == (dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1)
        assert np.array_equal(ids, np.arange(len(ids)))
        s.close()
