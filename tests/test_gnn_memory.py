"""Training where the device cannot hold the work area of eight samples: fewer
are then trained together.  The memory is taken by one allocation that leaves
room for a sample or two.  Gradients are FP32 sums over the same cells, grouped
by sample: they agree to 1e-4 (a sample left out changes them by a tenth)."""
import numpy as np
import pytest

from minicombust_app_b200 import flow, gnn

pytestmark = pytest.mark.gpu


def test_training_takes_fewer_samples_when_memory_is_short(gpu):
    import torch
    mesh = flow.Mesh.box(64, 32, 32, 0.2, 0.1, 0.1)
    g = torch.Generator(device="cuda").manual_seed(5)
    samples = [tuple(torch.randn(mesh.n_cells, device="cuda", generator=g) + shift for shift in (0.0, 4.0, 0.0, 0.0))
               for _ in range(8)]
    nets = [gnn.GuessNet(seed=3) for _ in range(2)]
    graphs = [n.graph(mesh) for n in nets]
    loss, grad = nets[0].loss_grad(graphs[0], samples)
    one = nets[0].loss_grad(graphs[0], samples[:1])[1]  # also: every kernel is loaded
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hold = torch.empty(free - (160 << 20), dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            l2, g2 = nets[1].loss_grad(graphs[1], samples)
            assert abs(l2 - loss) <= 1e-6 * abs(loss)
            assert np.linalg.norm(g2 - grad) <= 1e-4 * np.linalg.norm(grad)
        y = torch.empty(mesh.n_cells, device="cuda")
        nets[1].predict(graphs[1], *samples[0][:3], y=y)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert np.linalg.norm(one - grad) > 1e-3 * np.linalg.norm(grad)
    l3, g3 = nets[1].loss_grad(graphs[1], samples)
    assert np.linalg.norm(g3 - grad) <= 1e-4 * np.linalg.norm(grad)
