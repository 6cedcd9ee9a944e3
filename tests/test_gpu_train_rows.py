"""A training step takes its rows through the shuffled index in place: the same
parameters, bit for bit, from inputs at a 16-byte boundary and 4 bytes past one, at
the edges of the 64-sample tiles; and for one sample (no shuffle) from the gradient
and the update called one after the other."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 63, 64, 65, 130])
def test_training_step_rows(rows):
    import torch
    import plum_gb300 as pg
    g = torch.Generator().manual_seed(rows)
    x = (torch.rand((rows, 96), generator=g) * 20).cuda()
    t = torch.randn(rows, generator=g).cuda()
    nets = [pg.Surrogate(seed=4) for _ in range(3)]
    for net in nets:
        net.set_norm(np.full(96, 5.0, np.float32), np.full(96, 0.2, np.float32), 3.0)
    store = torch.zeros(rows * 96 + 1, device="cuda")
    store[1:] = x.ravel()
    shifted = store[1:].view(rows, 96)
    assert x.data_ptr() % 16 == 0 and shifted.data_ptr() % 16 == 4
    a = nets[0].train(x, t, batch=rows, lr=1e-3, seed=2)
    b = nets[1].train(shifted, t, batch=rows, lr=1e-3, seed=2)
    np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(nets[0].params(), nets[1].params())
    if rows == 1:
        grad, loss = nets[2].grad(x.cpu().numpy(), t.cpu().numpy())
        nets[2].adam_step(grad, 1e-3)
        assert loss == a[0]
        np.testing.assert_array_equal(nets[0].params(), nets[2].params())
