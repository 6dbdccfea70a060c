"""The MLP's device memory, and that nothing stale in it reaches a result.

A net of narrow layers with a large max_batch must fit where one activation,
one pre-activation and the gradients' two buffers per row fit: 2 bytes for
each width, 4 for each layer's output, 8 for the widest, and per parameter
the master copy, gradient, moments, places and BF16 copies (rows padded to
32) -- with 16 MB for alignment and the allocator.

A pass over NaN inputs fills every buffer with NaN; the next, smaller batch
must come out as if it had not been there."""
import numpy as np
import pytest

import lbib
import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,batch", [([16] * 17, 1 << 18), ([3, 40, 40, 1], 1 << 20), ([1, 1], 1 << 22),
                                          ([5, 256, 256, 192], 1 << 17)])
def test_memory_of_a_large_batch(gpu, widths, batch):
    import torch
    wp = [(w + 15) // 16 * 16 for w in widths]
    row = 2 * sum(wp) + 4 * sum(wp[1:]) + 8 * max(wp)
    params = sum(a * b + b for a, b in zip(wp, wp[1:]))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    net = lbib.MLP(widths, max_batch=batch, seed=1)
    used = before - torch.cuda.mem_get_info()[0]
    net.close()
    assert used <= row * batch + 64 * params + (16 << 20)


@pytest.mark.parametrize("widths,large,small", [([7, 40, 130, 20, 64, 3], 300, 130), ([5, 64, 64, 1], 256, 1),
                                                ([300, 24, 200, 17], 257, 65)])
def test_nothing_stale(gpu, widths, large, small):
    import torch
    rng = np.random.default_rng(4)
    with lbib.MLP(widths, max_batch=large, seed=3) as net:
        p = net.params()
        bad = torch.full((large, widths[0]), float("nan"), device="cuda")
        net.gradient(bad, torch.zeros(large, widths[-1], device="cuda"))
        assert torch.isnan(net.forward(bad)).all()
        X = rng.normal(0, 1, (small, widths[0])).astype(np.float32)
        T = rng.normal(0, 0.5, (small, widths[-1])).astype(np.float32)
        Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
        g, loss = net.gradient(Xd, Td)
        Y = net.forward(Xd).cpu().numpy()
    with lbib.MLP(widths, max_batch=large, seed=3) as fresh:
        g2, loss2 = fresh.gradient(Xd, Td)
        np.testing.assert_array_equal(g, g2)
        assert loss == loss2
        np.testing.assert_array_equal(Y, fresh.forward(Xd).cpu().numpy())
    lr, gr = mlp_ref.loss_and_grad(p, widths, X, T)
    assert abs(loss - lr) <= 1e-2 * lr
    assert np.linalg.norm(g - gr) <= 2e-2 * np.linalg.norm(gr)
