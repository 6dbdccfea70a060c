"""The MLP's tile kernels at the sizes where their tiling can go wrong:
batches around the row tile (128) and the K unit of the weight gradients
(64), widths around the column tile (32) and the 16-column padding, K
beyond the staged slices (256), an FP32 input wider than they hold, and a
batch smaller than the one before it on the same net (whose rows must not
leak into the gradients).

Against tests/mlp_ref.py, which rounds to bf16 where the kernels do and
sums in FP64, with the bars of test_gpu_mlp.py: outputs to 1e-2 of the
largest, gradients to 2e-2 relative L2 (an activation that rounds the other
way moves by 2^-8)."""
import numpy as np
import pytest

import lbib
import mlp_ref

pytestmark = pytest.mark.gpu


def _check(net, widths, p, batch, rng):
    import torch
    X = rng.normal(0, 1, (batch, widths[0])).astype(np.float32)
    T = rng.normal(0, 0.5, (batch, widths[-1])).astype(np.float32)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    Y = net.forward(Xd).cpu().numpy()
    g, loss = net.gradient(Xd, Td)
    Yr, _, _ = mlp_ref.forward(p, widths, X)
    assert np.max(np.abs(Y - Yr)) <= 1e-2 * np.max(np.abs(Yr))
    lr, gr = mlp_ref.loss_and_grad(p, widths, X, T)
    assert abs(loss - lr) <= 1e-2 * lr
    assert np.linalg.norm(g - gr) <= 2e-2 * np.linalg.norm(gr)


@pytest.mark.parametrize("widths,batches", [
    ([1, 16, 1], [1, 2]),
    ([5, 33, 31, 17], [127, 128, 129]),
    ([7, 129, 65], [63, 64, 65]),
    ([4, 300, 288, 8], [200, 130]),
    ([300, 40, 3], [257, 40]),
    ([3, 64, 64, 64, 1], [1000, 300]),
])
def test_tiles_match_cpu(gpu, widths, batches):
    rng = np.random.default_rng(11)
    with lbib.MLP(widths, max_batch=max(batches), seed=5) as net:
        p = net.params()
        p += rng.normal(0, 0.02, p.size).astype(np.float32)
        net.set_params(p)
        for b in sorted(batches, reverse=True):   # the larger batch first: its rows stay in the buffers
            _check(net, widths, p, b, rng)
