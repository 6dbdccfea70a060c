"""The MLP's FP32 input, rounded by layer 0 itself (up to 16 columns) or by a
launch before it: at the border, at widths that end inside a chunk of 8 or a
block of 64 columns, at batches around a block of 32 and of 128 rows, and
from rows that are not 16-byte aligned.

Against tests/mlp_ref.py with the bars of test_gpu_mlp_tiles.py; the same
rows from another place give the same bits."""
import numpy as np
import pytest

import lbib
import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w0", [15, 16, 17, 20, 63, 64, 72, 131, 520])
@pytest.mark.parametrize("batch", [1, 31, 33, 128, 257])
def test_input_columns(gpu, w0, batch):
    import torch
    widths = [w0, 40, 24, 3]
    rng = np.random.default_rng(w0 + batch)
    X = rng.normal(0, 1, (batch, w0)).astype(np.float32)
    T = rng.normal(0, 0.5, (batch, 3)).astype(np.float32)
    Td = torch.from_numpy(T).cuda()
    with lbib.MLP(widths, max_batch=300, seed=9) as net:
        p = net.params()
        net.gradient(torch.full((300, w0), float("nan"), device="cuda"), torch.zeros(300, 3, device="cuda"))
        got = []
        for shift in (0, 1):             # 16-byte aligned rows where w0 allows it, and not
            buf = torch.full((batch * w0 + 4,), float("nan"), device="cuda")
            Xd = buf[shift:shift + batch * w0].view(batch, w0)
            Xd.copy_(torch.from_numpy(X))
            got.append((net.forward(Xd).cpu().numpy(), *net.gradient(Xd, Td)))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
    Y, g, loss = got[0]
    Yr, _, _ = mlp_ref.forward(p, widths, X)
    assert np.max(np.abs(Y - Yr)) <= 1e-2 * np.max(np.abs(Yr))
    lr, gr = mlp_ref.loss_and_grad(p, widths, X, T)
    assert abs(loss - lr) <= 1e-2 * lr
    assert np.linalg.norm(g - gr) <= 2e-2 * np.linalg.norm(gr)
