"""Training gradients at the edges of the kernel's 64-row tiles: one row, just
below, at and above a tile, and more tiles than the blocks that share them."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRAD_RTOL = 2e-3   # FP32 gradients vs FP64 oracle, relative to the largest entry (as in test_gpu_mlp.py)


@pytest.mark.parametrize("n", [1, 63, 64, 65, 129, 40_001])
def test_gradient_matches_oracle(n):
    import torch
    from oracle import mlp_oracle as mo
    from tsr_b200 import core
    rng = np.random.default_rng(n)
    theta = mo.init(n).astype(np.float32)
    theta += rng.normal(0, 0.05, theta.shape).astype(np.float32)
    x = rng.normal(size=(n, mo.NF)).astype(np.float32)
    y = (rng.uniform(size=(n, mo.NO)) < 0.3).astype(np.float32)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    xd, yd, td = (torch.from_numpy(a).cuda() for a in (x, y, theta))
    grads, loss = torch.zeros(mo.NPARAM, device="cuda"), torch.zeros(1, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    core._check(core.lib.tsr_mlp_train_batch(p(xd), p(yd), n, p(td), p(grads), p(loss), 3.0, 2.0, stream))
    l_ref, g_ref = mo.loss_and_grad(theta, x, y, (3.0, 2.0))
    assert abs(float(loss.item()) - l_ref) <= 1e-4 * abs(l_ref)
    assert np.max(np.abs(grads.cpu().numpy() - g_ref)) <= GRAD_RTOL * np.max(np.abs(g_ref))
