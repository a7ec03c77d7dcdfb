"""The proposer's gradient at the edges of its kernel's tiles: part of a warp's
16 rows, of a block's 128, one tile more than there are blocks.  Tolerance: FP32
accumulation in another order than the oracle's, 1e-3 of the gradient's norm."""
import os
import sys

import numpy as np
import pytest

from hbtg import learned

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 17, 127, 128, 129, 152 * 128 + 1])
def test_gradient_of_ragged_rows(unbinder, n):
    import mlp_ref
    import torch
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 6)).astype(np.float32)
    y = (rng.random(n) < 0.5).astype(np.float32)
    sw = rng.random(n).astype(np.float32)
    w = learned.initial_weights(n)
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    grad, loss = learned.mlp_backward(t(w), t(x), t(y), t(sw))
    l_ref, g_ref, _ = mlp_ref.loss_and_grad(w, x, y, sw)
    g = grad.cpu().numpy().astype(np.float64)
    assert np.linalg.norm(g - g_ref) <= 1e-3 * np.linalg.norm(g_ref)
    assert float(loss.item()) == pytest.approx(l_ref, rel=1e-4)
