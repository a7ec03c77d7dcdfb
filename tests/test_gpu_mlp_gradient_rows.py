"""The proposer's gradient over many rows is as near to 64 bits as sums of FP32
additions are: a weight's gradient is m rounded additions one after the other
(the rows of a block by 16, then the blocks), whose errors of 2^-24 each add up
as sqrt(m), 1.4e-6 of the norm for the 411 + 152 of 1e6 rows."""
import os
import sys

import numpy as np
import pytest

from hbtg import learned

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65_536, 1_000_000])
def test_gradient_of_many_rows(unbinder, n):
    import mlp_ref
    import torch
    rng = np.random.default_rng(n)
    x = rng.standard_normal((n, 6)).astype(np.float32)
    y = (x[:, 0] + 0.5 * rng.standard_normal(n) < 0).astype(np.float32)
    w = learned.initial_weights(2)
    ref = sum(mlp_ref.loss_and_grad(w, x[a:a + 100_000], y[a:a + 100_000])[1] for a in range(0, n, 100_000))
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    grad = learned.mlp_backward(t(w), t(x), t(y))[0].cpu().numpy().astype(np.float64)
    at = 0
    for name, size in mlp_ref.SIZES:
        g, r = grad[at:at + size], ref[at:at + size]
        assert np.linalg.norm(g - r) <= 2e-6 * np.linalg.norm(r), (name, np.linalg.norm(g - r) / np.linalg.norm(r))
        at += size
