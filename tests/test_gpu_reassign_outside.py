"""Reassignment of particles whose coordinates lie outside the box: a wrapped
offset is as accurate as any other, so the nearest tracer is the oracle's."""
import numpy as np
import pytest

from hbtg import abi, oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1])
@pytest.mark.parametrize("shift", [0.0, -60.0])
def test_particles_one_box_away(unbinder, shift, k):
    rng = np.random.default_rng(k)
    n, box = 10_000, 60.0
    pos = (0.02 * rng.random((n, 3))).astype(np.float32)
    typ = np.where(np.arange(n) % 2 == 0, 1, 0).astype(np.uint8)  # dark matter, which traces, and gas
    gas = typ == 0
    pos[gas] = (pos[gas].astype(np.float64) + shift).astype(np.float32)
    n_sub = 40
    offsets = (np.arange(n_sub + 1) * (n // n_sub)).astype(np.int64)
    zero = np.zeros((n_sub, 3), np.float32)
    inp = abi.Inputs(offsets, pos, np.zeros((n, 3), np.float32), np.ones(n, np.float32), np.arange(n) + 5, typ,
                     np.zeros(n, np.float32), zero, zero.copy(), zero.copy(), zero.copy(), np.zeros(n_sub, np.int64))
    group_off = np.array([0, n_sub], np.int64)
    prm = abi.parity_params(thermal=1, box_size=box)
    got = unbinder.reassign(inp, group_off, prm, k)
    ref = oracle.reassign(inp, group_off, prm, k)
    assert (ref >= 0).sum() > 1000
    assert np.array_equal(got, ref), (got != ref).sum()
