"""Several subhaloes too large for a block's team do not wait for one another:
six copies of one with many iterations left take less than twice as long as one."""
import time

import numpy as np
import pytest

from hbtg import abi, synthetic
from hbtg.gpu import DeviceBatch

pytestmark = pytest.mark.gpu


def _copies(one, m):
    n = one.n_particles
    cat = lambda a: np.concatenate([a] * m)  # noqa: E731
    return abi.Inputs(np.arange(m + 1, dtype=np.int64) * n, cat(one.pos), cat(one.vel), cat(one.mass), np.arange(m * n) + 5,
                      None, None, cat(one.ref_pos), cat(one.ref_vel), cat(one.mostbound_pos), cat(one.mostbound_vel),
                      cat(one.most_bound_id))


def test_six_large_subhaloes(unbinder):
    import torch
    prm = abi.parity_params(dm_only=1, box_size=500.0)
    one = synthetic.stripped(n_sub=1, seed=1, nmin=16_000, nmax=16_001)
    ms = {}
    for m in (1, 6):
        db = DeviceBatch(_copies(one, m))
        best = []
        for _ in range(12):
            db.reset_inout()
            torch.cuda.synchronize()
            t = time.perf_counter()
            unbinder.unbind_device(prm, db.c)
            torch.cuda.synchronize()
            best.append(time.perf_counter() - t)
        ms[m] = min(best) * 1e3
        nb = db.outputs().nbound
        assert np.all(nb == nb[0]) and nb[0] > 0
    assert ms[6] < 2 * ms[1], ms


@pytest.mark.parametrize("sizes", [(256,), (257,), (1024,), (1025,), (1024,) * 50, (8192, 8193), (9000,) * 6, (20_480,), (20_481, 9000), (21_000, 20_480, 8193)])
def test_the_same_bits_whichever_team(unbinder, sizes):
    """Sizes about the limits between blocks, clusters and the grid, alone and several, against lock step."""
    prm = abi.parity_params(dm_only=1, box_size=500.0)
    parts = [synthetic.stripped(n_sub=1, seed=3 + k, nmin=n, nmax=n + 1) for k, n in enumerate(sizes)]
    cat = lambda k: np.concatenate([getattr(p, k) for p in parts])  # noqa: E731
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    inp = abi.Inputs(off, cat("pos"), cat("vel"), cat("mass"), np.arange(off[-1]) + 5, None, None, cat("ref_pos"),
                     cat("ref_vel"), cat("mostbound_pos"), cat("mostbound_vel"), cat("most_bound_id"))
    got, team = unbinder.unbind(inp, prm), unbinder.stats()
    unbinder.count_interactions(True)
    try:
        ref, lock = unbinder.unbind(inp, prm), unbinder.stats()
    finally:
        unbinder.count_interactions(False)
    assert got.nbound.min() > 0 and team["walk_launches"] < lock["walk_launches"]  # teams did take over
    for k in ("nbound", "mbound", "ref_pos", "ref_vel", "iterations", "status", "most_bound_id", "order"):
        assert np.array_equal(getattr(got, k), getattr(ref, k)), k
    for s in range(inp.n_sub):
        r = slice(off[s], off[s] + got.nbound[s])
        assert np.array_equal(got.energy[r], ref.energy[r]), s
