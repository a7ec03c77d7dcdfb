"""Sorts and scans at the sizes where their launches change: one block, several
tiles, the last tile of the digit table that a histogram's last block scans,
and one more; the potentials of the tree built from the sorted keys, and the
order of a call's energies."""
import numpy as np
import pytest

from hbtg import abi, oracle, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2048, 2049, 8192, 8193, 128 * 2048, 128 * 2048 + 1])
def test_tree_of_n_sources(unbinder, n):
    inp = synthetic.nfw_single(n=n, seed=n)
    prm = abi.parity_params(dm_only=1, box_size=100.0)
    tgt = np.random.default_rng(n).choice(n, 40, replace=False)
    got = unbinder.tree_potential(prm, inp.pos, inp.mass, tgt).astype(np.float64)
    ref = oracle.tree_potential(prm, inp.pos, inp.mass, inp.pos[tgt], inp.mass[tgt])
    rel = np.abs(got - ref) / np.abs(ref)
    assert np.median(rel) <= 2e-6 and rel.max() <= 1e-4, (np.median(rel), rel.max())


@pytest.mark.parametrize("n_sub, total", [(1, 70_000), (300, 70_000), (2, 300_000)])
def test_energies_come_back_in_order(unbinder, n_sub, total):
    inp = synthetic.batched(n_sub=n_sub, seed=3, nmin=total // n_sub, nmax=total // n_sub + 1)
    out = unbinder.unbind(inp, abi.parity_params(dm_only=1, box_size=500.0))
    assert out.nbound.sum() > 0.3 * inp.n_particles
    for s in range(n_sub):
        a, b, nb = inp.offsets[s], inp.offsets[s + 1], out.nbound[s]
        assert np.array_equal(np.sort(out.order[a:b]), np.arange(b - a))
        assert np.all(np.diff(out.energy[a:a + nb]) >= 0)
