"""hbtg_tree_potential_device orders its targets for the walk: the potential of
a particle does not depend on how the targets are listed, beyond the rounding
of one FP32 sum (the terms are the same, grouped differently)."""
import numpy as np
import pytest

from hbtg import abi, synthetic
from hbtg.gpu import UnbindError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, n_tgt", [(1, 1), (1, 70), (2, 33), (3000, 1), (3000, 2049), (3000, 20_000)])
def test_any_list_of_targets(unbinder, n, n_tgt):
    rng = np.random.default_rng(n_tgt)
    inp = synthetic.nfw_single(n=max(n, 2), seed=3)
    prm = abi.parity_params(dm_only=1, box_size=100.0)
    pos, mass = inp.pos[:n], inp.mass[:n]
    every = unbinder.tree_potential(prm, pos, mass, np.arange(n)).astype(np.float64)
    tgt = rng.integers(0, n, n_tgt)  # repeats, any order, more targets than sources
    got = unbinder.tree_potential(prm, pos, mass, tgt).astype(np.float64)
    tol = 4e-7 * np.abs(every[tgt]) + 3 * np.spacing(np.float32(1.0 / prm.softening))
    assert np.all(np.abs(got - every[tgt]) <= tol)


def test_targets_outside_the_sources_are_refused(unbinder):
    inp = synthetic.nfw_single(n=100, seed=3)
    prm = abi.parity_params(dm_only=1, box_size=100.0)
    for bad in (-1, 100):
        with pytest.raises(UnbindError):
            unbinder.tree_potential(prm, inp.pos, inp.mass, [0, bad, 5])
