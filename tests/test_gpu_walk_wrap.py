"""The tree walk where targets wrap around the periodic box: sets across a
corner (each target group on one side of a face), sets over the whole box
(groups whose targets wrap differently) and coordinates outside the box,
against the oracle's FP64 tree.  Tolerances as for the unwrapped walk: the same
interactions in FP32, a few ulps of the sum, and the self term's ulp where the
potential is made of few particles."""
import numpy as np
import pytest

from hbtg import abi, oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 33, 257, 4000])
@pytest.mark.parametrize("layout", ["corner", "box", "outside"])
def test_wrapped_potentials_match_the_oracle_tree(unbinder, layout, n):
    rng = np.random.default_rng(n)
    prm = abi.parity_params(dm_only=1, box_size=100.0, softening=0.02)
    if layout == "box":
        pos = rng.random((n, 3)) * 100.0
    else:
        pos = rng.standard_normal((n, 3)) * 1.5
        if layout == "corner":
            pos = np.mod(pos, 100.0)
        else:  # some particles one box away
            pos += 100.0 * rng.integers(-1, 2, (n, 3))
    pos[0] = [0.01, 0.01, 0.01]
    pos[1] = [99.99, 99.99, 99.99]
    pos = pos.astype(np.float32)
    mass = rng.uniform(0.5, 1.5, n).astype(np.float32)
    tgt = rng.permutation(n)
    got = unbinder.tree_potential(prm, pos, mass, tgt).astype(np.float64)
    ref = oracle.tree_potential(prm, pos, mass, pos[tgt], mass[tgt])
    tol = 3 * np.spacing(np.float32(mass[tgt] / prm.softening)).astype(np.float64)
    rel = np.maximum(np.abs(got - ref) - tol, 0.0) / np.abs(ref)
    assert np.median(rel) <= 2e-6, np.median(rel)
    assert np.percentile(rel, 99) <= 1e-4, np.percentile(rel, 99)
    assert rel.max() <= 5e-3, rel.max()
