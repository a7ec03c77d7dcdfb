"""Cell masses and centres where their integer sums reach their limits: masses
of one value, of a wide spread and tiny (a massless cell has no centre in the oracle), coordinates around zero, across a
binade and on a coarse grid (centres halfway between floats), more than eight
particles in one place.  The potentials of the tree against the oracle's FP64
tree, at the walk's tolerance."""
import numpy as np
import pytest

from hbtg import abi, oracle

pytestmark = pytest.mark.gpu

MASSES = {
    "unit": lambda r, n: np.ones(n),
    "species": lambda r, n: r.choice([0.19, 1.0, 50.0], n),
    "spread": lambda r, n: np.exp(r.normal(0, 4, n)),
    "some tiny": lambda r, n: np.where(r.random(n) < 0.3, 1e-30, 1.0),
}
PLACES = {
    "inside a binade": lambda r, n: 70.0 + r.normal(0, 0.5, (n, 3)),
    "across a binade": lambda r, n: 64.0 + r.normal(0, 0.5, (n, 3)),
    "around zero": lambda r, n: r.normal(0, 0.5, (n, 3)),
    "grid": lambda r, n: 70.0 + r.integers(-2000, 2000, (n, 3)) * 2.0 ** -13,
    "heaps": lambda r, n: 70.0 + r.normal(0, 0.5, (n // 12 + 1, 3))[r.integers(0, n // 12 + 1, n)],
}


@pytest.mark.parametrize("place", PLACES)
@pytest.mark.parametrize("mass", MASSES)
def test_potentials_of_the_tree(unbinder, mass, place):
    rng = np.random.default_rng(len(mass) + 7 * len(place))
    n = 3000
    pos = PLACES[place](rng, n).astype(np.float32)
    m = MASSES[mass](rng, n).astype(np.float32)
    prm = abi.parity_params(dm_only=1, box_size=100.0, softening=0.01, periodic=0)
    tgt = np.arange(0, n, 3)
    got = unbinder.tree_potential(prm, pos, m, tgt).astype(np.float64)
    ref = oracle.tree_potential(prm, pos, m, pos[tgt], m[tgt])
    # the self term's cancellation leaves an ulp of m / softening
    tol = 3 * np.spacing(np.maximum(m[tgt], np.float32(1e-30)) / np.float32(prm.softening)).astype(np.float64)
    rel = np.maximum(np.abs(got - ref) - tol, 0.0) / np.abs(ref)
    assert np.median(rel) <= 2e-6, np.median(rel)
    assert np.percentile(rel, 99) <= 1e-4, np.percentile(rel, 99)
    assert rel.max() <= 5e-3, rel.max()
