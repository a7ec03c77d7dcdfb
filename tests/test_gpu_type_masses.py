"""Per-type bound masses (hbtg_batch.mbound_type) are the reference's own
sequential float sums (CountParticleTypes, src/subhalo.cpp:311-393) whatever
the masses: equal ones, a wide spread, and ones that fall halfway between the
sum's representable values."""
import numpy as np
import pytest

from hbtg import abi, synthetic

pytestmark = pytest.mark.gpu


def _masses(kind, inp, rng):
    n = inp.n_particles
    if kind == "species":  # one value per species
        return inp.mass
    if kind == "spread":
        return np.exp(rng.normal(0.0, 2.0, n)).astype(np.float32)
    if kind == "ties":  # multiples of a half, with sums far above 2^24 halves
        return (rng.integers(1, 64, n) * 0.5 + 4096.0 * (rng.random(n) < 0.5)).astype(np.float32)
    m = inp.mass.copy()  # some massless and some tiny particles
    m[rng.random(n) < 0.1] = 0.0
    m[rng.random(n) < 0.1] = np.float32(1e-30)
    return m


@pytest.mark.parametrize("kind", ["species", "spread", "ties", "tiny"])
def test_type_masses_are_the_sequential_float_sums(unbinder, kind):
    rng = np.random.default_rng(5)
    # the sizes end inside a row of 32, inside a step of 256, and far above both
    parts = [synthetic.hydro(seed=q, n_sub=3, nmin=n, nmax=n + 1, box=200.0) for q, n in
             enumerate((100, 288, 1025, 40_000))]
    for inp in parts:
        inp.mass = _masses(kind, inp, rng)
        out = unbinder.unbind(inp, abi.parity_params(thermal=1, box_size=200.0))
        assert out.nbound.max() > 50
        for s in range(inp.n_sub):
            rows = inp.offsets[s] + out.order[inp.offsets[s]:inp.offsets[s] + out.nbound[s]]
            for t in range(6):
                m = inp.mass[rows[inp.type[rows] == t]]
                want = np.cumsum(m, dtype=np.float32)[-1] if len(m) else np.float32(0)
                assert out.mbound_type[s, t] == want, (kind, s, t)
