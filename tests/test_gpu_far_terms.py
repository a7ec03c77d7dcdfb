"""The walk's far term -m / r over the range of distances whose squares are
normal floats, against 64 bits.  Bound: 2^-22.9 for PTX's rsqrt.approx.ftz.f32
(its documented error), half of r^2's rounding (2^-25), the roundings of the
product and of the result (2^-24 each)."""
import numpy as np
import pytest

from hbtg import abi

pytestmark = pytest.mark.gpu

BOUND = 2.0 ** -22.9 + 2.0 ** -25 + 2 * 2.0 ** -24


@pytest.mark.parametrize("lo, hi", [(-17, -8), (-8, 0), (0, 8), (8, 17)])
def test_two_particles_at_any_distance(unbinder, lo, hi):
    rng = np.random.default_rng(hi + 20)
    for r in np.float32(10.0) ** rng.uniform(lo, hi, 60).astype(np.float32):
        prm = abi.parity_params(dm_only=1, box_size=100.0, periodic=0, softening=float(r) / 4)
        pos = np.array([[0, 0, 0], [r, 0, 0]], np.float32)
        got = float(unbinder.tree_potential(prm, pos, np.array([0, 3], np.float32), [0])[0])
        assert got == pytest.approx(-3.0 / float(r), rel=BOUND), r
