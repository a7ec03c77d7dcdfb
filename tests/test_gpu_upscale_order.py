"""Identical subsampled calls give identical results: the masses behind the
upscale factors are added in one order.  The particles outside the sample hold
one of 2^24 and many of half a unit in the last place of a double of that size,
so a sum in another order ends on another side of the point halfway between two
floats."""
import numpy as np
import pytest

from hbtg import abi, synthetic

pytestmark = pytest.mark.gpu


def test_repeated_calls_agree(unbinder):
    sample, tinies = 512, 512
    n = sample + 256 * tinies
    halo = synthetic.nfw_single(n=n, seed=3, interloper_frac=0.0)
    mass = np.zeros(n, np.float32)
    mass[:sample] = 2.0 ** -10
    mass[sample + 100::256] = 2.0 ** -29
    big = sample + 120 + 256 * (tinies // 2)
    mass[big] = 2.0 ** 24
    zero = np.zeros((1, 3), np.float32)
    inp = abi.Inputs(np.array([0, n], np.int64), halo.pos, np.zeros((n, 3), np.float32), mass, np.arange(n) + 5, None,
                     None, halo.ref_pos, zero.copy(), halo.pos[:1].copy(), zero.copy(), np.array([5], np.int64))
    prm = abi.parity_params(dm_only=1, box_size=100.0, max_sample_size=sample, prepared_subsample=1)
    for before in range(4, tinies, 8):  # how many of the small ones must be added before the large one to pass halfway
        mass[big + 1] = 0.5 - 2.0 ** -29 * before
        seen = {unbinder.unbind(inp, prm, allow_max_iter=True).energy.tobytes() for _ in range(6)}
        assert len(seen) == 1, (before, len(seen))
