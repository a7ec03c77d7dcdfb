"""Properties of bound sets whose sizes end anywhere in a row of 32 items, in a
warp's 256 and in a block's 2048, several subhaloes to a row: the profile
quantities are the oracle's, the shape sums to the ulps that a double sum in
another order moves."""
import numpy as np
import pytest

from hbtg import abi, oracle, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2, 3, 29, 1, 40, 31, 33), (257, 255, 1, 2, 511), (2048, 7, 2049, 300)])
def test_rows_shared_by_subhaloes(unbinder, sizes):
    parts = [synthetic.nfw_single(n=max(n, 2), seed=n, box=100.0) for n in sizes]
    cut = lambda k: np.concatenate([getattr(p, k)[:n] for p, n in zip(parts, sizes)])  # noqa: E731
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    head = lambda k: np.concatenate([getattr(p, k) for p in parts])  # noqa: E731
    inp = abi.Inputs(off, cut("pos"), cut("vel"), cut("mass"), np.arange(off[-1]) + 5, None, None, head("ref_pos"),
                     head("ref_vel"), head("mostbound_pos"), head("mostbound_vel"), head("most_bound_id"))
    prm = abi.parity_params(dm_only=1, box_size=100.0, hubble=10.0)
    out = abi.CallBuffers(inp).out  # every particle bound, in input order
    out.order[:] = np.concatenate([np.arange(n) for n in sizes])
    out.nbound[:] = sizes
    out.mbound[:] = sizes
    out.mostbound_pos[:] = inp.pos[off[:-1]]
    got = unbinder.subhalo_properties(inp, out, prm)
    ref = oracle.subhalo_properties(inp, out, prm)
    for k in ("rmax", "vmax", "rhalf", "renclose", "m200", "last_vmax", "rmax_last", "snap_last", "nsource"):
        assert np.array_equal(getattr(got, k), getattr(ref, k)), k
    np.testing.assert_allclose(got.r200, ref.r200, rtol=3e-7)
    for k in ("inertia", "inertia_w"):
        g, r = getattr(got, k), getattr(ref, k)
        assert np.array_equal(np.isnan(g), np.isnan(r)), k
        scale = np.nanmax(np.abs(r), axis=1, keepdims=True, initial=0) + 1e-30
        assert np.all(np.nan_to_num(np.abs(g - r)) <= 4e-7 * scale), k
