"""Core phase-space properties for every sign of the core's size: a size that
the counted particles never reach takes them all, in small calls (a warp per
subhalo) as in large ones (a thread per subhalo) and as in the oracle."""
import numpy as np
import pytest

from hbtg import abi, oracle, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sub", [3, 4200])
@pytest.mark.parametrize("factor, least", [(0.0, 20), (0.25, 0), (-1.0, -5)])
def test_core_sizes(unbinder, factor, least, n_sub):
    inp = synthetic.batched(n_sub=n_sub, seed=2, nmin=25, nmax=40)
    prm = abi.parity_params(dm_only=1, box_size=500.0, sub_core_size_factor=factor, sub_core_size_min=least)
    got, ref = unbinder.unbind(inp, prm), oracle.run_port(inp, prm)
    assert np.isfinite(ref.core).all()
    np.testing.assert_allclose(got.core, ref.core, rtol=2e-5, atol=1e-5)
