"""The neighbour search of the particle reassignment where its first bound and
its list sizes change: every list size, groups with fewer tracers than
neighbours asked for (and none at all), coincident tracers, and enough
particles that the searches are sorted in several passes."""
import numpy as np
import pytest

from hbtg import abi, oracle, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_groups", [3, 24])
@pytest.mark.parametrize("k", [1, 8, 9, 16, 17, 32])
def test_neighbour_search_at_its_edges(unbinder, n_groups, k):
    inp, group_off = synthetic.fof_groups(seed=11 + n_groups, n_groups=n_groups, n_sat=3, box=60.0, swap=0.2)
    rng = np.random.default_rng(k)
    prm = abi.parity_params(thermal=1, box_size=60.0)
    tracer = ((1 << inp.type.astype(np.int64)) & prm.tracer_type_mask) != 0
    group = lambda h: slice(inp.offsets[group_off[h]], inp.offsets[group_off[h + 1]])  # noqa: E731
    first = np.nonzero(tracer[group(0)])[0] + inp.offsets[group_off[0]]
    inp.type[first[k - 1:]] = 0  # the first group: one tracer fewer than neighbours asked for (none for k = 1)
    second = np.nonzero(tracer[group(1)])[0] + inp.offsets[group_off[1]]
    inp.type[second[k:]] = 0  # the second: as many
    for s in range(group_off[2], group_off[3]):  # the third: coincident tracers, those of one subhalo together
        rows = np.nonzero(tracer[inp.offsets[s]:inp.offsets[s + 1]])[0] + inp.offsets[s]
        pick = rng.permutation(rows)[: 2 * (len(rows) // 4)].reshape(-1, 2)
        inp.pos[pick[:, 1]] = inp.pos[pick[:, 0]]
    got = unbinder.reassign(inp, group_off, prm, k)
    ref = oracle.reassign(inp, group_off, prm, k)
    assert (ref >= 0).sum() > 20
    assert np.array_equal(got, ref), (got != ref).sum()
