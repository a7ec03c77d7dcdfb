"""Host-pointer calls whose arrays fit one pinned buffer, and those that do not,
return what the device-pointer call returns, in/out frames and warm-start
priors included."""
import numpy as np
import pytest

from hbtg import abi, learned, synthetic
from hbtg.gpu import DeviceBatch

pytestmark = pytest.mark.gpu


def _device(unbinder, inp, prm, use_prior=None):
    db = DeviceBatch(inp)
    db.reset_inout()
    if use_prior is None:
        unbinder.unbind_device(prm, db.c)
    else:
        unbinder.unbind_learned_device(prm, db, use_prior=use_prior)
    return db.outputs()


def _same(inp, a, b):
    for k in a.__dict__:
        x, y = getattr(a, k), getattr(b, k)
        if k == "energy":
            rows = np.concatenate([np.arange(inp.offsets[s], inp.offsets[s] + a.nbound[s]) for s in range(inp.n_sub)])
            assert np.array_equal(x[rows.astype(np.int64)], y[rows.astype(np.int64)])
        elif x is not None and y is not None:
            assert np.array_equal(x, y), k


@pytest.mark.parametrize("total", [60, 3000, 4500, 30_000])  # the buffer takes about 4,500 particles
def test_host_and_device_calls_agree(unbinder, total):
    inp = synthetic.batched(total=total, seed=total, nmax=max(60, total // 3))
    prm = abi.parity_params(dm_only=1, box_size=500.0)
    _same(inp, unbinder.unbind(inp, prm), _device(unbinder, inp, prm))
    inp = synthetic.hydro(total=total, seed=total, nmin=50, nmax=max(100, total // 3), box=200.0)
    prm = abi.parity_params(thermal=1, box_size=200.0)
    _same(inp, unbinder.unbind(inp, prm), _device(unbinder, inp, prm))


@pytest.mark.parametrize("n_sub", [4, 200])
def test_warm_start_priors(unbinder, n_sub):
    learned.Model.load().install(unbinder)
    inp = synthetic.stripped(n_sub=n_sub, seed=5, nmin=100, nmax=900)
    prm = abi.parity_params(dm_only=1, box_size=500.0)
    _same(inp, unbinder.unbind_learned(inp, prm), _device(unbinder, inp, prm, use_prior=True))


def test_empty_batches(unbinder):
    inp = synthetic.small_cases(seed=1)
    prm = abi.parity_params(dm_only=1, box_size=100.0)
    empty = inp.subset([int(np.nonzero(np.diff(inp.offsets) == 0)[0][0])])
    out = unbinder.unbind(empty, prm)
    assert out.nbound.tolist() == [0] and out.status.tolist() == [abi.SUB_EMPTY]
