"""Subhaloes that a team takes over (csrc/settle.cuh) end with the same bits as
in lock step: every output of a call against the same call with the
interaction counter on, which keeps to lock step.  Sizes around a warp's 32
targets, a block's 256 threads, the 1024 targets that one block takes and the
2048 tree sources of a team; species, thermal energies, potential subsamples,
wrapped subhaloes, warm starts and a bound on the iterations."""
import numpy as np
import pytest

from hbtg import abi, learned, synthetic

pytestmark = pytest.mark.gpu


def _same(a, b):
    for k in a.__dict__:
        x, y = getattr(a, k), getattr(b, k)
        if x is None:
            continue
        if k in ("energy", "potential"):  # written for the bound particles only
            continue
        assert np.array_equal(x, y), (k, np.argwhere(np.asarray(x != y))[:5].tolist())


def _energies(inp, a, b):
    for s in range(inp.n_sub):
        r = slice(inp.offsets[s], inp.offsets[s] + a.nbound[s])
        assert np.array_equal(a.energy[r], b.energy[r]), s


def _both(unbinder, inp, prm, call="unbind", **kw):
    got = getattr(unbinder, call)(inp, prm, **kw)
    unbinder.count_interactions(True)
    try:
        ref = getattr(unbinder, call)(inp, prm, **kw)
    finally:
        unbinder.count_interactions(False)
    _same(got, ref)
    _energies(inp, got, ref)
    return got


@pytest.mark.parametrize("n", [20, 33, 64, 257, 1023, 1025, 2047, 2049, 4100, 30_000])
def test_one_halo(unbinder, n):
    inp = synthetic.nfw_single(n=n, seed=n, interloper_frac=0.3, interloper_speed=1.3)
    out = _both(unbinder, inp, abi.parity_params(dm_only=1, box_size=100.0))
    assert out.nbound[0] > 0 or n < 64  # the smallest disrupt, in both


@pytest.mark.parametrize("seed", [0, 1])
def test_edge_cases_and_wrapped_haloes(unbinder, seed):
    _both(unbinder, synthetic.small_cases(seed=seed), abi.parity_params(dm_only=1, box_size=100.0))


@pytest.mark.parametrize("n_sub, nmax", [(60, 900), (25, 8000), (1900, 60)])
def test_batches(unbinder, n_sub, nmax):
    inp = synthetic.batched(n_sub=n_sub, seed=n_sub, nmin=20, nmax=nmax)
    assert inp.n_particles <= 65536
    _both(unbinder, inp, abi.parity_params(dm_only=1, box_size=500.0))


def test_the_last_iterations_of_a_large_batch(unbinder):
    """Lock step first, teams once 65,536 bound particles are left."""
    inp = synthetic.stripped(n_sub=1500, seed=9, nmax=100_000)
    assert inp.n_particles > 2 * 65536
    _both(unbinder, inp, abi.parity_params(dm_only=1, box_size=500.0))


@pytest.mark.parametrize("max_sample", [0, 100, 1000])
def test_species_and_subsamples(unbinder, max_sample):
    inp = synthetic.hydro(seed=4, n_sub=14, nmin=100, nmax=4000, box=200.0)
    prm = abi.parity_params(thermal=1, box_size=200.0, max_sample_size=max_sample, prepared_subsample=1)
    _both(unbinder, inp, prm)


def test_hubble_flow_and_open_box(unbinder):
    inp = synthetic.batched(n_sub=30, seed=3, nmin=50, nmax=2000)
    _both(unbinder, inp, abi.parity_params(dm_only=1, box_size=500.0, hubble=5.0, scale_factor=0.7))
    _both(unbinder, inp, abi.parity_params(dm_only=1, box_size=500.0, periodic=0))


@pytest.mark.parametrize("limit", [1, 2, 5])
def test_bounded_iterations(unbinder, limit):
    inp = synthetic.stripped(n_sub=40, seed=2, nmax=3000)
    _both(unbinder, inp, abi.parity_params(dm_only=1, box_size=500.0, max_iterations=limit), allow_max_iter=True)


def test_near_coincident_particles_return_to_lock_step(unbinder):
    """Pairs far closer than their neighbours: chains of single-child cells fill a team's tree slots."""
    inp = synthetic.nfw_single(n=1800, seed=8)
    half = inp.n_particles // 2
    inp.pos[half:2 * half] = inp.pos[:half] + np.float32(1e-5)
    prm = abi.parity_params(dm_only=1, box_size=100.0, softening=1e-4)
    _both(unbinder, inp, prm)


def test_warm_start(unbinder):
    learned.Model.load().install(unbinder)
    inp = synthetic.stripped(n_sub=60, seed=12, nmax=4000)
    _both(unbinder, inp, abi.parity_params(dm_only=1, box_size=500.0), call="unbind_learned")
