"""Sums that the kernels form in FP32 words hold at least what a sum in double
holds: frames of small subhaloes, shape tensors and the masses behind the
upscale factors, on values whose large terms cancel (or end halfway between two
floats) and whose small ones lie 2^-50 below them.  Every sum here is exact in
double whatever its order, so the expected value has no tolerance."""
import numpy as np
import pytest

from hbtg import abi, oracle, synthetic

pytestmark = pytest.mark.gpu

BIG = np.array([1.9000001, 1.7000002], np.float32)  # their sum is not a float


def _inputs(pos, vel, mass):
    n = len(pos)
    zero = np.zeros((1, 3), np.float32)
    return abi.Inputs(np.array([0, n], np.int64), pos.astype(np.float32), vel.astype(np.float32), mass.astype(np.float32),
                      np.arange(n) + 5, None, None, zero.copy(), zero.copy(), pos[:1].astype(np.float32), zero.copy(),
                      np.array([5], np.int64))


@pytest.mark.parametrize("n", [200, 700, 1500, 9000, 20_000])  # the teams of one block, of a cluster and of the grid
def test_frame_of_a_bound_subhalo(unbinder, n):
    halo = synthetic.nfw_single(n=n, seed=n, interloper_frac=0.0)
    rng = np.random.default_rng(n)
    vel = np.zeros((n, 3))
    vel[:, 0] = rng.integers(0, 1024, n) * 2.0 ** -50
    vel[0:2, 0], vel[32:34, 0] = BIG, -BIG
    inp = _inputs(halo.pos, vel, np.ones(n))
    inp.ref_pos[:] = halo.ref_pos
    out = unbinder.unbind(inp, abi.parity_params(dm_only=1, box_size=100.0))
    assert out.nbound[0] == n
    want = np.float32(inp.vel[:, 0].astype(np.float64).sum() / n)
    assert out.ref_vel[0, 0] == want, (out.ref_vel[0, 0], want)


def test_shape_sums(unbinder):
    n = 700
    rng = np.random.default_rng(1)
    pos = np.zeros((n, 3))
    pos[1:, 0], pos[1:, 1] = rng.integers(0, 1024, n - 1) * 2.0 ** -50, 1.0
    pos[[1, 33], 0], pos[[301, 333], 0] = BIG, -BIG
    inp = _inputs(pos, np.zeros((n, 3)), np.ones(n))
    out = abi.CallBuffers(inp).out  # every particle bound, in input order
    out.order[:], out.nbound[:], out.mbound[:] = np.arange(n), n, n
    prm = abi.parity_params(dm_only=1, box_size=100.0, periodic=0)
    got = unbinder.subhalo_properties(inp, out, prm)
    ref = oracle.subhalo_properties(inp, out, prm)
    assert ref.inertia[0, 1] == np.float32(np.float32((inp.pos[:, 0].astype(np.float64)).sum()) / np.float32(n))
    assert got.inertia[0, 1] == ref.inertia[0, 1], (got.inertia, ref.inertia)


def test_upscale_masses(unbinder):
    """The energies of a subsampled subhalo do not depend on where in its list a particle outside the sample
    stands.  Its mass, with one particle of 2^-48, decides on which side of a halfway point the total lies."""
    n, sample = 3000, 500
    halo = synthetic.nfw_single(n=n, seed=7, interloper_frac=0.0)
    mass = np.full(n, 2.0 ** -13)
    mass[768], mass[800], mass[832] = BIG[0], BIG[1], 2.0 ** -48  # one lane of a warp
    rest = np.delete(mass, 832).sum()
    half = 2.0 ** -23  # of the spacing of floats in [2, 4)
    mass[0] += half * ((1 - round(rest / half)) % 4)  # the total without it: an odd number of halves, down if rounded to even
    total = np.delete(mass, 832).sum()
    assert 2 < total < 4 and round(total / half) % 4 == 1
    prm = abi.parity_params(dm_only=1, box_size=100.0, max_sample_size=sample, prepared_subsample=1)
    energies = []
    for perm in (np.arange(n), np.r_[0:832, 2000, 833:2000, 832, 2001:n]):
        inp = _inputs(halo.pos[perm], np.zeros((n, 3)), mass[perm])
        inp.ref_pos[:] = halo.ref_pos
        out = unbinder.unbind(inp, prm)
        assert out.nbound[0] == n and out.iterations[0] == 1
        e = np.zeros(n, np.float32)
        e[perm[out.order]] = out.energy
        energies.append(e)
    walked = np.arange(n) // 32  # the targets of a warp, whose terms are grouped by what its 32 see
    same = (walked != 832 // 32) & (walked != 2000 // 32)
    assert np.array_equal(energies[0][same], energies[1][same]), (energies[0] != energies[1])[same].sum()
