"""What a program that uses this framework has it do, as cases that can be timed and compared.

listed() names the cases, draw(rng) gives more of the same ranges, prepare(case, seed) makes what the program
has in hand before the call, run(state) makes the call through the public entry points, work(case) counts the
bytes and operations that the call cannot do without, and exact(case, seed) gives its result in 64 bits where
that has one.

Every input is synthetic, with the shapes, sizes and value distributions of hbtg.synthetic (NFW haloes with
isotropic Jeans velocities), made on the GPU so that a batch of 5e7 particles takes a fraction of a second.
One library handle serves the process, as one per host thread does in a program.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "hbt-herons_gb300"))

from hbtg import abi, gpu, learned, synthetic  # noqa: E402

DEV = "cuda:0"
HALO_BOX = 500.0  # the batched workloads' periodic box
FLOPS = 13  # per interaction of the tree walk: 3 sub, 5 for r^2, 2 opening test, 1 rsqrt, 2 accumulate


# ---------------------------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------------------------
def listed():
    return [
        # one resolved subhalo through the host-pointer call, as the C++ shim makes it for Subhalo_t::Unbind:
        # the smallest call, all launches and latency
        dict(name="host one subhalo 300", kind="host_one", n=300),
        # one massive halo with 10 % interlopers on the GPU: the single-halo configuration
        dict(name="one halo 1e5", kind="one", n=100_000),
        # a snapshot's subhaloes in one plain call: the reference's own method, batched
        dict(name="batched plain 5e6", kind="plain", n=5_000_000),
        # the benchmark's workload, warm-started by the proposer network: the largest call
        dict(name="batched learned 5e7", kind="learned", n=50_000_000),
        # a hydrodynamical snapshot: four species, thermal energies, tracer types
        dict(name="hydro learned 4e6", kind="hydro_learned", n=4_000_000),
        # tidally stripped subhaloes with what the previous output knew of them
        dict(name="stripped learned 3e6", kind="stripped", n=3_000_000),
        # the production configuration: potentials from subsamples of 1000 particles, most-bound refinement
        dict(name="subsampled hydro 1e6", kind="subsampled", n=1_000_003, sample=1000),
        # the literal 20,000 subhaloes end to end from pinned host arrays, copies included
        dict(name="host learned 20000", kind="host_learned", n=5_900_000),
        # the tree potential of one host halo that straddles a face of its periodic box
        dict(name="potential wrapped 2e5", kind="potential", n=200_003, targets=200_003, wrap=True),
        # profiles, shapes and truncation after unbinding
        dict(name="properties 5e6", kind="properties", n=5_000_000),
        # gas reassignment before unbinding, ten neighbours, FoF groups of a host and its satellites
        dict(name="reassign 3e5", kind="reassign", n=300_000, groups=40, k=10),
        # one gradient of the proposer's training: forward and backward over a mini-batch
        dict(name="train gradient 65536", kind="train", n=65_536, weighted=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host_one", "one", "plain", "learned", "hydro", "hydro_learned", "stripped", "subsampled",
                       "host_learned", "potential", "properties", "reassign", "train"])
    if kind == "host_one":
        return dict(kind=kind, n=_log_int(rng, 30, 20_000))
    if kind == "one":
        return dict(kind=kind, n=_log_int(rng, 2_000, 1_000_000))
    if kind in ("plain", "learned"):
        return dict(kind=kind, n=_log_int(rng, 20_000, 20_000_000))
    if kind in ("hydro", "hydro_learned"):
        return dict(kind=kind, n=_log_int(rng, 20_000, 6_000_000))
    if kind == "stripped":
        return dict(kind=kind, n=_log_int(rng, 20_000, 6_000_000))
    if kind == "subsampled":
        return dict(kind=kind, n=_log_int(rng, 20_000, 2_000_000), sample=rng.choice([500, 1000, 2000]))
    if kind == "host_learned":
        return dict(kind=kind, n=_log_int(rng, 20_000, 6_000_000))
    if kind == "potential":
        n = _log_int(rng, 500, 2_000_000)
        return dict(kind=kind, n=n, targets=rng.choice([n, max(1, n // 7)]), wrap=rng.choice([True, False]))
    if kind == "properties":
        return dict(kind=kind, n=_log_int(rng, 20_000, 10_000_000))
    if kind == "reassign":
        n = _log_int(rng, 20_000, 600_000)
        return dict(kind=kind, n=n, groups=rng.randrange(4, 81), k=rng.choice([1, 5, 10, 32]))
    return dict(kind=kind, n=_log_int(rng, 1_000, 1_000_000), weighted=rng.choice([True, False]))


# ---------------------------------------------------------------------------------------------------------
# Synthetic subhaloes on the GPU
# ---------------------------------------------------------------------------------------------------------
_KEEP = {}


def _unbinder():
    """The process's library handle, with the shipped proposer installed."""
    if "u" not in _KEEP:
        u = gpu.Unbinder(0)
        learned.Model.load().install(u)
        _KEEP["u"] = u
    return _KEEP["u"]


def _table():
    """The NFW tables of hbtg.synthetic on the GPU."""
    if "t" not in _KEEP:
        T = synthetic._tables()
        g = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        _KEEP["t"] = (g(T.mx), g(T.x), g(np.log(T.x)), g(T.f))
    return _KEEP["t"]


def _interp(q, x, y):
    i = torch.searchsorted(x, q.contiguous()).clamp_(1, len(x) - 1)
    x0, x1, y0, y1 = x[i - 1], x[i], y[i - 1], y[i]
    return y0 + ((q - x0) / (x1 - x0)).clamp_(0, 1) * (y1 - y0)


def _m(x):
    return np.log1p(x) - x / (1 + x)


def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _directions(g, n):
    v = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


def _counts(total, nmin, nmax):
    """Subhalo sizes N^-1.9 on [nmin, nmax], `total` particles in all: the case's own, whatever the seed, so that
    the outputs keep their shapes."""
    rng = np.random.default_rng(total)
    nmax = max(nmin, min(nmax, total // 3))
    c = synthetic._power_law_counts(rng, nmin, nmax, 1.9, total=total)
    over = int(c.sum()) - total
    while over > 0:  # the last subhaloes lose what is too much; one left with too few joins the one before
        c[-1] -= over
        over = 0
        if c[-1] < nmin and len(c) > 1:
            c[-2] += c[-1]
            c = c[:-1]
            over = int(c.sum()) - total
    return c.astype(np.int64)


def _nfw(g, counts, conc, cut):
    """Positions about the centre and velocities of NFW haloes cut at `cut` r_200."""
    mx, xs, lnx, f = _table()
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(DEV)  # noqa: E731
    n = int(counts.sum())
    seg = torch.repeat_interleave(torch.arange(len(counts), device=DEV), torch.from_numpy(counts).to(DEV))
    m200 = counts * _m(conc) / _m(conc * cut)
    r200 = synthetic.r200_of(m200)
    x = _interp(_rand(g, n) * to(_m(conc * cut))[seg], mx, xs).clamp_(min=1e-7)
    rs = to(r200 / conc)[seg]
    pos = _directions(g, n) * (x * rs)[:, None]
    vs2 = to(m200 / (r200 / conc) / _m(conc))[seg]
    vel = torch.randn(n, 3, generator=g, device=DEV, dtype=torch.float64)
    vel *= (vs2 * _interp(x.log(), lnx, f)).sqrt()[:, None]
    return dict(pos=pos, vel=vel, seg=seg, x=x, rs=rs, vs2=vs2, r200=r200, m200=m200, n=n)


def _heat(g, h, heat, lo, hi, interlopers=False):
    """Gives a fraction `heat` of each halo a speed of U(lo, hi) v_esc in a random direction."""
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(DEV)  # noqa: E731
    hot = _rand(g, h["n"]) < to(heat)[h["seg"]]
    x = h["x"]
    if interlopers:  # anywhere within 2 r_200
        r = 2 * to(h["r200"])[h["seg"]] * _rand(g, h["n"]) ** (1 / 3)
        h["pos"] = torch.where(hot[:, None], _directions(g, h["n"]) * r[:, None], h["pos"])
        x = torch.where(hot, (r / h["rs"]).clamp(min=1e-7), x)
    esc = (2 * h["vs2"] * torch.log1p(x) / x).sqrt() * (lo + (hi - lo) * _rand(g, h["n"]))
    h["vel"] = torch.where(hot[:, None], _directions(g, h["n"]) * esc[:, None], h["vel"])


def _batch(g, rng, h, counts, box, centre=None, mass=None, type_=None, u=None, prior=None):
    """The subhaloes as device tensors in the library's layout, with the initial frames: the mean position
    about the first particle and the mean velocity (in fixed point, so that they are the same every time)."""
    ns, n, seg = len(counts), h["n"], h["seg"]
    offsets = np.zeros(ns + 1, np.int64)
    np.cumsum(counts, out=offsets[1:])
    centre = rng.random((ns, 3)) * box if centre is None else centre
    bulk = rng.standard_normal((ns, 3)) * 50.0
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(DEV)  # noqa: E731
    pos = (h["pos"] + to(centre)[seg]).remainder_(box).float()
    pos[pos >= box] = 0.0
    vel = (h["vel"] + to(bulk)[seg]).float()
    mass = torch.ones(n, device=DEV) if mass is None else mass
    first = torch.from_numpy(offsets[:-1]).to(DEV)
    m = mass.double()
    d = pos.double() - pos[first].double()[seg]
    d = d - box * torch.round(d / box)

    def mean(v, scale):
        q = torch.zeros(ns, 3, dtype=torch.int64, device=DEV)
        q.index_add_(0, seg, (v * m[:, None] * scale).round().long())
        w = torch.zeros(ns, dtype=torch.int64, device=DEV)
        w.index_add_(0, seg, (m * 65536.0).round().long())
        return q.double() / scale / (w.double() / 65536.0)[:, None]

    b = dict(offsets=offsets, n=n, ns=ns, pos=pos, vel=vel, mass=mass, type=type_, u=u)
    b["id"] = torch.randperm(n, generator=g, device=DEV) * 7 + 11
    b["ref_pos"] = (mean(d, 2.0 ** 32) + pos[first].double()).float()
    b["ref_vel"] = mean(vel.double(), 2.0 ** 26).float()
    b["mb_pos"], b["mb_vel"], b["mb_id"] = pos[first].clone(), vel[first].clone(), b["id"][first].clone()
    b["prior_n"], b["prior_e"] = prior if prior is not None else (None, None)
    return b


def _one_batch(n, seed, box=100.0):
    """One c = 10 halo whose outskirts hold 10 % interlopers at three times the escape speed."""
    rng, g = np.random.default_rng(seed), _generator(seed)
    counts, conc = np.array([n], np.int64), np.array([10.0])
    h = _nfw(g, counts, conc, 2.0)
    _heat(g, h, np.array([0.1]), 3.0, 3.0, interlopers=True)
    return _batch(g, rng, h, counts, box)


def _plain_batch(total, seed):
    """N^-1.9 on [20, 1e6], c ~ logN(ln 8, 0.3), up to half of each heated to 1.5-4 v_esc."""
    rng, g = np.random.default_rng(seed), _generator(seed)
    counts = _counts(total, 20, 1_000_000)
    conc = np.exp(rng.normal(np.log(8.0), 0.3, len(counts)))
    h = _nfw(g, counts, conc, 2.0)
    _heat(g, h, rng.uniform(0, 0.5, len(counts)), 1.5, 4.0)
    return _batch(g, rng, h, counts, HALO_BOX)


def _hydro_batch(total, seed):
    """55 % dark matter, 35 % gas (thermal energy), 9.9 % stars (concentrated), 0.1 % black holes."""
    rng, g = np.random.default_rng(seed), _generator(seed)
    counts = _counts(total, 100, 200_000)
    conc = np.exp(rng.normal(np.log(8.0), 0.3, len(counts)))
    h = _nfw(g, counts, conc, 2.0)
    _heat(g, h, rng.uniform(0, 0.3, len(counts)), 1.5, 4.0)
    t = _rand(g, h["n"])
    type_ = torch.full((h["n"],), 1, dtype=torch.uint8, device=DEV)
    type_[t < 0.35] = 0
    type_[(t >= 0.35) & (t < 0.449)] = 4
    type_[(t >= 0.449) & (t < 0.45)] = 5
    mass = torch.ones(h["n"], device=DEV)
    mass[(type_ == 0) | (type_ == 4)] = 0.19
    mass[type_ == 5] = 50.0
    h["pos"] = torch.where((type_ == 4)[:, None], h["pos"] * 0.2, h["pos"])  # the stars sit deep inside
    h["pos"] = torch.where((type_ == 5)[:, None], h["pos"] * 0.01, h["pos"])
    sig2 = torch.from_numpy(h["m200"] / h["r200"] / 2).to(DEV)[h["seg"]]
    u = 0.3 * sig2 * torch.exp(0.5 * torch.randn(h["n"], generator=g, device=DEV, dtype=torch.float64))
    u = torch.where(type_ == 0, u, torch.zeros_like(u)).float()
    return _batch(g, rng, h, counts, HALO_BOX, mass=mass, type_=type_, u=u)


def _stripped_batch(total, seed):
    """Remnants cut at U(0.2, 1.5) r_200, up to 60 % of each kicked by 0.2-1.5 v_esc; the previous output's
    bound set (5 % of it wrong) comes first in each subhalo, with its binding energies."""
    rng, g = np.random.default_rng(seed), _generator(seed)
    counts = _counts(total, 20, 1_000_000)
    conc = np.exp(rng.normal(np.log(8.0), 0.3, len(counts)))
    cut = rng.uniform(0.2, 1.5, len(counts))
    h = _nfw(g, counts, conc, cut)
    phi = -h["vs2"] * torch.log1p(h["x"]) / h["x"]
    e = 0.5 * h["vel"].square().sum(1) + phi
    prev = (e < 0) ^ (_rand(g, h["n"]) < 0.05)
    kick = _rand(g, h["n"]) < torch.from_numpy(rng.uniform(0, 0.6, len(counts))).to(DEV)[h["seg"]]
    dv = _directions(g, h["n"]) * ((0.2 + 1.3 * _rand(g, h["n"])) * (-2 * phi).sqrt())[:, None]
    h["vel"] = torch.where(kick[:, None], h["vel"] + dv, h["vel"])
    order = torch.sort(h["seg"] * 2 + (~prev).long(), stable=True).indices
    nprev = torch.zeros(len(counts), dtype=torch.int64, device=DEV).index_add_(0, h["seg"], prev.long())
    h["pos"], h["vel"], e = h["pos"][order], h["vel"][order], e[order]
    return _batch(g, rng, h, counts, HALO_BOX, prior=(nprev, e.float()))


def _group_batch(total, groups, seed):
    """FoF groups of a host and three satellites inside it, four species; a tenth of the gas particles are
    listed under another subhalo of their group."""
    rng, g = np.random.default_rng(seed), _generator(seed)
    per = 4
    size = np.random.default_rng(total)  # the sizes are the case's own
    share = np.exp(size.normal(0, 0.6, groups))
    share = share / share.sum() * total
    host = np.maximum(200, 0.7 * share).astype(np.int64)
    sats = np.maximum(50, (0.3 / 3) * share[:, None] * size.uniform(0.3, 1.7, (groups, 3))).astype(np.int64)
    counts = np.concatenate([host[:, None], sats], 1).reshape(-1)
    conc = np.exp(rng.normal(np.log(8.0), 0.3, len(counts)))
    h = _nfw(g, counts, conc, 2.0)
    centre = rng.random((groups, 1, 3)) * HALO_BOX + np.zeros((1, per, 1))
    r200 = h["r200"].reshape(groups, per)
    away = rng.standard_normal((groups, 3, 3))
    centre[:, 1:] += away / np.linalg.norm(away, axis=2, keepdims=True) * (r200[:, :1] * rng.uniform(
        0.2, 1.0, (groups, 3)))[:, :, None]
    t = _rand(g, h["n"])
    type_ = torch.full((h["n"],), 1, dtype=torch.uint8, device=DEV)
    type_[t < 0.35] = 0
    type_[(t >= 0.35) & (t < 0.449)] = 4
    type_[(t >= 0.449) & (t < 0.45)] = 5
    pos = (h["pos"] + torch.from_numpy(centre.reshape(-1, 3)).to(DEV)[h["seg"]]).remainder_(HALO_BOX).float()
    pos[pos >= HALO_BOX] = 0.0
    swap = (type_ == 0) & (_rand(g, h["n"]) < 0.1)
    other = (h["seg"] // per) * per + (h["seg"] % per + 1 + (_rand(g, h["n"]) * 3).long().clamp(max=2)) % per
    seg, order = torch.sort(torch.where(swap, other, h["seg"]), stable=True)
    sizes = torch.bincount(seg, minlength=len(counts)).cpu().numpy()
    offsets = np.zeros(len(counts) + 1, np.int64)
    np.cumsum(sizes, out=offsets[1:])
    return dict(n=h["n"], ns=len(counts), offsets=offsets, pos=pos[order].contiguous(), type=type_[order].contiguous(),
                group_off=np.arange(0, len(counts) + 1, per, dtype=np.int64))


# ---------------------------------------------------------------------------------------------------------
# Calls
# ---------------------------------------------------------------------------------------------------------
IN_OUT = ("ref_pos", "ref_vel", "mb_pos", "mb_vel", "mb_id")


def _p(t):
    return None if t is None else t.data_ptr()


def _device_call(b):
    """Output tensors of a device-pointer call on batch b, and the call's descriptor."""
    n, ns = b["n"], b["ns"]
    z = lambda shape, dt: torch.zeros(shape, dtype=dt, device=DEV)  # noqa: E731
    o = dict(ref_pos=z((ns, 3), torch.float32), ref_vel=z((ns, 3), torch.float32), mb_pos=z((ns, 3), torch.float32),
             mb_vel=z((ns, 3), torch.float32), mb_id=z(ns, torch.int64), order=z(n, torch.int64),
             nbound=z(ns, torch.int64), mbound=z(ns, torch.float32), nbound_type=z((ns, 6), torch.int64),
             mbound_type=z((ns, 6), torch.float32), tracer=z(ns, torch.int64), kin=z((ns, 5), torch.float32),
             core=z((ns, 8), torch.float32), energy=z(n, torch.float32), iterations=z(ns, torch.int32),
             status=z(ns, torch.int32))
    c = abi.CBatch(ns, b["offsets"].ctypes.data, _p(b["pos"]), _p(b["vel"]), _p(b["mass"]), _p(b["u"]), _p(b["id"]),
                   _p(b["type"]), _p(o["ref_pos"]), _p(o["ref_vel"]), _p(o["mb_pos"]), _p(o["mb_vel"]), _p(o["mb_id"]),
                   _p(o["order"]), _p(o["nbound"]), _p(o["mbound"]), _p(o["nbound_type"]), _p(o["mbound_type"]),
                   _p(o["tracer"]), _p(o["kin"]), _p(o["core"]), _p(o["energy"]), None, _p(o["iterations"]),
                   _p(o["status"]))
    return o, c


def _host_call(b, pinned):
    """Host arrays of batch b with a host-pointer call's descriptor (pinned: page-locked, as a program that
    wants the full copy rate holds them)."""
    keep = []

    def host(t):
        if t is None:
            return None
        c = t.cpu()
        c = c.pin_memory() if pinned else c
        keep.append(c)
        return c

    n, ns = b["n"], b["ns"]
    z = lambda *shape, dt: host(torch.zeros(shape, dtype=dt))  # noqa: E731
    i = {k: host(b[k]) for k in ("pos", "vel", "mass", "u", "id", "type", "prior_n", "prior_e") + IN_OUT}
    o = {k: host(b[k].clone()) for k in IN_OUT}
    o.update(order=z(n, dt=torch.int64), nbound=z(ns, dt=torch.int64), mbound=z(ns, dt=torch.float32),
             nbound_type=z(ns, 6, dt=torch.int64), mbound_type=z(ns, 6, dt=torch.float32),
             tracer=z(ns, dt=torch.int64), kin=z(ns, 5, dt=torch.float32), core=z(ns, 8, dt=torch.float32),
             energy=z(n, dt=torch.float32), iterations=z(ns, dt=torch.int32), status=z(ns, dt=torch.int32))
    c = abi.CBatch(ns, b["offsets"].ctypes.data, _p(i["pos"]), _p(i["vel"]), _p(i["mass"]), _p(i["u"]), _p(i["id"]),
                   _p(i["type"]), _p(o["ref_pos"]), _p(o["ref_vel"]), _p(o["mb_pos"]), _p(o["mb_vel"]), _p(o["mb_id"]),
                   _p(o["order"]), _p(o["nbound"]), _p(o["mbound"]), _p(o["nbound_type"]), _p(o["mbound_type"]),
                   _p(o["tracer"]), _p(o["kin"]), _p(o["core"]), _p(o["energy"]), None, _p(o["iterations"]),
                   _p(o["status"]))
    return i, o, c, keep


def _params(case):
    k = case["kind"]
    if k in ("host_one", "one"):
        return abi.parity_params(dm_only=1, box_size=100.0)
    if k in ("hydro", "hydro_learned"):
        return abi.parity_params(thermal=1, box_size=HALO_BOX)
    if k == "subsampled":
        return abi.parity_params(thermal=1, box_size=HALO_BOX, max_sample_size=case["sample"], prepared_subsample=1)
    if k == "potential":
        return abi.parity_params(dm_only=1, box_size=100.0)
    if k == "properties":  # a Hubble rate that puts R200 inside the haloes
        return abi.parity_params(dm_only=1, box_size=HALO_BOX, hubble=25.0)
    if k == "reassign":
        return abi.parity_params(box_size=HALO_BOX)
    return abi.parity_params(dm_only=1, box_size=HALO_BOX)


def _host_halo(n, seed, n_tgt, wrap):
    """A c = 5 host in a 100-unit box, cut by a face of it (wrap) or not, and the particles whose potential is
    asked for."""
    g = _generator(seed)
    counts, conc = np.array([n], np.int64), np.array([5.0])
    h = _nfw(g, counts, conc, 2.0)
    c = np.array([[0.3 * h["r200"][0] if wrap else 50.0, 50.0, 50.0]])
    pos = (h["pos"] + torch.from_numpy(c).to(DEV)).remainder_(100.0).float()
    pos[pos >= 100.0] = 0.0
    mass = (0.5 + _rand(g, n)).float()
    tgt = torch.arange(n, device=DEV) if n_tgt == n else torch.randperm(n, generator=g, device=DEV)[:n_tgt]
    return pos.contiguous(), mass, tgt.contiguous()


def prepare(case, seed):
    k, n = case["kind"], case["n"]
    s = dict(kind=k, params=_params(case))
    if k == "train":
        g = _generator(seed)
        # the ranges of the six features, labels that mostly follow them, weights as training starts from
        f = torch.randn(n, 6, generator=g, device=DEV)
        f = torch.stack([f[:, 0].abs(), 2 * f[:, 1].abs(), 3 * f[:, 2], f[:, 3], f[:, 4].sign(),
                         torch.zeros(n, device=DEV)], 1).contiguous()
        s["features"] = f
        s["labels"] = ((f[:, 2] + 0.3 * torch.randn(n, generator=g, device=DEV)) < 0).float()
        s["weights"] = torch.from_numpy(learned.initial_weights(seed % 1000)).to(DEV)
        s["sample_weights"] = torch.rand(n, generator=g, device=DEV) if case["weighted"] else None
        return s
    u = s["u"] = _unbinder()
    if k == "potential":
        s["pos"], s["mass"], s["tgt"] = _host_halo(n, seed, case["targets"], case["wrap"])
        s["out"] = torch.zeros(len(s["tgt"]), device=DEV)
        return s
    if k == "reassign":
        b = s["b"] = _group_batch(n, case["groups"], seed)
        s["dest"] = torch.full((b["n"],), -1, dtype=torch.int64, device=DEV)
        s["c"] = abi.CReassign(len(b["group_off"]) - 1, b["group_off"].ctypes.data, b["ns"], b["offsets"].ctypes.data,
                               _p(b["pos"]), _p(b["type"]), _p(s["dest"]))
        s["k"] = case["k"]
        return s
    if k in ("host_one", "one"):
        b = _one_batch(n, seed)
    elif k in ("hydro", "hydro_learned", "subsampled"):
        b = _hydro_batch(n, seed)
    elif k == "stripped":
        b = _stripped_batch(n, seed)
    else:
        b = _plain_batch(n, seed)
    s["b"] = b
    if k == "subsampled":  # PrepareParticlesForSubsampling, which the program runs before the call
        perm = np.zeros(b["n"], np.int64)
        types = b["type"].cpu().numpy()
        c = abi.CBatch(b["ns"], b["offsets"].ctypes.data)
        c.type = types.ctypes.data
        f = u.lib.hbtg_prepare_subsampling
        f.argtypes = [ctypes.c_void_p] * 3
        if f(ctypes.byref(s["params"]), ctypes.byref(c), perm.ctypes.data) != 0:
            raise RuntimeError("hbtg_prepare_subsampling")
        seg = np.repeat(np.arange(b["ns"]), np.diff(b["offsets"]))
        rows = torch.from_numpy(perm + b["offsets"][:-1][seg]).to(DEV)
        for q in ("pos", "vel", "mass", "u", "type", "id"):
            b[q] = b[q][rows].contiguous()
    if k in ("host_one", "host_learned"):
        s["i"], s["o"], s["c"], s["keep"] = _host_call(b, pinned=k == "host_learned")
        s["b"] = dict(offsets=b["offsets"])
        s["prior"] = abi.CPrior(None, None)
        return s
    s["o"], s["c"] = _device_call(b)
    s["prior"] = abi.CPrior(_p(b["prior_n"]), _p(b["prior_e"]))
    if k == "properties":  # the bound sets that the unbinding of these subhaloes gives
        for q in IN_OUT:
            s["o"][q].copy_(b[q])
        u.unbind_device(abi.parity_params(dm_only=1, box_size=HALO_BOX), s["c"])
        ns = b["ns"]
        s["p"] = {q: torch.zeros(ns, device=DEV) for q in abi.PROPS_FLOAT}
        s["p"].update(snap_last=torch.full((ns,), -1, dtype=torch.int32, device=DEV),
                      inertia=torch.zeros(ns, 6, device=DEV), inertia_w=torch.zeros(ns, 6, device=DEV),
                      nsource=torch.zeros(ns, dtype=torch.int64, device=DEV))
        s["cp"] = abi.CProps(*[_p(s["p"][q]) for q, _ in abi.CProps._fields_])
        f = u.lib.hbtg_subhalo_properties_device
        f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int32, ctypes.c_double, ctypes.c_void_p, ctypes.c_void_p]
    return s


def _ok(rc, what):
    if rc not in (0, 4):
        raise gpu.UnbindError(rc, what)


def run(s):
    k, prm = s["kind"], s["params"]
    if k == "train":
        return learned.mlp_backward(s["weights"], s["features"], s["labels"], s["sample_weights"])
    u = s["u"]
    stream = torch.cuda.current_stream().cuda_stream
    if k == "potential":
        _ok(u.lib.hbtg_tree_potential_device(u.h, ctypes.byref(prm), len(s["mass"]), _p(s["pos"]), _p(s["mass"]),
                                             len(s["tgt"]), _p(s["tgt"]), _p(s["out"]), stream), "tree potential")
        return s["out"]
    if k == "reassign":
        f = u.lib.hbtg_reassign_particles_device
        _ok(f(u.h, ctypes.byref(prm), ctypes.byref(s["c"]), ctypes.c_int(s["k"]), ctypes.c_void_p(stream)), "reassign")
        return s["dest"]
    if k == "properties":
        for q in ("r200", "m200", "last_vmax", "rmax_last"):  # the in/out members start from what they were
            s["p"][q].zero_()
        s["p"]["snap_last"].fill_(-1)
        _ok(u.lib.hbtg_subhalo_properties_device(u.h, ctypes.byref(prm), ctypes.byref(s["c"]), 1, 3.0,
                                                 ctypes.byref(s["cp"]), stream), "properties")
        return s["p"]
    if k in ("host_one", "host_learned"):
        for q in IN_OUT:  # the in/out frames start from the inputs
            s["o"][q].copy_(s["i"][q])
        if k == "host_one":
            u.unbind_raw(prm, s["c"])
            s["o"]["energy"][int(s["o"]["nbound"][0]):] = 0.0  # only the bound particles' energies are written
            return s["o"]
        _ok(u.lib.hbtg_unbind_batch_learned(u.h, ctypes.byref(prm), ctypes.byref(s["c"]), ctypes.byref(s["prior"])),
            "hbtg_unbind_batch_learned")
        # the energies are copied back too, but those past each bound set are not the call's: left out here
        return {q: v for q, v in s["o"].items() if q != "energy"}
    for q in IN_OUT:
        s["o"][q].copy_(s["b"][q])
    if k in ("learned", "hydro_learned", "stripped"):
        _ok(u.lib.hbtg_unbind_batch_learned_device(u.h, ctypes.byref(prm), ctypes.byref(s["c"]),
                                                   ctypes.byref(s["prior"]), stream), "learned")
    else:
        u.unbind_device(prm, s["c"], stream)
    return s["o"]


# ---------------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------------------------------------
def _interactions(n, total, nmin, nmax):
    """Interactions of one evaluation of every particle: about min(N, 95 log2 N - 400) of a subhalo of N (the
    opening angle 0.45), averaged over the particles of N^-1.9 sizes on [nmin, nmax]."""
    one = lambda N: np.minimum(N, np.maximum(95 * np.log2(N) - 400, 64))  # noqa: E731
    if nmin == nmax:
        return total * float(one(np.array(float(nmin))))
    N = np.exp(np.linspace(math.log(nmin), math.log(max(nmin + 1, min(nmax, total))), 400))
    w = N ** -0.9 * N  # particles per log N
    return total * float((w * one(N)).sum() / w.sum())


def work(case):
    k, n = case["kind"], case["n"]
    if k == "train":  # forward, backward and weight gradients of the 6-64-64-1 network
        return {"bytes": n * 4 * (6 + 1 + case["weighted"]) + 2 * 4 * 4673, "flops": 6 * n * (6 * 64 + 64 * 64 + 64)}
    if k == "potential":
        t = case["targets"]
        return {"bytes": 16 * n + 12 * t, "flops": FLOPS * _interactions(n, t, n, n)}
    if k == "properties":  # positions, masses, order in; nine floats of each subhalo out
        return {"bytes": 24 * n, "flops": 40 * n}
    if k == "reassign":  # 45 % of the particles look up k neighbours among the others
        return {"bytes": 21 * n, "flops": 0.36 * n * 8 * 30 * case["k"]}
    # pos, vel, mass, id in; order, energy out; species, thermal energies and priors where there are any
    bytes_ = n * (12 + 12 + 4 + 8 + 8 + 4)
    bytes_ += n * 5 if k in ("hydro", "hydro_learned", "subsampled") else 0
    bytes_ += n * 4 if k == "stripped" else 0
    if k in ("host_one", "one"):
        inter = _interactions(n, n, n, n)
    elif k == "subsampled":
        inter = n * 600.0
    elif k in ("hydro", "hydro_learned"):
        inter = _interactions(n, n, 100, 200_000)
    else:
        inter = _interactions(n, n, 20, 1_000_000)
    return {"bytes": bytes_, "flops": FLOPS * inter}


# ---------------------------------------------------------------------------------------------------------
# In 64 bits
# ---------------------------------------------------------------------------------------------------------
def _exact_potential(case, seed):
    """The direct sum over all particles with the cubic-spline softening."""
    prm = _params(case)
    pos, mass, tgt = _host_halo(case["n"], seed, case["targets"], case["wrap"])
    pos, mass = pos.double(), mass.double()
    box, h = float(np.float32(prm.box_size)), 2.8 * float(np.float32(prm.softening))
    out = torch.zeros(len(tgt), dtype=torch.float64, device=DEV)
    step = max(1, 30_000_000 // len(mass))
    for a in range(0, len(tgt), step):
        t = tgt[a:a + step]
        r2 = torch.zeros(len(t), len(mass), dtype=torch.float64, device=DEV)
        for d in range(3):
            x = pos[t, d][:, None] - pos[None, :, d]
            if case["wrap"]:
                x -= box * torch.round(x / box)
            r2 += x * x
        near = r2 < h * h
        w = r2.rsqrt().neg_()
        i, j = torch.nonzero(near, as_tuple=True)
        v = r2[i, j].sqrt() / h
        inner = -2.8 + v * v * (16 / 3 + v * v * (6.4 * v - 9.6))
        outer = -3.2 + (1 / 15) / v + v * v * (32 / 3 + v * (-16 + v * (9.6 - 32 / 15 * v)))
        w[i, j] = torch.where(v < 0.5, inner, outer) / h
        w[torch.arange(len(t), device=DEV), t] = 0  # not itself
        out[a:a + step] = w @ mass
    return out * (prm.G / prm.scale_factor)


def _exact_gradient(case, seed):
    s = prepare(case, seed)
    w = s["weights"].double().requires_grad_()
    at, parts = 0, []
    for _, size in learned.LAYERS:
        parts.append(w[at:at + size])
        at += size
    W1, b1, W2, b2, w3, b3 = parts
    x, y = s["features"].double(), s["labels"].double()
    z = torch.relu(torch.relu(x @ W1.view(6, 64) + b1) @ W2.view(64, 64) + b2) @ w3 + b3
    losses = torch.nn.functional.binary_cross_entropy_with_logits(z, y, reduction="none")
    loss = (losses if s["sample_weights"] is None else losses * s["sample_weights"].double()).sum()
    loss.backward()
    return w.grad, loss.detach().reshape(1)


def _G(s):
    return s["params"].G / s["params"].scale_factor


def _exact_properties(case, seed):
    """The quantities that do not hang on which of two nearly equal radii wins."""
    s = prepare(case, seed)
    b, o = s["b"], s["o"]
    off = torch.from_numpy(b["offsets"]).to(DEV)
    nb = o["nbound"]
    seg = torch.repeat_interleave(torch.arange(b["ns"], device=DEV), nb)
    first = torch.cumsum(nb, 0) - nb
    k = torch.arange(len(seg), device=DEV) - first[seg]
    g = off[:-1][seg] + o["order"][off[:-1][seg] + k]
    d = b["pos"][g].double() - o["mb_pos"][seg].double()
    d -= HALO_BOX * torch.round(d / HALO_BOX)
    m = b["mass"][g].double()
    r = d.square().sum(1).sqrt()
    o1 = torch.sort(r, stable=True).indices
    o2 = o1[torch.sort(seg[o1], stable=True).indices]
    rs, ss = r[o2].clamp(min=float(np.float32(s["params"].softening))), seg[o2]
    has = nb > 1
    last = (first + nb - 1).clamp(min=0)
    half = (first + nb // 2).clamp(max=len(rs) - 1)
    zero = torch.zeros(b["ns"], dtype=torch.float64, device=DEV)
    run_ = torch.cumsum(m[o2], 0)
    base = torch.where(first > 0, run_[(first - 1).clamp(min=0)], zero)
    v = (run_ - base[ss]) / rs
    vmax = torch.zeros(b["ns"], dtype=torch.float64, device=DEV).scatter_reduce_(0, ss, v, "amax")
    q = [d[:, 0] * d[:, 0], d[:, 0] * d[:, 1], d[:, 0] * d[:, 2], d[:, 1] * d[:, 1], d[:, 1] * d[:, 2],
         d[:, 2] * d[:, 2]]
    inner = k > 0
    mb = torch.zeros(b["ns"], dtype=torch.float64, device=DEV).index_add_(0, seg, m)
    inertia = torch.stack([torch.zeros(b["ns"], dtype=torch.float64, device=DEV).index_add_(
        0, seg, torch.where(inner, x * m, torch.zeros_like(m))) for x in q], 1) / mb.clamp(min=1e-30)[:, None]
    w = lambda t: torch.where(has, t, zero)  # noqa: E731
    e = dict.fromkeys([c for c, _ in abi.CProps._fields_])
    e.update(rhalf=w(rs[half]), renclose=w(rs[last]), vmax=w((vmax * _G(s)).sqrt()),
             inertia=torch.where(has[:, None], inertia, torch.zeros_like(inertia)))
    return e


def exact(case, seed):
    """An unbinding has no closed result in 64 bits: which particles stay is decided by the iteration itself."""
    if case["kind"] == "train":
        return _exact_gradient(case, seed)
    if case["kind"] == "properties":
        return _exact_properties(case, seed)
    if case["kind"] == "potential" and case["n"] * case["targets"] <= 5e10:
        return _exact_potential(case, seed)
    return None
