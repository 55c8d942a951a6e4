"""Performance cases of the gravity path: what a program that uses this
library has it do, through its public entry points.

A case names one kind of call:

* ``force``     one force pass of particles on the device (GravitySimulation.
                start_down), the results left on the device
* ``step``      one Driver::run iteration (run(1)) and the state read back
* ``trip``      host arrays in, one force pass, host accelerations out
* ``periodic``  one force pass of a displaced lattice in a periodic cube
* ``gradient``  a list-recording force pass and its adjoint (host cotangent in,
                host gradients out)
* ``chain``     the gradient through eight leapfrog steps (chain_grad)
* ``density``   the SPH example's density pass
* ``pressure``  the SPH example's density and pressure passes

``exact`` restates the same calls in plain FP64 torch: the octree, the opening
test and the interaction lists, evaluated with dense batches of buckets.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from paratreet_b200.gravity import GravitySimulation, GravityVisitor

DEV = "cuda"
F64 = torch.float64
FIELDS = ("x", "y", "z", "vx", "vy", "vz", "m", "soft")


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest calls (the golden workloads' size): launches and latency
        dict(name="fp64 plummer 4k", kind="force", ics="plummer", n=4096, eps=0.01, precision="fp64",
             bucket=16, theta=0.7),
        # the 10,000-particle Plummer workload in the mixed form
        dict(name="mixed plummer 10k", kind="force", ics="plummer", n=10000, eps=0.01, precision="mixed",
             bucket=16, theta=0.7),
        # ... and as a program that steps it and reads its state every iteration
        dict(name="fp64 step 10k", kind="step", ics="plummer", n=10000, eps=0.01, precision="fp64",
             bucket=16, theta=0.7, dt=0.01),
        # a host program that keeps its particles (odd count) and calls for forces
        dict(name="mixed host trip 100k", kind="trip", ics="mixture", n=100003, eps=1e-3, precision="mixed",
             bucket=32, theta=0.7),
        # the differentiation workload: a recording force pass and its adjoint
        dict(name="gradient hernquist 262k", kind="gradient", ics="hernquist", n=262144, eps=0.01,
             precision="mixed", bucket=16, theta=0.6),
        # eight leapfrog steps differentiated on a smaller halo
        dict(name="chain hernquist 12k", kind="chain", ics="hernquist", n=12345, eps=0.01, precision="mixed",
             bucket=16, theta=0.6, dt=0.005),
        # the reference-exact form on the clumped mixture
        dict(name="fp64 mixture 1m", kind="force", ics="mixture", n=1 << 20, eps=1e-4, precision="fp64",
             bucket=16, theta=0.7),
        # a mid-sized odd count at a smaller opening angle
        dict(name="mixed plummer 1.5m", kind="force", ics="plummer", n=1500007, eps=1e-3, precision="mixed",
             bucket=32, theta=0.5),
        # the headline workload
        dict(name="mixed plummer 16m", kind="force", ics="plummer", n=1 << 24, eps=1e-3, precision="mixed",
             bucket=32, theta=0.7),
        # cosmological initial conditions: 27 replica walks and the Ewald sums
        dict(name="periodic mixed 128^3", kind="periodic", ngrid=128, precision="mixed", bucket=32, theta=0.7),
        # the SPH example's passes
        dict(name="density plummer 1m", kind="density", ics="plummer", n=1000003, eps=1e-3, bucket=32),
        dict(name="pressure plummer 131k", kind="pressure", ics="plummer", n=131072, eps=1e-3, bucket=16),
    ]


def draw(rng):
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) | rng.choice((0, 1))

    kind = rng.choice(("force", "force", "force", "step", "trip", "periodic", "gradient", "chain", "density",
                       "pressure"))
    bucket = rng.choice((8, 12, 16, 24, 32))
    if kind == "periodic":
        return dict(kind=kind, ngrid=rng.randint(24, 128), precision=rng.choice(("mixed", "mixed", "fp64")),
                    bucket=bucket, theta=rng.choice((0.6, 0.7, 0.8)))
    if kind == "density":
        return dict(kind=kind, ics=rng.choice(("plummer", "mixture")), n=size(4000, 2000000), eps=1e-3,
                    bucket=bucket)
    if kind == "pressure":
        return dict(kind=kind, ics=rng.choice(("plummer", "hernquist")), n=size(4000, 260000), eps=1e-3,
                    bucket=bucket)
    ics = rng.choice(("plummer", "mixture", "hernquist"))
    eps = rng.choice((1e-4, 1e-3, 0.01))
    theta = rng.choice((0.5, 0.6, 0.7, 0.8, 1.0))
    case = dict(kind=kind, ics=ics, eps=eps, precision=rng.choice(("mixed", "fp64", "fp64_lists")), bucket=bucket,
                theta=theta)
    if kind == "chain":
        return dict(case, n=size(2000, 30000), eps=0.01, dt=0.005)
    if kind == "gradient":
        return dict(case, n=size(4000, 400000), eps=0.01, theta=rng.choice((0.6, 0.7)))
    if kind == "step":
        return dict(case, n=size(2000, 300000), dt=1e-4)
    if kind == "trip":
        return dict(case, n=size(4000, 1000000))
    return dict(case, n=size(2000, 4000000))


# ---------------------------------------------------------------- particles
def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _uniform(n, g):
    return torch.rand(n, generator=g, device=DEV, dtype=F64)


def _directions(n, g):
    cz = 2.0 * _uniform(n, g) - 1.0
    phi = 2.0 * math.pi * _uniform(n, g)
    sz = torch.sqrt(1.0 - cz * cz)
    return torch.stack([sz * torch.cos(phi), sz * torch.sin(phi), cz])


def _plummer_radii(n, g, a):
    x = _uniform(n, g).clamp_(min=1e-300) * (10.0 ** 3 / (1.0 + 10.0 ** 2) ** 1.5)  # r <= 10 a
    return a / torch.sqrt(x ** (-2.0 / 3.0) - 1.0)


def _positions(case, g):
    n = case["n"]
    if case["ics"] == "plummer":
        return _plummer_radii(n, g, 1.0) * _directions(n, g)
    if case["ics"] == "hernquist":
        s = torch.sqrt(_uniform(n, g)) * (20.0 / 21.0)  # r <= 20 a
        return s / (1.0 - s) * _directions(n, g)
    n_uni = n // 2  # mixture: half uniform, half in 32 clumps
    uni = _uniform(3 * n_uni, g).view(3, -1)
    centres = _uniform(96, g).view(3, 32)
    clump = torch.arange(n - n_uni, device=DEV) % 32
    return torch.cat([uni, centres[:, clump] + _plummer_radii(n - n_uni, g, 0.01) * _directions(n - n_uni, g)], 1)


def _lattice(ngrid, g):
    """ngrid^3 lattice in the unit cube displaced by a P(k) ~ k^-2 field, rms a quarter of a cell."""
    k = torch.fft.fftfreq(ngrid, device=DEV, dtype=F64) * ngrid
    kz = torch.fft.rfftfreq(ngrid, device=DEV, dtype=F64) * ngrid
    ks = torch.meshgrid(k, k, kz, indexing="ij")
    k2 = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
    keep = (ks[0].abs() < ngrid // 2) & (ks[1].abs() < ngrid // 2) & (ks[2] < ngrid // 2) & (k2 > 0)
    amp = torch.where(keep, 1.0 / k2, torch.zeros_like(k2))
    white = torch.fft.rfftn(torch.randn(ngrid, ngrid, ngrid, generator=g, device=DEV, dtype=F64))
    d = torch.stack([torch.fft.irfftn(1j * kk * amp * white, s=(ngrid,) * 3) for kk in ks])
    d *= 0.25 / ngrid / torch.sqrt((d * d).sum(0).mean())
    c = (torch.arange(ngrid, device=DEV, dtype=F64) + 0.5) / ngrid
    grid = torch.stack(torch.meshgrid(c, c, c, indexing="ij"))
    return torch.remainder(grid + d, 1.0).reshape(3, -1)


def _velocities(x, g):
    """Plummer velocities (Aarseth's rejection sampling of q)."""
    n = x.shape[1]
    q, y = _uniform(4 * n + 1000, g), _uniform(4 * n + 1000, g)
    q = q[0.1 * y < q * q * (1.0 - q * q) ** 3.5][:n]
    return q * math.sqrt(2.0) * (1.0 + (x * x).sum(0)) ** -0.25 * _directions(n, g)


def _particles(case, seed):
    """Device tensors x (3, n), v (3, n), m, soft and the generator, from the seed alone."""
    g = _generator(seed)
    x = _lattice(case["ngrid"], g) if case["kind"] == "periodic" else _positions(case, g)
    n = x.shape[1]
    moving = case["kind"] in ("step", "pressure") or case["kind"] == "force" and case["ics"] == "plummer"
    v = _velocities(x, g) if moving else torch.zeros_like(x)
    m = torch.full((n,), 1.0 / n, device=DEV, dtype=F64)
    eps = 0.5 / case["ngrid"] if case["kind"] == "periodic" else case["eps"]
    return x, v, m, torch.full_like(m, eps), g


# ---------------------------------------------------------------- the calls
class State:
    pass


class _Array:
    """A device array of the simulation, which lives as long as a tensor over it does."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3,
                                         "strides": None, "stream": None}


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _pinned(n):
    return torch.zeros(n, dtype=F64).pin_memory().numpy()


def prepare(case, seed):
    s = State()
    s.case = case
    x, v, m, soft, g = _particles(case, seed)
    s.n = n = m.numel()
    kind = case["kind"]
    conf = dict(max_particles_per_leaf=case["bucket"], theta=case.get("theta", 0.7),
                precision=case.get("precision", "fp64"))
    if kind == "periodic":
        conf.update(periodic=True, n_replicas=1, period=1.0, ewald_hcut=math.sqrt(10.0))
    if kind == "gradient":
        conf["record_lists"] = True
    if "dt" in case:
        conf["max_timestep"] = case["dt"]
    s.sim = GravitySimulation(**conf)
    s.visitor = GravityVisitor(theta=conf["theta"])
    s.views = {}
    if kind == "trip":
        s.input = dict(zip(FIELDS, [_host(t) for t in (*x, *v, m, soft)]))
        s.acc = {k: np.zeros(n) for k in ("ax", "ay", "az", "pot", "pot_full")}
        return s
    s.particles = [t.contiguous() for t in (*x, *v, m, soft)]
    torch.cuda.synchronize()
    s.sim.set_particles_device(n, [t.data_ptr() for t in s.particles])
    torch.cuda.synchronize()
    if kind == "gradient":
        s.cot = [_host(t) for t in _cotangent(n, g)]
        s.grad = {k: _pinned(n) for k in ("gx", "gy", "gz", "gm")}
    elif kind == "chain":
        s.target = [_host(t) for t in _target(x, g)]
    elif kind == "pressure":
        s.u = _host(_energy(n, g))
    return s


def _cotangent(n, g):
    return torch.randn(3, n, generator=g, device=DEV, dtype=F64)


def _target(x, g):
    return x + 1e-3 * torch.randn(x.shape, generator=g, device=DEV, dtype=F64)


def _energy(n, g):
    return 0.5 + _uniform(n, g)


def _results(s):
    """The device arrays of the last force pass (key order) and the key order itself."""
    p = [ctypes.c_void_p() for _ in range(6)]
    s.sim._check(s.sim._lib.pt_device_accel(s.sim._h, *[ctypes.byref(q) for q in p]))
    out = {}
    for name, q in zip(("ax", "ay", "az", "pot", "pot_full", "order"), p):
        if q.value not in s.views:
            kind = "<i4" if name == "order" else "<f8"
            s.views[q.value] = torch.as_tensor(_Array(s.sim, q.value, s.n, kind), device=DEV)
        out[name] = s.views[q.value]
    return out


def run(s):
    kind = s.case["kind"]
    if kind in ("force", "periodic"):
        s.sim.start_down(s.visitor)
        return _results(s)
    if kind == "step":
        s.sim.run(1)
        return s.sim.state()
    if kind == "trip":
        s.sim.set_particles(s.input)
        s.sim.start_down(s.visitor)
        return s.sim.accelerations(s.acc)
    if kind == "gradient":
        s.sim.start_down(s.visitor)
        return dict(_results(s), **s.sim.adjoint(*s.cot, out=s.grad))
    if kind == "chain":
        loss, grads = s.sim.chain_grad(CHAIN_STEPS, s.case["dt"], s.target)
        return dict(grads, loss=loss)
    if kind == "density":
        return dict(zip(("density", "ball"), s.sim.sph_density()))
    return dict(zip(("density", "ax", "ay", "az", "pdv"), s.sim.sph_pressure(s.u)))


CHAIN_STEPS = 8


def work(case):
    """Bytes: each input field read and each result written once.  Flops: 20 per
    particle pair and 66 per node evaluation, with the interactions per particle
    of these distributions (measured at their sizes, as a law in log2 n)."""
    n = case["ngrid"] ** 3 if case["kind"] == "periodic" else case["n"]
    kind, bucket, theta = case["kind"], case["bucket"], case.get("theta", 0.7)
    if kind in ("density", "pressure"):
        return {"bytes": n * 8.0 * (5 if kind == "density" else 12), "flops": n * 32.0 * (20 if kind == "density" else 120)}
    pairs = min(n, (700.0 + 60.0 * bucket) * (0.7 / theta) ** 3)
    nodes = max(20.0, 85.0 * (math.log2(n) - 11.0)) * (0.7 / theta) ** 3
    flops = n * (20.0 * pairs + 66.0 * nodes)
    size = {"force": 84, "step": 136, "trip": 104, "periodic": 84, "gradient": 140, "chain": 144}[kind]
    passes = {"gradient": 3.0, "chain": 5.0 * CHAIN_STEPS, "periodic": 0.4}.get(kind, 1.0)
    return {"bytes": n * float(size), "flops": flops * passes}


# ---------------------------------------------------------------- the same in plain FP64 torch
class Tree:
    """Octree of key-sorted particles: nodes breadth first, children in groups of 8; moments per node."""

    def __init__(self, x, m, eps, bucket, theta):
        n = m.numel()
        d = x.detach()
        lo, hi = d.amin(1), d.amax(1)
        half = (1.0 + 1.91e-6) * 0.5 * (hi - lo).max()
        mid = (lo + hi) / 2.0
        ulo, uhi = mid - half, mid + half
        q = ((d - ulo[:, None]) / (uhi - ulo)[:, None] * 2097152.0).clamp(0, 2097151).to(torch.int64)
        key = torch.zeros_like(q[0])
        for b in range(21):
            for k in range(3):
                key |= ((q[k] >> b) & 1) << (3 * b + 2 - k)
        key, self.order = torch.sort(key, stable=True)
        self.x, self.m, self.eps = x[:, self.order], m[self.order], eps
        # topology, level by level
        start = [torch.zeros(1, dtype=torch.int64, device=DEV)]
        count = [torch.full((1,), n, dtype=torch.int64, device=DEV)]
        nkey = torch.zeros(1, dtype=torch.int64, device=DEV)
        inner, first, base = [], [], 0
        eight = torch.arange(8, device=DEV)
        for depth in range(22):
            idx = torch.nonzero((count[-1] > bucket) & (depth < 21))[:, 0]
            inner.append(idx)
            f = torch.full_like(count[-1], -1)
            base += count[-1].numel()
            f[idx] = base + 8 * torch.arange(idx.numel(), device=DEV)
            first.append(f)
            if idx.numel() == 0:
                break
            ck = nkey[idx][:, None] * 8 + eight
            s, c = start[-1][idx], count[-1][idx]
            ends = torch.searchsorted(key, ((ck[:, :7] + 1) << (60 - 3 * depth)).contiguous())
            ends = torch.cat([ends, (s + c)[:, None]], 1)
            begins = torch.cat([s[:, None], ends[:, :7]], 1)
            start.append(begins.reshape(-1))
            count.append((ends - begins).reshape(-1))
            nkey = ck.reshape(-1)
        self.start, self.count, self.first = torch.cat(start), torch.cat(count), torch.cat(first)
        self.leaf = (self.first < 0) & (self.count > 0)
        leaves = torch.nonzero(self.leaf)[:, 0]
        self.buckets = leaves[torch.argsort(self.start[leaves])]
        per = self.count[self.buckets]
        of = torch.repeat_interleave(torch.arange(per.numel(), device=DEV), per)  # each particle's bucket

        # moments bottom up: mass, mass * cm, then second moments about each cm, and particle boxes
        def upward(leafvals, combine, fill):
            node = torch.full((self.count.numel(),) + leafvals.shape[1:], fill, dtype=F64, device=DEV)
            node = node.index_put((self.buckets,), leafvals)
            sizes = [c.numel() for c in count]
            level = list(torch.split(node, sizes))
            for k in range(len(level) - 2, -1, -1):
                kids = level[k + 1].reshape(-1, 8, *leafvals.shape[1:])
                level[k] = level[k].index_put((inner[k],), combine(kids, k + 1, inner[k]))
            return torch.cat(level)

        offs = np.concatenate([[0], np.cumsum([c.numel() for c in count])])
        sums = torch.zeros(per.numel(), 4, dtype=F64, device=DEV).index_add(
            0, of, torch.cat([self.m[:, None], self.m[:, None] * self.x.t()], 1))
        sums = upward(sums, lambda kids, k, idx: kids.sum(1), 0.0)
        self.M = sums[:, 0]
        self.cm = sums[:, 1:] / self.M.clamp(min=1e-300)[:, None]

        def second(d):
            return torch.stack([d[..., i] * d[..., j] for i, j in ((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))], -1)

        quads = torch.zeros(per.numel(), 6, dtype=F64, device=DEV).index_add(
            0, of, self.m[:, None] * second(self.x.t() - self.cm[self.buckets][of]))

        def shift(kids, k, idx):
            parent = self.cm[offs[k - 1]:offs[k]][idx]
            d = self.cm[offs[k]:offs[k + 1]].reshape(-1, 8, 3) - parent[:, None]
            return (kids + self.M[offs[k]:offs[k + 1]].reshape(-1, 8)[..., None] * second(d)).sum(1)

        self.Q = upward(quads, shift, 0.0)
        d = self.x.detach().t()
        big = torch.full((per.numel(), 3), 1e300, dtype=F64, device=DEV)
        of3 = of[:, None].expand(-1, 3)
        self.lo = upward(big.scatter_reduce(0, of3, d, "amin"), lambda kids, k, idx: kids.amin(1), 1e300)
        self.hi = upward((-big).scatter_reduce(0, of3, d, "amax"), lambda kids, k, idx: kids.amax(1), -1e300)
        c = self.cm.detach()
        reach2 = torch.maximum(c - self.lo, self.hi - c).square().sum(1)
        self.open2 = torch.where(self.first >= 0, reach2 * (4.0 / 3.0 / (theta * theta)), torch.zeros_like(reach2))
        self.pad = self.count.numel()  # the index of a record that stands for no node

    def lists(self, b0, b1, off):
        """(bucket, leaf) and (bucket, node, monopole) of the buckets [b0, b1), sorted by bucket."""
        cm, eight = self.cm.detach(), torch.arange(8, device=DEV)
        tn = self.buckets[b0:b1]
        lo, hi, tc = self.lo[tn], self.hi[tn], cm[tn]
        fb = torch.arange(b1 - b0, device=DEV)
        fn = torch.zeros_like(fb)
        pp, pc = [], []
        while fb.numel():
            leaf = self.leaf[fn]
            pp.append(torch.stack([fb[leaf], fn[leaf]]))
            fb, fn = fb[~leaf], fn[~leaf]
            c = cm[fn] + off
            gap2 = torch.maximum(lo[fb] - c, c - hi[fb]).clamp(min=0).square().sum(1)
            opened = (gap2 <= self.open2[fn]) | (self.count[fn] <= 6)
            kept = ~opened
            r1 = 2.0 * self.eps
            mono = ((c - tc[fb]).square().sum(1) <= 4 * r1 * r1) | (gap2 <= r1 * r1)
            pc.append(torch.stack([fb[kept], fn[kept], mono[kept].to(torch.int64)]))
            kids = (self.first[fn[opened]][:, None] + eight).reshape(-1)
            fb = torch.repeat_interleave(fb[opened], 8)
            some = self.count[kids] > 0
            fb, fn = fb[some], kids[some]
        pp, pc = torch.cat(pp, 1), torch.cat(pc, 1)
        return pp[:, torch.argsort(pp[0], stable=True)], pc[:, torch.argsort(pc[0], stable=True)]


def _dense(row, value, rows, pad):
    """value of each (sorted) row side by side, padded: (rows, longest)."""
    per = torch.bincount(row, minlength=rows)
    first = torch.cumsum(per, 0) - per
    out = torch.full((rows, max(1, int(per.max()))), pad, dtype=value.dtype, device=DEV)
    out[row, torch.arange(row.numel(), device=DEV) - first[row]] = value
    return out


def _pairs(xt, xs, ms, reach):
    """Spline-softened sums over sources: accelerations (B, T, 3) and potentials (B, T)."""
    d = [xs[:, None, :, k] - xt[:, :, None, k] for k in range(3)]
    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    r2 = r2.masked_fill(r2 == 0, math.inf)
    a = torch.rsqrt(r2)
    b = a * a * a
    near = torch.nonzero(r2 < reach * reach, as_tuple=True)
    if near[0].numel():
        r = torch.sqrt(r2[near])
        h = 2.0 / reach
        u = r * h
        a_in = h * (7 / 5 - 2 / 3 * u ** 2 + 3 / 10 * u ** 4 - 1 / 10 * u ** 5)
        b_in = h ** 3 * (4 / 3 - 6 / 5 * u ** 2 + 1 / 2 * u ** 3)
        a_out = -1 / 15 / r + h * (8 / 5 - 4 / 3 * u ** 2 + u ** 3 - 3 / 10 * u ** 4 + 1 / 30 * u ** 5)
        b_out = -1 / 15 / r ** 3 + h ** 3 * (8 / 3 - 3 * u + 6 / 5 * u ** 2 - 1 / 6 * u ** 3)
        a = a.index_put(near, torch.where(u < 1, a_in, a_out))
        b = b.index_put(near, torch.where(u < 1, b_in, b_out))
    w = b * ms[:, None]
    return torch.stack([(w * dk).sum(2) for dk in d], 2), -(a * ms[:, None]).sum(2)


def _nodes(xt, cs, M, Q):
    """Monopole and quadrupole sums over nodes: accelerations and potentials (each node's)."""
    r = [xt[:, :, None, k] - cs[:, None, :, k] for k in range(3)]
    Q, M = Q[:, None], M[:, None]
    a = torch.rsqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2])
    a2 = a * a
    b = a * a2
    c = 3.0 * b * a2
    q = [Q[..., 0] * r[0] + Q[..., 1] * r[1] + Q[..., 2] * r[2],
         Q[..., 1] * r[0] + Q[..., 3] * r[1] + Q[..., 4] * r[2],
         Q[..., 2] * r[0] + Q[..., 4] * r[1] + Q[..., 5] * r[2]]
    qir = 0.5 * (q[0] * r[0] + q[1] * r[1] + q[2] * r[2])
    tr = 0.5 * (Q[..., 0] + Q[..., 3] + Q[..., 5])
    f = b * M + 5.0 * c * a2 * qir - c * tr
    return torch.stack([(c * qk - f * rk).sum(2) for qk, rk in zip(q, r)], 2), b * tr - M * a - c * qir


def _field(x, m, eps, bucket, theta, offsets=((0.0, 0.0, 0.0),), cot=None):
    """Accelerations (3, n) and potentials (quadrupole part, all) in key order with the key order; with a
    cotangent (3, n, caller order) also the gradients of sum(cot * acc) by x and m (caller order)."""
    x, m = x.detach(), m.detach()
    if cot is not None:
        x.requires_grad_(True)
        m.requires_grad_(True)
    T = Tree(x, m, eps, bucket, theta)
    n, nb = m.numel(), T.buckets.numel()
    # particle and node records with a padding entry at the end
    X = torch.cat([T.x.detach().t(), torch.full((1, 3), 1e10, dtype=F64, device=DEV)])
    W = torch.cat([T.m.detach(), torch.zeros(1, dtype=F64, device=DEV)])
    C = torch.cat([T.cm.detach(), torch.full((1, 3), 1e10, dtype=F64, device=DEV)])
    M = torch.cat([T.M.detach(), torch.zeros(1, dtype=F64, device=DEV)])
    Q = torch.cat([T.Q.detach(), torch.zeros(1, 6, dtype=F64, device=DEV)])
    out = torch.zeros(n + 1, 5, dtype=F64, device=DEV)
    if cot is not None:
        ct = torch.cat([cot[:, T.order].t(), torch.zeros(1, 3, dtype=F64, device=DEV)])
        g = [torch.zeros_like(t) for t in (X, W, C, M, Q)]
    width = max(1, int(T.count[T.buckets].max()))
    for b0 in range(0, nb, 8192):
        b1 = min(nb, b0 + 8192)
        for off in offsets:
            off = torch.tensor(off, dtype=F64, device=DEV)
            pp, pc = T.lists(b0, b1, off)
            longest = 1 + sum(int(torch.bincount(p[0], w, minlength=1).max()) if p.shape[1] else 0
                              for p, w in ((pp, T.count[pp[1]].double()), (pc, torch.ones_like(pc[0]).double())))
            size = max(1, (1 << 24 if cot is None else 1 << 22) // (width * longest))
            edges = torch.arange(0, b1 - b0 + size, size, device=DEV)
            cut_pp = torch.searchsorted(pp[0].contiguous(), edges).tolist()
            cut_pc = torch.searchsorted(pc[0].contiguous(), edges).tolist()
            for k in range(len(cut_pp) - 1):
                lo, hi = k * size, min(b1 - b0, (k + 1) * size)
                if lo >= hi:
                    break
                tn = T.buckets[b0 + lo:b0 + hi]
                tgt = T.start[tn][:, None] + torch.arange(width, device=DEV)
                tgt = torch.where(torch.arange(width, device=DEV) < T.count[tn][:, None], tgt, n)
                centre = C[tn][:, None]
                xt = X[tgt] - centre
                xt = torch.where((tgt == n)[..., None], 0.0, xt)
                p, c = pp[:, cut_pp[k]:cut_pp[k + 1]], pc[:, cut_pc[k]:cut_pc[k + 1]]
                if p.shape[1]:
                    per = T.count[p[1]]
                    row = torch.repeat_interleave(p[0] - lo, per)
                    at = torch.arange(row.numel(), device=DEV) - torch.repeat_interleave(torch.cumsum(per, 0) - per, per)
                    src = _dense(row, torch.repeat_interleave(T.start[p[1]], per) + at, hi - lo, n)
                    xs, ms = X[src] + off - centre, W[src]
                    if cot is None:
                        acc, pot = _pairs(xt, xs, ms, 2.0 * eps)
                        out.index_add_(0, tgt.reshape(-1), torch.cat([acc, 0 * pot[..., None], pot[..., None]], 2).view(-1, 5))
                    else:
                        v = [t.requires_grad_(True) for t in (xt.clone(), xs, ms)]
                        acc, _ = _pairs(*v, 2.0 * eps)
                        d = torch.autograd.grad((acc * ct[tgt]).sum(), v)
                        g[0].index_add_(0, tgt.reshape(-1), d[0].reshape(-1, 3))
                        g[0].index_add_(0, src.reshape(-1), d[1].reshape(-1, 3))
                        g[1].index_add_(0, src.reshape(-1), d[2].reshape(-1))
                        out[:, :3].index_add_(0, tgt.reshape(-1), acc.detach().reshape(-1, 3))
                if c.shape[1]:
                    node = _dense(c[0] - lo, c[1], hi - lo, T.pad)
                    mono = _dense(c[0] - lo, c[2], hi - lo, 0)
                    cs, Ms, Qs = C[node] + off - centre, M[node], Q[node] * (mono == 0)[..., None]
                    if cot is None:
                        acc, pot = _nodes(xt, cs, Ms, Qs)
                        quad = (pot * (mono == 0)[:, None]).sum(2)
                        out.index_add_(0, tgt.reshape(-1), torch.cat([acc, quad[..., None], pot.sum(2)[..., None]], 2).view(-1, 5))
                    else:
                        v = [t.requires_grad_(True) for t in (xt.clone(), cs, Ms, Qs)]
                        acc, _ = _nodes(*v)
                        d = torch.autograd.grad((acc * ct[tgt]).sum(), v)
                        g[0].index_add_(0, tgt.reshape(-1), d[0].reshape(-1, 3))
                        g[2].index_add_(0, node.reshape(-1), d[1].reshape(-1, 3))
                        g[3].index_add_(0, node.reshape(-1), d[2].reshape(-1))
                        g[4].index_add_(0, node.reshape(-1), (d[3] * (mono == 0)[..., None]).reshape(-1, 6))
                        out[:, :3].index_add_(0, tgt.reshape(-1), acc.detach().reshape(-1, 3))
    if cot is None:
        return out[:n].t(), T
    through = torch.autograd.grad([T.cm, T.M, T.Q, T.x, T.m], [x, m],
                                  [g[2][:-1], g[3][:-1], g[4][:-1], g[0][:-1].t(), g[1][:-1]])
    return out[:n].t(), T, through[0].detach(), through[1].detach()


def _ewald(x, T, out, n_replicas, rcut, hcut):
    """Adds the Ewald correction of the root's monopole and quadrupole in the unit cube."""
    M, Q, d0 = T.M[0], T.Q[0], x - T.cm[0][:, None]
    alpha = 2.0
    tr = 0.5 * (Q[0] + Q[3] + Q[5])
    ka = 2.0 * alpha / math.sqrt(math.pi)
    pot = torch.full_like(x[0], 0.0) + M * math.pi / alpha ** 2
    acc = torch.zeros_like(x)
    reps = max(math.ceil(rcut), n_replicas)
    span = range(-reps, reps + 1)
    for i, j, k in ((i, j, k) for i in span for j in span for k in span):
        d = d0 + torch.tensor([[i], [j], [k]], dtype=F64, device=DEV)
        hole = max(abs(i), abs(j), abs(k)) <= n_replicas
        r2 = (d * d).sum(0)
        inv = torch.rsqrt(r2)
        inv2 = inv * inv
        e = torch.exp(-r2 * alpha ** 2) * ka * inv2
        g = [(-torch.erf(alpha / inv) if hole else torch.erfc(alpha / inv)) * inv]
        g.append(g[0] * inv2 + e)
        g.append(3 * g[1] * inv2 + 2 * alpha ** 2 * e)
        g.append(5 * g[2] * inv2 + 4 * alpha ** 4 * e)
        s = r2 * alpha ** 2
        small = r2 < 1.2e-3
        for o, (p, q) in enumerate(((1 / 3, 1.0), (1 / 5, 1 / 3), (1 / 7, 1 / 5), (1 / 9, 1 / 7))):
            g[o] = torch.where(small, ka * (2 * alpha ** 2) ** o * (p * s - q), g[o])
        if not hole:
            g = [torch.where(r2 > rcut * rcut, 0.0, gk) for gk in g]
        q = torch.stack([Q[0] * d[0] + Q[1] * d[1] + Q[2] * d[2], Q[1] * d[0] + Q[3] * d[1] + Q[4] * d[2],
                         Q[2] * d[0] + Q[4] * d[1] + Q[5] * d[2]])
        qir = 0.5 * (q * d).sum(0)
        pot -= g[0] * M - g[1] * tr + g[2] * qir
        acc += g[2] * q - d * (g[1] * M - g[2] * tr + g[3] * qir)
    top = math.ceil(hcut)
    span = range(-top, top + 1)
    for h in ((i, j, k) for i in span for j in span for k in span):
        h2 = h[0] ** 2 + h[1] ** 2 + h[2] ** 2
        if h2 == 0 or h2 > hcut * hcut:
            continue
        g0 = math.exp(-math.pi ** 2 / alpha ** 2 * h2) / (math.pi * h2)
        g2 = -4 * math.pi ** 2 * g0
        qir = 0.5 * (Q[0] * h[0] ** 2 + Q[3] * h[1] ** 2 + Q[5] * h[2] ** 2) + Q[1] * h[0] * h[1] + \
            Q[2] * h[0] * h[2] + Q[4] * h[1] * h[2]
        w = -g2 * qir - g0 * M
        hv = 2 * math.pi * torch.tensor(h, dtype=F64, device=DEV)
        phase = hv @ d0
        pot += w * torch.cos(phase)
        acc += hv[:, None] * (w * torch.sin(phase))
    return torch.cat([out[:3] + acc, out[3:] + pot])


def _neighbours(x, k=32):
    """d2 and indices of the k nearest particles of each (itself included)."""
    n = x.shape[1]
    rows = max(1, (1 << 27) // n)
    d2, idx = [], []
    for i in range(0, n, rows):
        d = [x[a, i:i + rows, None] - x[a] for a in range(3)]
        v, j = torch.topk(d[0] * d[0] + d[1] * d[1] + d[2] * d[2], k, dim=1, largest=False)
        d2.append(v)
        idx.append(j)
    return torch.cat(d2), torch.cat(idx)


def _sph_exact(x, v, m, u):
    d2, idx = _neighbours(x)
    ball = d2.amax(1)
    ar2 = d2 * (4.0 / ball)[:, None]
    ak = 2.0 - torch.sqrt(ar2)
    kern = torch.where(ar2 < 1.0, 1.0 - 0.75 * ak * ar2, 0.25 * ak ** 3)
    rho = (kern * m[idx]).sum(1) / (math.pi / 8 * ball ** 1.5)
    if u is None:
        return {"density": rho.cpu(), "ball": ball.cpu()}
    adk = torch.sqrt(ar2)
    dk = torch.where(ar2 < 1.0, -3 + 2.25 * adk, -0.75 * (2.0 - adk) ** 2 / adk.clamp(min=1e-300))
    t = dk * d2 * m[idx]
    corr = t.sum(1) / rho / (t / rho[idx]).sum(1)
    ih2 = 4.0 / ball
    rs = dk * (0.5 / math.pi * ih2 * ih2 / (0.5 * torch.sqrt(ball)) * corr)[:, None]
    dx = x[:, idx] - x[:, :, None]
    dv = (v[:, idx] - v[:, :, None]).mul(dx).sum(0)
    aP = u[:, None] * (2.0 / 3.0) / rho[idx]
    bP = u[idx] * (2.0 / 3.0) / rho[:, None]
    acc = (aP + bP) * rs
    own = (acc * m[idx] * dx).sum(2)
    pdv = (rs * m[idx] * aP * dv).sum(1)
    flat = idx.reshape(-1)
    for k in range(3):
        own[k].index_add_(0, flat, -(acc * m[:, None] * dx[k]).reshape(-1))
    other = idx != torch.arange(m.numel(), device=DEV)[:, None]
    pdv.index_add_(0, flat, (rs * m[:, None] * aP * dv * other).reshape(-1))
    return {"density": rho.cpu(), "ax": own[0].cpu(), "ay": own[1].cpu(), "az": own[2].cpu(), "pdv": pdv.cpu()}


def _caller(T, out):
    r = torch.empty_like(out)
    r[:, T.order] = out
    return r


def exact(case, seed):
    x, v, m, soft, g = _particles(case, seed)
    kind, n, bucket, theta = case["kind"], m.numel(), case["bucket"], case.get("theta", 0.7)
    if kind in ("density", "pressure"):
        if n > 300000:  # every particle against every other: over 20 seconds
            return None
        return _sph_exact(x, v, m, _energy(n, g) if kind == "pressure" else None)
    eps = float(soft[0])
    names = ("ax", "ay", "az", "pot", "pot_full")
    if kind == "periodic":
        offs = [(i, j, k) for i in (-1.0, 0.0, 1.0) for j in (-1.0, 0.0, 1.0) for k in (-1.0, 0.0, 1.0)]
        out, T = _field(x, m, eps, bucket, theta, offs)
        return dict(zip(names, _ewald(T.x, T, out, 1, 2.6, math.sqrt(10.0))), order=None)
    if kind == "force":
        out, T = _field(x, m, eps, bucket, theta)
        return dict(zip(names, out), order=None)
    if kind == "trip":
        out, T = _field(x, m, eps, bucket, theta)
        return dict(zip(names, _caller(T, out).cpu()))
    if kind == "step":
        out, T = _field(x, m, eps, bucket, theta)
        dt = case["dt"]
        size = (1.0 + 1.91e-6) * (x.amax(1) - x.amin(1)).max()
        dt = min(float(size / v.square().sum(0).max().sqrt() / n ** (1 / 3)) if bool((v != 0).any()) else dt, dt)
        v = v + _caller(T, out[:3]) * dt
        return dict(zip(("x", "y", "z", "vx", "vy", "vz"), torch.cat([x + v * dt, v]).cpu()))
    if kind == "gradient":
        cot = _cotangent(n, g)
        out, T = _field(x, m, eps, bucket, theta)
        _, _, gx, gm = _field(x, m, eps, bucket, theta, cot=cot)
        return dict(zip(names, out), order=None, gx=gx[0].cpu(), gy=gx[1].cpu(), gz=gx[2].cpu(), gm=gm.cpu())
    # chain: leapfrog steps forward, then their adjoints from the last to the first
    y, dt = _target(x, g), case["dt"]

    def acc(x):
        out, T = _field(x, m, eps, bucket, theta)
        return _caller(T, out[:3])

    xs, a = [x], acc(x)
    for _ in range(CHAIN_STEPS):
        v = v + 0.5 * dt * a
        xs.append(xs[-1] + dt * v)
        a = acc(xs[-1])
        v = v + 0.5 * dt * a
    loss = 0.5 * (xs[-1] - y).square().sum()
    xb, vb, mb, pend = xs[-1] - y, torch.zeros_like(x), torch.zeros_like(m), torch.zeros_like(x)
    for s in range(CHAIN_STEPS, -1, -1):
        pend = pend + 0.5 * dt * vb if s else pend
        if s < CHAIN_STEPS:
            _, _, gx, gm = _field(xs[s], m, eps, bucket, theta, cot=pend)
            xb, mb = xb + gx, mb + gm
        if s:
            vb = vb + dt * xb
            pend = 0.5 * dt * vb
    return dict(zip(("gx", "gy", "gz", "gvx", "gvy", "gvz"), torch.cat([xb, vb]).cpu()), gm=mb.cpu(), loss=float(loss))
