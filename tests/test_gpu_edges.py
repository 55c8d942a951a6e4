"""Sizes at which a pass changes its kernels or tiles, against the CPU oracle
(FP64: bit for bit) or the FP64 form (mixed).

* keys and tree: the rank sort's largest size and the first radix-sorted one,
  the tree build's tile of 1024 particles, the radix sort's change of tile at
  2^19 keys, runs of equal keys longer than a tile;
* FP64 walk: a CTA or a warp per bucket (24 buckets per SM), one to 32 targets
  per bucket, both visit orders;
* mixed evaluation: a CTA or a warp per bucket (96 buckets per SM);
* periodic mixed pass: batches of 32 replicas."""
import numpy as np
import pytest

from oracle import oracle as O
from paratreet_b200 import ics

pytestmark = pytest.mark.gpu

OUT = ("ax", "ay", "az", "pot", "pot_full")


def sim(**kw):
    from paratreet_b200.gravity import GravitySimulation
    return GravitySimulation(**kw)


def assert_tree_and_forces(p, bucket, theta, traversal="transposed"):
    ref = O.PortSim(p, bucket=bucket, theta=theta, threads=8)
    if traversal == "basic":
        ref.set_basic_down()
    ref.forces()
    with sim(max_particles_per_leaf=bucket, theta=theta, traversal=traversal) as s:
        s.set_particles(p)
        s.start_down()
        assert np.array_equal(s.keys(), ref.keys())
        tg, tr = O.sort_tree(s.tree()), O.sort_tree(ref.tree())
        assert np.array_equal(tg.keys, tr.keys)
        assert np.array_equal(tg.types, tr.types)
        assert np.array_equal(tg.count, tr.count)
        assert np.array_equal(tg.moments, tr.moments)
        a = s.accelerations()
        for k, w in zip(OUT, ref.acc()):
            assert np.array_equal(a[k], w), k
        return s.counters()["n_buckets"]


@pytest.mark.parametrize("n", [1023, 1024, 1025, 2049, 16383, 16384, 16385])
def test_tiles_and_sorts_bit_exact(n):
    assert_tree_and_forces(ics.mixture(n, seed=n, clump_a=0.02), 8, 0.9)


@pytest.mark.parametrize("n", [(1 << 19) - 1, (1 << 19) + 1])
def test_radix_tile_change_bit_exact(n):
    assert_tree_and_forces(ics.mixture(n, seed=5), 32, 1.2)


@pytest.mark.parametrize("bucket", [1, 8, 32])
def test_equal_keys_across_tiles(bucket):
    """1100 particles at one point (a depth-21 leaf longer than a tile of the
    build) among 1500 others, and 33 at another."""
    p = ics.plummer(2633, seed=9)
    for k in ("x", "y", "z"):
        p[k][500:1600] = p[k][0]
        p[k][1700:1733] = p[k][1]
    assert_tree_and_forces(p, bucket, 0.7)


# 24 buckets per SM are 3552 on 148 SMs: both sides of the line, and every
# number of targets a bucket can have
@pytest.mark.parametrize("gen,n,bucket,traversal", [
    ("plummer", 700, 1, "transposed"), ("plummer", 40, 32, "transposed"), ("hernquist", 3000, 17, "transposed"),
    ("mixture", 9000, 32, "basic"), ("plummer", 3000, 2, "basic"), ("mixture", 12000, 11, "transposed"),
    ("mixture", 24000, 13, "transposed"),
])
def test_fp64_walk_team_and_warp_bit_exact(gen, n, bucket, traversal):
    nb = assert_tree_and_forces(getattr(ics, gen)(n, seed=31), bucket, 0.8, traversal)
    print(gen, n, bucket, "buckets", nb)


# 96 buckets per SM are 14208; the tolerance is the mixed form's everywhere
@pytest.mark.parametrize("n,bucket", [(900, 1), (3001, 32), (50000, 16), (90001, 16), (20000, 1)])
def test_mixed_team_and_warp_match_fp64(n, bucket):
    p = ics.plummer(n, seed=17)
    out = {}
    for prec in ("fp64", "mixed"):
        with sim(max_particles_per_leaf=bucket, precision=prec) as s:
            s.set_particles(p)
            s.start_down()
            out[prec] = s.accelerations()
            c = s.counters()
            out[prec + "n"] = (c["n_pp"], c["n_pc"], c["n_open"], int(s.bucket_work().sum()))
    assert out["fp64n"] == out["mixedn"]
    a, m = out["fp64"], out["mixed"]
    num = sum((a[k] - m[k]) ** 2 for k in ("ax", "ay", "az"))
    den = sum(a[k] ** 2 for k in ("ax", "ay", "az"))
    assert np.sqrt(np.mean(num / den)) < 1e-5


# one batch that is not full (27), and four, the last of 29 (125 replicas).  The
# residual accelerations of a 12^3 lattice are about 0.2; every replica adds
# terms of size 1 with FP32 rounding 6e-8, so 125 of them leave less than 1e-5
@pytest.mark.parametrize("nrep,bucket", [(1, 8), (2, 16), (2, 32)])
def test_mixed_replica_batches_match_fp64(nrep, bucket):
    p = ics.lattice(12, seed=3, rms_cells=0.3, soft_cells=0.5)
    out = {}
    for prec in ("fp64", "mixed"):
        with sim(max_particles_per_leaf=bucket, theta=0.7, periodic=True, n_replicas=nrep, precision=prec) as s:
            s.set_particles(p)
            s.start_down()
            out[prec] = s.accelerations()
            c = s.counters()
            out[prec + "n"] = (c["n_pp"], c["n_pc"], c["n_open"], int(s.bucket_work().sum()))
    assert out["fp64n"] == out["mixedn"]
    for k in ("ax", "ay", "az"):
        assert np.abs(out["mixed"][k] - out["fp64"][k]).max() < 1e-5
    for k in ("pot", "pot_full"):
        assert np.abs(out["mixed"][k] - out["fp64"][k]).max() < 1e-5 * (2 * nrep + 1) ** 2


def test_mixed_replica_batches_over_bucket_ranges():
    p = ics.lattice(10, seed=4, rms_cells=0.3, soft_cells=0.5)
    with sim(max_particles_per_leaf=16, periodic=True, n_replicas=1, precision="mixed") as s:
        s.set_particles(p)
        s.start_down()
        full = s.accelerations()
        nb = s.bucket_keys().size
        parts = []
        for rng in ((0, nb // 3), (nb // 3, nb)):
            s.start_down(buckets=rng)
            parts.append(s.accelerations())
    for k in OUT:
        assert np.allclose(parts[0][k] + parts[1][k], full[k], rtol=0, atol=1e-6), k


# a later replica's (batch's) lists outgrow the pools: the walk of that batch is
# repeated, which costs a launch in the first pass and none in the second
@pytest.mark.parametrize("prec,nrep,theta", [("fp64_lists", 1, 0.25), ("mixed", 2, 0.35)])
def test_repeated_walk_counts_its_work_once(prec, nrep, theta):
    p = ics.lattice(12, seed=3, rms_cells=0.3, soft_cells=0.2)
    kw = dict(max_particles_per_leaf=1, theta=theta, periodic=True, n_replicas=nrep)
    with sim(precision="fp64", **kw) as s:
        s.set_particles(p)
        s.start_down()
        want, c0 = s.bucket_work(), s.counters()
    with sim(precision=prec, **kw) as s:
        s.set_list_region(64)
        s.set_particles(p)
        s.start_down()
        first, c1 = s.bucket_work(), s.counters()
        s.start_down()
        second, c2 = s.bucket_work(), s.counters()
    print(prec, "launches", c1["launches"], c2["launches"], "entries per bucket", c0["n_pc"] / c0["n_buckets"], c0["n_pp"] / c0["n_buckets"])
    assert c1["launches"] > c2["launches"]
    for c in (c1, c2):
        assert [c[k] for k in ("n_pp", "n_pc", "n_open")] == [c0[k] for k in ("n_pp", "n_pc", "n_open")]
    assert np.array_equal(second, want)
    assert np.array_equal(first, want)


def test_one_handle_across_sizes():
    """One handle keeps its sort scratch (look-back words of both tile sizes,
    told apart by their tags), node arrays and list descriptors from size to size:
    every pass is a fresh handle's bit for bit."""
    sizes = [(1 << 19) + 1, 20000, 5000, (1 << 19) - 1, 300, 1 << 20, 16384, 16385, (1 << 19) + 1]
    kw = dict(max_particles_per_leaf=32, theta=1.2)
    for prec in ("fp64", "mixed"):
        with sim(precision=prec, **kw) as s:
            for n in sizes:
                p = ics.mixture(n, seed=n)
                s.set_particles(p)
                s.start_down()
                got, keys = s.accelerations(), s.keys()
                with sim(precision=prec, **kw) as f:
                    f.set_particles(p)
                    f.start_down()
                    want = f.accelerations()
                    assert np.array_equal(keys, f.keys()), (prec, n)
                for k in OUT:
                    assert np.array_equal(got[k], want[k]), (prec, n, k)


@pytest.mark.parametrize("n", [20000, (1 << 19) + 1])
def test_sort_tags_start_over(n):
    """The look-back words are cleared after 127 sorts, and the tags begin again."""
    p, q = ics.plummer(n, seed=21), ics.mixture(n, seed=22)
    with sim(max_particles_per_leaf=32, theta=1.5, precision="mixed") as s:
        want = []
        for r in (p, q):
            s.set_particles(r)
            s.start_down()
            want.append((s.keys(), s.accelerations()))
        for k in range(270):
            i = k % 2
            s.set_particles((p, q)[i])
            s.start_down()
            if 120 <= k < 132 or 246 <= k < 260 or k > 266:
                assert np.array_equal(s.keys(), want[i][0]), k
                a = s.accelerations()
                for c in OUT:
                    assert np.array_equal(a[c], want[i][1][c]), (k, c)


# a bucket's list is cut into min(8, 75,776 / buckets) slices on 148 SMs: eight, a
# few, two, and one
@pytest.mark.parametrize("n", [9000, 40000, 55000, 120000])
def test_adjoint_slices_match_finite_differences(n):
    """The derivative along one direction of all positions and masses, against
    central differences of the frozen lists.  h = 1e-6 of the positions' scale:
    truncation (h / softening)^2 = 2.5e-9, rounding below 1e-16 sqrt(n) / h = 4e-8
    of the objective."""
    p = ics.plummer(n, seed=12, soft=0.02)
    rng = np.random.default_rng(3)
    cot, d = rng.normal(size=(3, n)), rng.normal(size=(4, n))
    h = 1e-6
    with sim(max_particles_per_leaf=4, record_lists=True) as s:
        s.set_particles(p)
        s.start_down()
        nb = s.counters()["n_buckets"]
        g = s.adjoint(*cot)

        def objective(sign):
            a = s.forces_frozen(*[p[k] + sign * h * d[i] for i, k in enumerate("xyz")], p["m"] * (1 + sign * h * d[3]))
            return sum(float(np.dot(cot[i], a[k])) for i, k in enumerate(("ax", "ay", "az")))

        fd = (objective(1) - objective(-1)) / (2 * h)
    parts = [float(np.dot(g["g" + k], d[i])) for i, k in enumerate("xyz")] + [float(np.dot(g["gm"], p["m"] * d[3]))]
    scale = max(abs(v) for v in parts)
    print(n, "buckets", nb, "slices", max(1, min(8, 75776 // nb)), "fd", fd, "adjoint", sum(parts))
    assert abs(fd - sum(parts)) < 1e-5 * scale
