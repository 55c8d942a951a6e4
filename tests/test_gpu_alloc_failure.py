"""Refused device allocations (pt_set_alloc_limit, a host-side limit: nothing is
allocated to make room scarce).  A pass that fails behind the sort has moved the
particles, so the results of the pass before it are refused until a pass
succeeds; the handle stays usable, and its next pass equals a fresh handle's."""
import numpy as np
import pytest

from paratreet_b200 import ics
from paratreet_b200._lib import PtError

pytestmark = pytest.mark.gpu

OUT = ("ax", "ay", "az", "pot", "pot_full")


def sim(**kw):
    from paratreet_b200.gravity import GravitySimulation
    return GravitySimulation(**kw)


def refused(call, code):
    with pytest.raises(PtError) as e:
        call()
    assert e.value.code == code, e.value
    return str(e.value)


NOMEM, STATE = -3, -4


def test_failed_pass_drops_earlier_results():
    """The FP64 form's source records do not fit: the tree is rebuilt and the
    particles are in a new order when the pass stops."""
    p = ics.plummer(5000, seed=8, soft=1e-2)
    with sim(precision="mixed", max_timestep=0.5) as s:
        s.set_particles(p)
        s.start_down()
        s.advance()  # the next sort gives another order
        moved = s.state()
        s.accelerations()  # the last pass's, still the positions' old order
        s.set_precision("fp64")
        s.set_alloc_limit(1)
        refused(s.start_down, NOMEM)
        refused(s.accelerations, STATE)
        refused(s.keys, STATE)
        refused(s.advance, STATE)
        refused(s.lists, STATE)
        refused(lambda: s.list_digests("two_phase"), STATE)
        got = s.state()
        for k in moved:
            assert np.array_equal(got[k], moved[k]), k
        s.set_alloc_limit(0)
        s.start_down()
        a = s.accelerations()
    q = dict(p, **moved)
    with sim(precision="fp64") as f:
        f.set_particles(q)
        f.start_down()
        want = f.accelerations()
    for k in OUT:
        assert np.array_equal(a[k], want[k]), k


def test_failed_pass_drops_earlier_lists():
    """The mixed form's FP32 source records do not fit: the recorded lists are of
    the tree before."""
    p = ics.plummer(5000, seed=8, soft=1e-2)
    with sim(precision="fp64", max_timestep=0.5, record_lists=True) as s:
        s.set_particles(p)
        s.start_down()
        s.lists()
        s.advance()
        s.set_precision("mixed")
        s.set_alloc_limit(1)
        refused(s.start_down, NOMEM)
        refused(s.lists, STATE)
        refused(lambda: s.list_digests("recorded"), STATE)
        refused(lambda: s.adjoint(p["x"], p["y"], p["z"]), STATE)
        refused(lambda: s.forces_frozen(x=p["x"]), STATE)
        s.set_alloc_limit(0)
        s.start_down()
        assert s.lists().offsets[-1] > 0


def test_sph_pass_drops_earlier_lists():
    """The density pass rebuilds the tree; the two-phase lists are of the one before."""
    p = ics.plummer(3000, seed=4, soft=1e-2)
    with sim(precision="mixed", max_particles_per_leaf=8) as s:
        s.set_particles(p)
        s.start_down()
        s.list_digests("two_phase")
        s.sph_density()
        refused(lambda: s.list_digests("two_phase"), STATE)
        refused(s.accelerations, STATE)
        s.start_down()
        s.list_digests("two_phase")


# limits between the sizes of a pass's arrays: the refused one is another each
# time (n = 20,000: 0.5 MB of bucket counters at most, 2 MB of node arrays, 4 MB
# of particles, the list pools far larger)
@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp64_lists"])
@pytest.mark.parametrize("record", [False, True])
def test_refused_growth_is_tried_again(precision, record):
    """A handle that served a small system meets a larger one under a limit, then
    the larger one without it, and the small one again."""
    small, large = ics.plummer(600, seed=2, soft=1e-2), ics.plummer(20000, seed=3, soft=1e-2)
    kw = dict(precision=precision, record_lists=record, max_particles_per_leaf=4, theta=0.9)
    want = {}
    for name, p in (("small", small), ("large", large)):
        with sim(**kw) as f:
            f.set_particles(p)
            f.start_down()
            want[name] = f.accelerations()
    failed = set()
    tol = 1e-4 if precision == "mixed" else 1e-12
    for limit in [1 << k for k in range(8, 24)]:
        with sim(**kw) as s:
            s.set_particles(small)
            s.start_down()
            s.set_particles(large)
            s.set_alloc_limit(limit)
            for _ in range(2):
                try:
                    s.start_down()
                except PtError as e:
                    assert e.code == NOMEM
                    failed.add(limit)
                    refused(s.accelerations, STATE)
            s.set_alloc_limit(0)
            for name, p in (("small", small), ("large", large)):
                s.set_particles(p)
                s.start_down()
                a = s.accelerations()
                for k in OUT[:3]:  # the forms that replace refused list pools sum in another order
                    assert np.abs(a[k] - want[name][k]).max() <= tol * np.abs(want[name][k]).max(), (limit, k)
    assert len(failed) >= 4


def test_refused_sph_and_adjoint_arrays_are_tried_again():
    small, large = ics.plummer(600, seed=2, soft=1e-2), ics.plummer(6000, seed=3, soft=1e-2)
    for limit in [1 << k for k in range(12, 22)]:
        with sim(precision="fp64", record_lists=True) as s, sim(precision="fp64", record_lists=True) as f:
            for h in (s, f):
                h.set_particles(small)
                h.sph_density(neighbors=True)
                h.start_down()
                h.adjoint(small["x"], small["y"], small["z"])
                h.set_particles(large)
            s.set_alloc_limit(limit)
            for call in (s.sph_density, lambda: s.sph_density(neighbors=True), s.start_down,
                         lambda: s.adjoint(large["x"], large["y"], large["z"])):
                try:
                    call()
                except PtError as e:
                    assert e.code in (NOMEM, STATE)
            s.set_alloc_limit(0)
            out = []
            for h in (s, f):
                d = h.sph_density(neighbors=True)
                h.start_down()
                out.append((d, h.accelerations(), h.adjoint(large["x"], large["y"], large["z"])))
            for a, b in zip(out[0][0], out[1][0]):
                assert np.array_equal(a, b)
            for k in OUT:
                assert np.array_equal(out[0][1][k], out[1][1][k])
            for k in ("gx", "gy", "gz", "gm"):  # atomic adds: the last bits vary
                b = out[1][2][k]
                assert np.abs(out[0][2][k] - b).max() <= 1e-9 * np.abs(b).max()


def test_headroom_gives_way():
    """Recorded lists that fit without the eighth of headroom: n entries of four
    bytes are the largest allocation of this pass behind the first handle's."""
    p = ics.plummer(30000, seed=5, soft=1e-2)
    kw = dict(precision="fp64_lists", record_lists=True, max_particles_per_leaf=4, theta=0.5)
    with sim(**kw) as f:
        f.set_particles(p)
        f.start_down()
        total = int(f.lists().offsets[-1])
        want = f.accelerations()
    q = ics.plummer(30000, seed=5, soft=1e-2)
    with sim(**dict(kw, theta=0.9)) as s:  # shorter lists: every other array has its size
        s.set_particles(q)
        s.start_down()
        assert s.lists().offsets[-1] * 9 // 8 < total
        s.set_theta(0.5)
        s.set_alloc_limit(4 * total + 256)
        s.start_down()
        assert int(s.lists().offsets[-1]) == total
        a = s.accelerations()
    for k in OUT:
        assert np.array_equal(a[k], want[k]), k


# bytes per entry of the first pools: 13 leaves batches of one replica (no replica
# bytes), 20 of half the 27
@pytest.mark.parametrize("nrep,room", [(1, 13), (1, 20), (2, 13)])
def test_replica_lists_that_do_not_fit_take_smaller_batches(nrep, room):
    """The lists of a full batch of replicas outgrow the limit, those of a few fit:
    the pass takes fewer replicas at a time instead of the fused form, which
    leaves no potential (pot) of the quadrupole terms."""
    p = ics.lattice(24, seed=6, rms_cells=0.3, soft_cells=0.3)
    kw = dict(precision="mixed", max_particles_per_leaf=4, theta=0.4, periodic=True, n_replicas=nrep)
    out, counts, launches = [], [], []
    # as test_mixed_replica_batches_match_fp64 (tests/test_gpu_edges.py)
    scale = {"a": 1, "p": (2 * nrep + 1) ** 2}
    for limit in (0, 1):
        with sim(**kw) as s:
            s.set_list_region(64)
            s.set_particles(p)
            if limit:
                s.set_alloc_limit(room * (1024 * nb + 148 * 7 * 4 * 64))
            s.start_down()
            nb = s.counters()["n_buckets"]
            out.append(s.accelerations())
            c = s.counters()
            counts.append((c["n_pp"], c["n_pc"], c["n_open"], int(s.bucket_work().sum())))
            s.start_down()
            again = s.accelerations()
            launches.append((c["launches"], s.counters()["launches"]))
            for k in OUT:
                assert np.abs(again[k] - out[-1][k]).max() < 1e-5 * scale[k[0]], k
    print("launches", launches)
    assert counts[0] == counts[1]
    assert launches[1][1] > launches[0][1]
    for k in OUT:
        assert np.abs(out[0][k] - out[1][k]).max() < 1e-5 * scale[k[0]], k


def test_ordered_walk_in_the_middle_of_a_pass():
    """PT_FP64_LISTS under the same limit: the replicas whose lists do not fit are
    walked in order, the sums before them stay, and no work is counted twice."""
    p = ics.lattice(24, seed=6, rms_cells=0.3, soft_cells=0.3)
    kw = dict(max_particles_per_leaf=4, theta=0.4, periodic=True, n_replicas=1)
    out = []
    for prec in ("fp64", "fp64_lists"):
        with sim(precision=prec, **kw) as s:
            s.set_list_region(64)
            s.set_particles(p)
            s.set_alloc_limit(8 * (1024 * 8583 + 148 * 7 * 4 * 64))  # 8583 buckets
            s.start_down()
            out.append((s.accelerations(), s.bucket_work(), s.counters()))
    (a, wa, ca), (b, wb, cb) = out
    assert ca["n_buckets"] == 8583 and cb["launches"] != ca["launches"]
    assert np.array_equal(wa, wb)
    assert all(ca[k] == cb[k] for k in ("n_pp", "n_pc", "n_open"))
    for k in OUT:  # sums of 27 replicas of size 1 each in another order
        assert np.abs(a[k] - b[k]).max() <= 1e-11 * (1 if k[0] == "a" else 27), k


def test_fused_form_in_the_middle_of_a_pass_leaves_no_potential():
    """Where even one replica's lists do not fit, the replicas before it must not
    leave their part of pot: the fused form has none (pot_full has it)."""
    p = ics.lattice(24, seed=6, rms_cells=0.3, soft_cells=0.3)
    with sim(precision="mixed", max_particles_per_leaf=4, theta=0.4, periodic=True, n_replicas=1) as s:
        s.set_list_region(64)
        s.set_particles(p)
        s.set_alloc_limit(8 * (1024 * 8583 + 148 * 7 * 4 * 64))  # 8583 buckets
        s.start_down()
        assert s.counters()["n_buckets"] == 8583
        first, n1 = s.accelerations(), s.counters()["launches"]
        s.start_down()  # fused from the first replica on
        second, n2 = s.accelerations(), s.counters()["launches"]
    assert n1 != n2
    for k in OUT:
        assert np.abs(first[k] - second[k]).max() < 1e-5 * (1 if k[0] == "a" else 9), k
