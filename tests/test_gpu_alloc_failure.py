"""Refused device allocations (pt_set_alloc_limit, a host-side limit: nothing is
allocated to make room scarce).  A pass that fails behind the sort has moved the
particles, so the results of the pass before it are refused until a pass
succeeds; the handle stays usable, and its next pass equals a fresh handle's."""
import numpy as np
import pytest

from paratreet_b200 import ics

pytestmark = pytest.mark.gpu

OUT = ("ax", "ay", "az", "pot", "pot_full")


def sim(**kw):
    from paratreet_b200.gravity import GravitySimulation
    return GravitySimulation(**kw)


def refused(call, code):
    from paratreet_b200._lib import PtError
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
