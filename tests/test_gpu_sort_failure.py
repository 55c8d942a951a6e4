"""The key sort's bounded wait as a tested failure path.

Each digit pass of the onesweep radix sort resolves a tile's offsets by a
look-back over earlier tiles that polls an unpublished tile a bounded number
of times.  With the bound set to 0 a look-back gives up at the first tile it
finds unpublished, which on a multi-tile sort happens in practice on every
pass.  The force pass must then return PT_E_DEVICE naming the sort, stop
before it permutes the particles (look-backs cut short leave no permutation), and
leave the handle usable: with the default bound the next pass equals a fresh
handle's bit for bit.  No wait in this test is left
to run out on its own; the bound only cuts waits short."""
import numpy as np
import pytest

from paratreet_b200 import ics

pytestmark = pytest.mark.gpu


def test_sort_lookback_limit_reports_and_recovers():
    from paratreet_b200._lib import PtError
    from paratreet_b200.gravity import GravitySimulation

    n = 1 << 22  # 1024 tiles of 4096 keys per digit pass
    p = ics.plummer(n, seed=5, soft=1e-3)
    with GravitySimulation(max_particles_per_leaf=32, theta=0.7, precision="fp64") as ref:
        ref.set_particles(p)
        ref.start_down()
        want = ref.accelerations()
    with GravitySimulation(max_particles_per_leaf=32, theta=0.7, precision="fp64") as s:
        s.set_particles(p)
        s.set_sort_spin_limit(0)
        msgs = []
        for _ in range(5):  # each pass of 8 x 1024 tiles x 256 digits races many times
            try:
                s.start_down()
            except PtError as e:
                msgs.append(str(e))
                break
        assert msgs, "no look-back gave up in 5 passes with a spin limit of 0"
        assert "radix sort look-back timed out" in msgs[0]
        s.set_sort_spin_limit()
        s.start_down()
        got = s.accelerations()
    for k in ("ax", "ay", "az", "pot", "pot_full"):
        assert np.array_equal(got[k], want[k]), k


# both tile sizes; with a limit above 0 only some look-backs give up, which is
# what can send a later digit pass past the end (tests/test_sort_lookback_model.py)
@pytest.mark.parametrize("n", [300_001, (1 << 21) + 5])
@pytest.mark.parametrize("polls", [0, 1, 4])
def test_failed_sort_leaves_the_particles(n, polls):
    from paratreet_b200._lib import PtError
    from paratreet_b200.gravity import GravitySimulation

    p = ics.plummer(n, seed=6, soft=1e-3)
    failed = 0
    with GravitySimulation(max_particles_per_leaf=32, theta=1.0, precision="mixed") as s:
        s.set_particles(p)
        s.start_down()  # the particles are in key order, and the alternate buffers full
        want = s.keys()
        s.set_sort_spin_limit(polls)
        for _ in range(6):
            try:
                s.start_down()
            except PtError as e:
                assert "radix sort look-back timed out" in str(e)
                failed += 1
            st = s.state()
            for k in ("x", "y", "z", "vx", "vy", "vz"):
                assert np.array_equal(st[k], p[k]), k
        assert failed or polls > 0
        s.set_sort_spin_limit()
        s.start_down()
        assert np.array_equal(s.keys(), want)


def test_failed_sort_keeps_results_but_no_keys():
    """The accelerations of the pass before a failed sort still line up with the
    particles; its keys were overwritten."""
    from paratreet_b200._lib import PtError
    from paratreet_b200.gravity import GravitySimulation

    n = (1 << 21) + 5
    p = ics.plummer(n, seed=6, soft=1e-3)
    with GravitySimulation(max_particles_per_leaf=32, theta=1.0, precision="mixed") as s:
        s.set_particles(p)
        s.start_down()
        want, keys = s.accelerations(), s.keys()
        s.set_sort_spin_limit(0)
        for _ in range(6):
            try:
                s.start_down()
            except PtError:
                break
        else:
            pytest.fail("no look-back gave up in 6 passes with a spin limit of 0")
        got = s.accelerations()
        for k in want:
            assert np.array_equal(got[k], want[k]), k
        with pytest.raises(PtError) as e:
            s.keys()
        assert e.value.code == -4
        s.set_sort_spin_limit()
        s.start_down()
        assert np.array_equal(s.keys(), keys)
