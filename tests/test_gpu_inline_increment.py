"""The time increment inside the cycle's kernels (small FP64 sets) against the
k_time_increment launch: lmesh boxes in a box's own order keep the launch and
compute the structured run's bits, so both must agree cycle by cycle, through
the cycle cap, the stop time and an error, and a batch's jobs must each stop at
their own cap with their blocks still in the launches."""
import numpy as np
import pytest

import lmesh

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "ss", "x", "xd"]


@pytest.mark.parametrize("nx,its", [(1, -1), (2, 17), (5, -1), (6, 9), (16, 5)])
def test_same_as_the_launch(lulesh, tmp_path, nx, its):
    path = str(tmp_path / "m.lmesh")
    lmesh.write(path, lmesh.box(nx))

    def deposit(s):  # the lmesh run deposits the -s 45 energy at any size
        e = np.zeros(nx ** 3)
        e[0] = 3.948746e7
        s.set_field("e", e)

    with lulesh.LuleshSet(nx=nx, its=its) as a, lulesh.LuleshSet.from_mesh(path, its=its) as b:
        deposit(a), deposit(b)
        dt = lulesh.JobState(time=0.0, deltatime=1e-7)
        for s in (a, b):
            s.host_cycle(dt)
        for _ in range(4):
            a.step(3), b.step(3)
            assert a.state() == b.state()
        assert a.run() == b.run() == lulesh.OK
        assert a.state() == b.state() and a.state()["done"] == 1
        for f in FIELDS:
            assert np.array_equal(a.field(f), b.field(f)), f
        c = a.state()["cycle"]
        a.step(2)
        assert a.state()["cycle"] == c


@pytest.mark.parametrize("tp", [1, 2])
def test_error_stops_at_the_launch_form_cycle(lulesh, tp):
    """A volume error found by the force kernel ends the job at the next
    cycle's start, with the erring cycle counted."""
    with lulesh.LuleshSet(nx=4, tp=tp, its=-1) as s:
        s.step(3)
        v = s.field("v")
        v[5] = -1.0
        s.set_field("v", v)
        assert s.run() == lulesh.VOLUME_ERROR
        st = s.state()
        assert (st["cycle"], st["bad_elem"], st["done"]) == (4, 5, 1)


def test_jobs_of_a_batch_stop_alone(lulesh):
    jobs = [lulesh.JobSpec(nx, its=its) for nx, its in ((3, 4), (9, 30), (1, 11), (6, 1))]
    with lulesh.LuleshSet.batch(jobs) as b:
        assert b.run() == lulesh.OK
        for j, spec in enumerate(jobs):
            with lulesh.LuleshSet(nx=spec.nx, its=spec.its) as s:
                assert s.run() == lulesh.OK
                # (one element reaches the stop time in its first cycle)
                assert b.state(j) == s.state() and 1 <= b.state(j)["cycle"] <= spec.its
                for f in FIELDS:
                    assert np.array_equal(b.field(f, j), s.field(f)), (j, f)
