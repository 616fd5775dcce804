"""Several cycles per graph launch: lulesh_run_graph's loop takes four a turn
and the cap's rest after it, and lulesh_step goes over to four-cycle graphs
after 256 cycles.  Any cap, and any split of a run into steps, ends in the
state of single cycles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "x", "xd"]


def _same(a, b, jobs=1):
    for j in range(jobs):
        assert a.state(j) == b.state(j)
        for f in FIELDS:
            assert np.array_equal(a.field(f, j), b.field(f, j)), f


@pytest.mark.parametrize("caps", [(1,), (3, 1), (4,), (5, 2, 6), (8, 3)])
def test_run_graph_caps(lulesh, caps):
    with lulesh.LuleshSet(nx=6) as a, lulesh.LuleshSet(nx=6) as b:
        for cap in caps:
            assert a.run_graph(max_cycles=cap) == lulesh.OK
        for _ in range(sum(caps)):
            b.step(1)
        assert a.state()["cycle"] == sum(caps)
        _same(a, b)


@pytest.mark.parametrize("kind", ["single", "batch", "subdomains"])
def test_steps_across_the_switch(lulesh, kind):
    def make():
        if kind == "batch":
            return lulesh.LuleshSet.batch([lulesh.JobSpec(7, its=270), lulesh.JobSpec(20, its=290)])
        return lulesh.LuleshSet(nx=20, tp=1) if kind == "single" else lulesh.LuleshSet(nx=10, tp=2)

    with make() as a, make() as b:
        for n in (200, 55, 1, 7, 4, 3, 0, 18):
            a.step(n)
        for _ in range(288):
            b.step(1)
        _same(a, b, 2 if kind == "batch" else 1)
