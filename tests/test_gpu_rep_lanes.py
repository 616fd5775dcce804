"""The reps of a small domain's costliest class shared between lanes (rep_lanes,
csrc/kernels.cu) against the same job in a batch, whose EOS runs every rep of an
element in one thread.  Every rep evaluates the EOS from the same inputs, so all
fields and the time state must be equal bit for bit: classes of 1, 2, 10 and
more reps, one smaller and larger than a warp, with the last group partial;
meshes below a block and to either side of one wave of blocks."""
import numpy as np
import pytest

import lmesh

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "ss", "x", "xd"]


def same(a, b, job=0):
    assert a.state() == b.state(job)
    for f in FIELDS:
        assert np.array_equal(a.field(f), b.field(f, job)), f


@pytest.mark.parametrize("regions,balance,cost", [(1, 1, 1), (2, 1, 0), (3, 1, 1), (11, 1, 1),
                                                  (20, 4, 3), (40, 1, 10)])
@pytest.mark.parametrize("nx,its,bs", [(1, -1, 128), (2, 30, 64), (5, 40, 256), (13, 25, 128),
                                       (48, 4, 128), (52, 4, 128), (53, 4, 64)])
def test_same_as_in_a_batch(lulesh, nx, its, bs, regions, balance, cost):
    job = lulesh.JobSpec(nx, numReg=regions, balance=balance, cost=cost, its=its)
    with lulesh.LuleshSet(nx=nx, numReg=regions, balance=balance, cost=cost, its=its) as a, \
            lulesh.LuleshSet.batch([job, lulesh.JobSpec(2, its=1)]) as b:
        a.set_tuning(elem_block=bs)
        assert a.run() == b.run() == lulesh.OK
        same(a, b)


@pytest.mark.parametrize("nx,its", [(3, 20), (14, 15)])
def test_lists_and_transients(lulesh, tmp_path, nx, its):
    """An lmesh set; one region has one rep, which nothing shares."""
    path = str(tmp_path / "m.lmesh")
    lmesh.write(path, lmesh.box(nx))
    flags = lulesh.FLAG_MATERIALIZE
    with lulesh.LuleshSet.from_mesh(path, its=its, flags=flags) as a, \
            lulesh.LuleshSet.from_mesh(path, numReg=1, its=its, flags=flags) as b:
        assert a.run() == b.run() == lulesh.OK
        same(a, b)
        for f in ("ql", "qq"):
            assert np.array_equal(a.field(f), b.field(f)), f
