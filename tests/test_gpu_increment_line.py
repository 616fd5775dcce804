"""Both sides of the line up to which a set's kernels make the time increment
themselves (inline_increment, csrc/set.hpp), for sets of several domains: 2x2x2
of -s 24 and 25 against the undecomposed mesh, batches of five and six jobs of
-s 28 against the jobs alone.  Fields and time states bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [24, 25])
def test_subdomains(lulesh, nx):
    G, cycles = 2 * nx, 10
    with lulesh.LuleshSet(nx=G, its=cycles) as whole, \
            lulesh.LuleshSet(nx=nx, tp=2, its=cycles) as sub:
        assert whole.run() == sub.run() == lulesh.OK
        assert whole.state() == sub.state()
        for f, k in (("x", 1), ("zd", 1), ("e", 0), ("q", 0)):
            want = whole.field(f).reshape((G + k,) * 3)
            for r in range(8):
                c, w, p = r % 2 * nx, r // 2 % 2 * nx, r // 4 * nx
                got = sub.field(f, domain=r)[:(nx + k) ** 3].reshape((nx + k,) * 3)
                assert np.array_equal(got, want[p:p + nx + k, w:w + nx + k, c:c + nx + k]), (r, f)


@pytest.mark.parametrize("jobs", [5, 6])
def test_batches(lulesh, jobs):
    its = [6 + 5 * j for j in range(jobs)]
    with lulesh.LuleshSet.batch([lulesh.JobSpec(28, its=i) for i in its]) as b:
        assert b.run_graph() == lulesh.OK
        for j, i in enumerate(its):
            with lulesh.LuleshSet(nx=28, its=i) as s:
                assert s.run() == lulesh.OK
                assert b.state(j) == s.state()
                for f in ("e", "x", "yd", "v"):
                    assert np.array_equal(b.field(f, j), s.field(f)), (j, f)
