"""Values read before the previous kernel has ended (pdl_enter, csrc/kernels.cuh)
must still be the newest: a single domain against the same job in a batch, whose
kernels read everything after it, and a packed lmesh against its lists, with the
caller's own values written between steps.  Every field bit for bit; one-cycle
graphs, graphs of four after 256 cycles, and one launch for a whole run."""
import numpy as np
import pytest

import lmesh

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "ss", "x", "y", "z", "xd", "yd", "zd"]


def nudge(s, rng_seed, domain=0):
    rng = np.random.default_rng(rng_seed)
    for f, scale in (("x", 1e-4), ("yd", 1e-3), ("e", 1e-3), ("q", 1e-3), ("elemMass", 1e-4),
                     ("nodalMass", 1e-4)):
        a = s.field(f, domain)
        s.set_field(f, a * (1.0 + scale * rng.random(a.shape)), domain)


def same(a, b):
    assert a.state() == b.state()
    for f in FIELDS:
        assert np.array_equal(a.field(f), b.field(f)), f


@pytest.mark.parametrize("nx,steps", [(2, (1, 3, 270, 9)), (9, (1, 2, 5)), (24, (1, 4, 260, 8))])
def test_single_domain(lulesh, nx, steps):
    with lulesh.LuleshSet(nx=nx, its=-1) as a, \
            lulesh.LuleshSet.batch([lulesh.JobSpec(nx), lulesh.JobSpec(2, its=1)]) as b:
        for k, n in enumerate(steps):
            a.step(n), b.step(n)
            same(a, b)
            if nx > 2:
                nudge(a, k), nudge(b, k)
        assert a.run_graph(12) == b.run_graph(12)
        same(a, b)


@pytest.mark.parametrize("nx", [3, 12])
def test_lmesh(lulesh, tmp_path, nx):
    rng = np.random.default_rng(nx)
    path = str(tmp_path / "m.lmesh")
    lmesh.write(path, lmesh.renumber(lmesh.box(nx), rng.permutation((nx + 1) ** 3),
                                     rng.permutation(nx ** 3)))
    with lulesh.LuleshSet.from_mesh(path) as a, \
            lulesh.LuleshSet.from_mesh(path, flags=lulesh.FLAG_MATERIALIZE) as b:
        for k, n in enumerate((1, 3, 7)):
            a.step(n), b.step(n)
            same(a, b)
            nudge(a, k), nudge(b, k)
        a.step(4), b.step(4)
        same(a, b)


@pytest.mark.parametrize("nx,k", [(2, 2), (6, 3), (13, 4)])
def test_packed_nodes_in_longer_graphs(lulesh, tmp_path, nx, k):
    """Only the first of a graph's cycles packs the nodes anew."""
    rng = np.random.default_rng(nx)
    path = str(tmp_path / "m.lmesh")
    lmesh.write(path, lmesh.renumber(lmesh.box(nx), rng.permutation((nx + 1) ** 3),
                                     rng.permutation(nx ** 3)))
    with lulesh.LuleshSet.from_mesh(path) as a, \
            lulesh.LuleshSet.from_mesh(path, flags=lulesh.FLAG_MATERIALIZE) as b:
        a.set_graph_cycles(k)
        for part, n in enumerate((k, 2 * k + 1, 3 * k)):
            a.step(n), b.step(n)
            same(a, b)
            nudge(a, part), nudge(b, part)
        assert a.run_graph(9) == b.run_graph(9)
        same(a, b)
