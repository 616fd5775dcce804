"""Scattered meshes (random node and element numbers) run from packed nodes and
corners (pack_scattered_mesh, csrc/set.cu); the same mesh with the materialize
flag runs from the lists.  The same arithmetic in the same order: every field
bit for bit, from one element to several blocks, and what the caller writes
between cycles counts."""
import numpy as np
import pytest

import lmesh

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "ss", "x", "y", "z", "xd", "yd", "zd", "delv", "vdov", "arealg"]


@pytest.mark.parametrize("nx", [1, 2, 5, 6, 12, 17])
def test_packed_equals_lists(lulesh, tmp_path, nx):
    rng = np.random.default_rng(nx)
    path = str(tmp_path / "m.lmesh")
    lmesh.write(path, lmesh.renumber(lmesh.box(nx), rng.permutation((nx + 1) ** 3),
                                     rng.permutation(nx ** 3)))
    with lulesh.LuleshSet.from_mesh(path) as a, \
            lulesh.LuleshSet.from_mesh(path, flags=lulesh.FLAG_MATERIALIZE) as b:
        saved = None
        for part in range(3):
            a.step(7)
            b.step(7)
            assert a.state() == b.state()
            for f in FIELDS:
                assert np.array_equal(a.field(f), b.field(f)), (part, f)
            if part == 0:
                saved = a.checkpoint()
            kick = 1e-3 * rng.uniform(-1.0, 1.0, a.field("xd").size)
            for s in (a, b):
                s.set_field("xd", s.field("xd") + kick)
        a.restore(saved)
        assert a.state()["cycle"] == 7
        a.run_graph(max_cycles=5)
        with lulesh.LuleshSet.from_mesh(path) as c:
            c.step(12)
            for f in FIELDS:
                assert np.array_equal(a.field(f), c.field(f)), f
