"""The packed kernels of scattered meshes at the sizes where they can go wrong:
the smallest mesh that runs packed, whole and partial warps and blocks, nodes
with one corner and with eight.  Each mesh is on the packed side of the rule,
and its fields equal bit for bit those of the same mesh run from its lists (the
materialize flag), from a state in which every element moves."""
import numpy as np
import pytest

import lmesh
from test_scattered_rule import islands, rule, shuffled

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "ss", "x", "y", "z", "xd", "yd", "zd", "delv", "vdov", "arealg",
          "delx_xi", "delv_eta", "fx_elem", "fy_elem", "fz_elem"]


@pytest.mark.parametrize("mesh", [islands(n) for n in (28, 31, 32, 60, 127, 128, 156, 256)] +
                         [shuffled(n) for n in (7, 8, 9, 11)],
                         ids=lambda m: f"{m.num_elem}-{m.num_node}")
def test_packed_equals_lists(lulesh, tmp_path, mesh):
    assert rule(tmp_path, mesh)[1]
    rng = np.random.default_rng(mesh.num_elem)
    path = str(tmp_path / "m.lmesh")
    lmesh.write(path, mesh)
    with lulesh.LuleshSet.from_mesh(path) as a, \
            lulesh.LuleshSet.from_mesh(path, flags=lulesh.FLAG_MATERIALIZE) as b:
        size = {f: a.field(f).size for f in ("e", "p", "q", "ss", "xd")}
        values = {"e": rng.uniform(1.0, 2.0, size["e"]), "p": rng.uniform(0.5, 1.0, size["p"]),
                  "q": rng.uniform(0.0, 0.1, size["q"]), "ss": rng.uniform(0.5, 1.0, size["ss"])}
        values.update({f: rng.uniform(-1.0, 1.0, size["xd"]) for f in ("xd", "yd", "zd")})
        for s in (a, b):
            for f, v in values.items():
                s.set_field(f, v)
        for run in (lambda s: s.step(1), lambda s: s.step(2), lambda s: s.set_graph_cycles(3),
                    lambda s: s.step(7), lambda s: s.run_graph(6)):
            run(a), run(b)
            assert a.state() == b.state() and a.state()["status"] == lulesh.OK
            for f in FIELDS:
                assert np.array_equal(a.field(f), b.field(f)), f
        assert a.state()["cycle"] == 16 and np.count_nonzero(a.field("vdov")) == size["e"]
