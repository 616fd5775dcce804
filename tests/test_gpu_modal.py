"""The element arithmetic in trilinear modes (csrc/elem_modal.cuh) against the
oracle's corner-by-corner form, on strongly distorted elements: one cycle
from a random state, every force, velocity and gradient.

Tolerance: the oracle sums raw coordinates for its hourglass modes, so its
rounding error is eps times the cube of (mesh edge / element edge), at most
1.1e-16 * 11^3 = 1.5e-13 here, over some tens of terms: 1e-11 of each field's
largest magnitude."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-11
NODE = ["x", "y", "z", "xd", "yd", "zd", "xdd", "ydd", "zdd", "fx", "fy", "fz"]
ELEM = ["vnew", "delv", "arealg", "vdov", "delx_xi", "delx_eta", "delx_zeta", "delv_xi",
        "delv_eta", "delv_zeta", "fx_elem", "fy_elem", "fz_elem"]


@pytest.mark.parametrize("nx,warp", [(1, 0.2), (2, 0.15), (5, 0.15), (11, 0.15), (11, 0.0)])
def test_distorted_elements_match_the_oracle(lulesh, oracle_mod, nx, warp):
    rng = np.random.default_rng(nx)
    orc = oracle_mod.Oracle(nx)
    with lulesh.LuleshSet(nx=nx, its=1, flags=lulesh.FLAG_MATERIALIZE) as gs:
        n, e = (nx + 1) ** 3, nx ** 3
        state = {f: orc.field(f)[:n] + warp * 1.125 / nx * rng.uniform(-1, 1, n)
                 for f in ("x", "y", "z")}
        state.update({f: rng.uniform(-50.0, 50.0, n) for f in ("xd", "yd", "zd")})
        state.update({f: rng.uniform(0.0, 4e3, e) for f in ("e", "p", "q")})
        state["v"] = rng.uniform(0.8, 1.2, e)
        state["ss"] = rng.uniform(10.0, 80.0, e)
        for f, a in state.items():
            gs.set_field(f, a)
            orc.set_real_field(f, a)
        assert orc.step() == 0
        assert gs.run() == lulesh.OK
        for f in NODE + ELEM:
            g, o = gs.field(f), orc.field(f)
            m = min(g.size, o.size, n if f in NODE else 8 * e if f.endswith("_elem") else e)
            if f.endswith("_elem"):  # [8][padded]: the elements of each corner
                ep = (e + 31) // 32 * 32
                g, o = (a[:8 * ep].reshape(8, ep)[:, :e].ravel() for a in (g, o))
                m = 8 * e
            diff, scale = np.max(np.abs(g[:m] - o[:m])), np.max(np.abs(o[:m]))
            assert diff <= RTOL * scale, (f, diff, scale)
    orc.close()


@pytest.mark.parametrize("sizes", [(1, 7), (5, 13), (32, 2)])
def test_mixed_records_by_value_and_by_table(lulesh, sizes):
    """A mixed single domain takes its record by value, a mixed batch from the
    table: the same kernels' arithmetic, the same bits."""
    jobs = [lulesh.JobSpec(nx, its=15) for nx in sizes]
    with lulesh.LuleshSet.batch(jobs, flags=lulesh.FLAG_MIXED) as b:
        assert b.run() == lulesh.OK
        for j, spec in enumerate(jobs):
            with lulesh.LuleshSet(nx=spec.nx, its=15, flags=lulesh.FLAG_MIXED) as s:
                assert s.run() == lulesh.OK
                for f in ("e", "p", "q", "v", "ss", "x", "y", "z", "xd", "yd", "zd"):
                    assert np.array_equal(b.field(f, j), s.field(f)), (spec.nx, f)
