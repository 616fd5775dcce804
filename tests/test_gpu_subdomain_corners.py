"""A small 2x2x2 set finds the corner forces across its subdomains' faces by
arithmetic (gather_corners_few, csrc/kernels.cu), a large one by the neighbours'
records: both must give the undecomposed mesh's fields bit for bit, from one
element a subdomain to either side of the line (-s 32 and 33)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,cycles", [(1, 60), (2, 60), (7, 40), (16, 20), (32, 8), (33, 8)])
def test_equals_the_whole_mesh(lulesh, nx, cycles):
    G = 2 * nx
    with lulesh.LuleshSet(nx=G, its=cycles) as whole, \
            lulesh.LuleshSet(nx=nx, tp=2, its=cycles) as sub:
        assert whole.run() == sub.run() == lulesh.OK
        for f, k in (("x", 1), ("yd", 1), ("zd", 1), ("e", 0), ("q", 0), ("v", 0)):
            want = whole.field(f).reshape((G + k,) * 3)
            for r in range(8):
                c, w, p = r % 2 * nx, r // 2 % 2 * nx, r // 4 * nx
                got = sub.field(f, domain=r)[:(nx + k) ** 3].reshape((nx + k,) * 3)
                assert np.array_equal(got, want[p:p + nx + k, w:w + nx + k, c:c + nx + k]), (r, f)
