"""The EOS kernel's block order (eos_block, csrc/kernels.cu): costly blocks are
spread among the others, so every slot must still be visited exactly once.
An EOS result does not depend on the regions, their sizes or the rep counts, so
every field must equal the one-region run's bit for bit: no costly class, one
smaller than a block, ones of several blocks with the last partial, and one
too large to spread; meshes below, at and past a block, and of ragged size."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "ss", "x", "xd"]


@pytest.mark.parametrize("nx", [3, 8, 17, 24])
@pytest.mark.parametrize("regions,balance,cost", [(2, 1, 0), (11, 1, 1), (11, 4, 4), (20, 2, 4),
                                                  (40, 1, 10)])
def test_every_slot_once(lulesh, nx, regions, balance, cost):
    out = []
    for r, b, c in ((1, 1, 1), (regions, balance, cost)):
        with lulesh.LuleshSet(nx=nx, numReg=r, balance=b, cost=c, its=12) as s:
            assert s.run() == lulesh.OK
            out.append(([s.field(f) for f in FIELDS], s.state()))
    assert out[0][1] == out[1][1]
    for f, a, b in zip(FIELDS, out[0][0], out[1][0]):
        assert np.array_equal(a, b), f
