"""A problem of one part driven phase by phase (lulesh_part_phase, as a program
written for several GPUs drives it on one) equals lulesh_step: the time
increment is a phase of its own there, also in sets small enough that
lulesh_step's kernels make it themselves.  Every field and the time state bit
for bit, the two ways of stepping also in turn on one set."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "ss", "vdov", "x", "y", "z", "xd", "yd", "zd"]


def same(a, b):
    assert a.state() == b.state()
    for d in range(a.num_domains):
        for f in FIELDS:
            assert np.array_equal(a.field(f, d), b.field(f, d)), (d, f)


@pytest.mark.parametrize("nx,tp", [(2, 1), (12, 1), (30, 1), (70, 1), (6, 2), (20, 2), (4, 3)])
def test_phases_equal_steps(lulesh, nx, tp):
    torch = pytest.importorskip("torch")
    import distributed as D

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        part = D.GpuPart(nx, tp, 1, 0, device=0, stream=stream)
        eng = D.Engine([part], D.LocalTransport())
        eng.setup()
        eng.run(9)
    torch.cuda.synchronize()
    with lulesh.LuleshSet(nx=nx, tp=tp, its=-1, device=0) as s:
        s.step(9)
        same(part.set, s)
        part.set.step(5)
        s.step(5)
        same(part.set, s)
        with torch.cuda.stream(stream):
            eng.run(3)
        torch.cuda.synchronize()
        s.step(3)
        same(part.set, s)
    part.close()
