"""Corner forces of a scattered mesh, whose cycle keeps them packed: fx_elem,
fy_elem and fz_elem read as those of the same mesh run from its lists (the
materialize flag), bit for bit, however the cycles are run and however the
arrays are read: by name, through device pointers, in a checkpoint, from a
graph of the caller's; and what is written to them stays until the next cycle."""
import numpy as np
import pytest

import lmesh
from test_gpu_handed_out import _Array, _capture, _view

pytestmark = pytest.mark.gpu

CORNERS = ["fx_elem", "fy_elem", "fz_elem"]


def same(a, b):
    for f in CORNERS + ["e", "x"]:
        assert np.array_equal(a.field(f), b.field(f)), f


@pytest.fixture(params=[7, 13])
def sets(lulesh, tmp_path, request):
    nx = request.param
    rng = np.random.default_rng(nx)
    path = str(tmp_path / "m.lmesh")
    lmesh.write(path, lmesh.renumber(lmesh.box(nx), rng.permutation((nx + 1) ** 3),
                                     rng.permutation(nx ** 3)))
    with lulesh.LuleshSet.from_mesh(path) as a, \
            lulesh.LuleshSet.from_mesh(path, flags=lulesh.FLAG_MATERIALIZE) as b:
        yield a, b


def test_by_name(lulesh, sets):
    a, b = sets
    same(a, b)
    for run in (lambda s: s.step(1), lambda s: s.step(6), lambda s: s.run_graph(5),
                lambda s: s.host_cycle(), lambda s: s.profile_phases(2), lambda s: s.step(270),
                lambda s: s.step(9)):
        run(a), run(b)
        assert a.state() == b.state()
        same(a, b)


def test_checkpoint_writes_and_a_finished_run(lulesh, sets):
    a, b = sets
    a.step(3), b.step(3)
    saved = a.checkpoint(), b.checkpoint()
    n = a.field("fx_elem").nbytes * 3
    assert n > 0 and saved[0].count(a.field("fx_elem").tobytes()) == 1
    a.step(4), b.step(4)
    a.restore(saved[0]), b.restore(saved[1])
    same(a, b)
    a.step(5), b.step(5)
    mine = np.arange(a.field("fy_elem").size, dtype=np.float64)  # with the padding
    for s in (a, b):
        s.set_field("fy_elem", mine)
        assert np.array_equal(s.field("fy_elem"), mine)
    same(a, b)
    a.autotune(trial_cycles=2, rounds=1)
    same(a, b)
    assert a.run() == b.run() == lulesh.OK
    same(a, b)
    for s in (a, b):
        s.set_field("fz_elem", mine)
        s.step(2)  # no work left: nothing is written
    same(a, b)


def test_through_pointers(lulesh, sets):
    torch = pytest.importorskip("torch")
    a, b = sets
    stream = torch.cuda.Stream()
    a.set_stream(stream.cuda_stream)
    a.step(2), b.step(2)
    w, n = _view(lulesh, a), b.field("fx_elem").size
    views = [torch.as_tensor(_Array(getattr(w, f), n), device="cuda") for f in CORNERS]

    def check():
        with torch.cuda.stream(stream):
            got = [v.cpu().numpy() for v in views]
        for f, g in zip(CORNERS, got):
            assert np.array_equal(g, b.field(f)), f

    check()
    for run in (lambda s: s.step(1), lambda s: s.step(5), lambda s: s.run_graph(6),
                lambda s: s.host_cycle()):
        run(a), run(b)
        check()
    g = _capture(torch, a, stream, 3)
    for _ in range(2):
        with torch.cuda.stream(stream):
            g.replay()
        b.step(3)
        check()
    del views, g
    torch.cuda.synchronize()


def test_captured_before_any_pointer(lulesh, sets):
    torch = pytest.importorskip("torch")
    a, b = sets
    stream = torch.cuda.Stream()
    g = _capture(torch, a, stream, 4)
    with torch.cuda.stream(stream):
        g.replay()
    torch.cuda.synchronize()
    b.step(4)
    same(a, b)
    del g


@pytest.mark.parametrize("k", [1, 3])
def test_pointers_with_longer_graphs(lulesh, tmp_path, k):
    """Several graph launches a call, whole or with a rest, before and after the
    set takes four cycles a graph by itself, and a cap inside a graph."""
    torch = pytest.importorskip("torch")
    path = str(tmp_path / "m.lmesh")
    rng = np.random.default_rng(9)
    lmesh.write(path, lmesh.renumber(lmesh.box(9), rng.permutation(1000), rng.permutation(729)))
    with lulesh.LuleshSet.from_mesh(path, its=320) as a, \
            lulesh.LuleshSet.from_mesh(path, its=320, flags=lulesh.FLAG_MATERIALIZE) as b:
        stream = torch.cuda.Stream()
        a.set_stream(stream.cuda_stream)
        w, n = _view(lulesh, a), b.field("fx_elem").size
        views = [torch.as_tensor(_Array(getattr(w, f), n), device="cuda") for f in CORNERS]
        a.set_graph_cycles(k)
        for cycles in (7, 9, 2, 250, 8, 9, 1, 31, 7, 4):
            a.step(cycles), b.step(cycles)
            with torch.cuda.stream(stream):
                got = [v.cpu().numpy() for v in views]
            for f, g in zip(CORNERS, got):
                assert np.array_equal(g, b.field(f)), (cycles, f)
        assert a.state() == b.state() and a.state()["cycle"] == 320
        del views
        torch.cuda.synchronize()
