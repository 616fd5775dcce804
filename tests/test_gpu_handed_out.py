"""Sets whose memory a caller may still be using on a stream of its own
(pointers from lulesh_domain_view_get, a captured step replayed elsewhere, phases
of a part, the Comm calls): lulesh_destroy frees their memory instead of
keeping it for the next set, so that the next set neither overtakes the
caller's work nor is written by it."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _View(ctypes.Structure):  # lulesh_domain_view
    _fields_ = ([(f"i{k}", ctypes.c_int) for k in range(15)] +
                [(n, ctypes.c_void_p) for n in (
                    "nodelist lxim lxip letam letap lzetam lzetap elemBC nodeElemCount "
                    "nodeElemStart nodeElemCornerList symmX symmY symmZ matElemlist regCSR regReps "
                    "regNumList regElemlist regSorted e p q ql qq v volo delv vdov arealg ss "
                    "elemMass x y z xd yd zd xdd ydd zdd fx fy fz nodalMass vnew delx_xi delx_eta "
                    "delx_zeta delv_xi delv_eta delv_zeta fx_elem fy_elem fz_elem").split()])


class _Array:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False),
                                         "version": 3, "strides": None}


def _view(lulesh, s):
    w = _View()
    assert s.lib.lulesh_domain_view_get(s.h, 0, ctypes.byref(w)) == lulesh.OK
    return w


def _capture(torch, s, stream, n):
    s.set_stream(stream.cuda_stream)
    s.step(0)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        s.step(n)
    return g


@pytest.mark.parametrize("how", ["view", "capture", "phase", "comm"])
def test_memory_goes_back_to_the_driver(lulesh, how):
    torch = pytest.importorskip("torch")
    nx, tp = (40, 2) if how == "comm" else (70, 1)
    size = lulesh.footprint_bytes([lulesh.JobSpec(nx)], tp=tp)
    stream = torch.cuda.Stream()
    s = lulesh.LuleshSet(nx=nx, tp=tp, its=-1)
    s.step(1)
    if how == "view":
        _view(lulesh, s)
    elif how == "capture":
        g = _capture(torch, s, stream, 2)
        del g
    elif how == "phase":
        assert s.lib.lulesh_part_phase(s.h, lulesh.PHASE_TIME_INCREMENT) == lulesh.OK
    else:
        s.comm_sync_posvel(-1)
    s.sync()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s.close()
    assert torch.cuda.mem_get_info()[0] - before > 0.9 * size


def test_copy_from_a_view_in_flight(lulesh):
    torch = pytest.importorskip("torch")
    nx = 30
    s = lulesh.LuleshSet(nx=nx, its=-1)
    s.step(20)
    s.sync()
    want = s.field("e")
    src = torch.as_tensor(_Array(_view(lulesh, s).e, nx ** 3), device="cuda")
    side = torch.cuda.Stream()
    dst = torch.empty(nx ** 3, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(50_000_000)  # some 25 ms, then the copy
        dst.copy_(src)
    s.close()
    with lulesh.LuleshSet(nx=nx, its=-1) as t:
        t.step(3)
        t.sync()
    torch.cuda.synchronize()
    assert np.array_equal(dst.cpu().numpy(), want)


def test_replay_on_another_stream_in_flight(lulesh):
    torch = pytest.importorskip("torch")
    nx, n = 30, 60
    with lulesh.LuleshSet(nx=nx, its=-1) as ref:
        first = {f: ref.field(f) for f in ("e", "x", "xd", "nodalMass")}
        ref.step(n)
        after = {f: ref.field(f) for f in ("e", "x", "xd", "v")}
        state = ref.state()
    s = lulesh.LuleshSet(nx=nx, its=-1)
    stream, side = torch.cuda.Stream(), torch.cuda.Stream()
    g = _capture(torch, s, stream, 50)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(16):
            g.replay()
    s.close()
    with lulesh.LuleshSet(nx=nx, its=-1) as t:
        for f, a in first.items():
            assert np.array_equal(t.field(f), a), f
        t.step(n)
        for f, a in after.items():
            assert np.array_equal(t.field(f), a), f
        assert t.state() == state
    torch.cuda.synchronize()
    del g
