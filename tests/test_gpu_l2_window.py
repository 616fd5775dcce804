"""Sets that share a stream share its L2 access window: each capture sets it
to the nodes of the set that captures (prepare_capture, csrc/set.cu), whichever
set had it last, and closing a set leaves none."""
import ctypes

import pytest

from test_gpu_handed_out import _view

pytestmark = pytest.mark.gpu

ACCESS_POLICY_WINDOW = 1  # cudaLaunchAttributeAccessPolicyWindow


class _Window(ctypes.Structure):  # cudaAccessPolicyWindow in a cudaLaunchAttributeValue
    _fields_ = [("base", ctypes.c_void_p), ("bytes", ctypes.c_size_t), ("ratio", ctypes.c_float),
                ("hit", ctypes.c_int), ("miss", ctypes.c_int), ("pad", ctypes.c_char * 32)]


def test_each_capture_sets_its_window(lulesh):
    torch = pytest.importorskip("torch")
    rt = ctypes.CDLL("libcudart.so.12")
    stream = torch.cuda.Stream()

    def window():
        w = _Window()
        assert rt.cudaStreamGetAttribute(ctypes.c_void_p(stream.cuda_stream), ACCESS_POLICY_WINDOW,
                                         ctypes.byref(w)) == 0
        return w.base if w.bytes else None

    a, b = lulesh.LuleshSet(nx=30, its=-1), lulesh.LuleshSet(nx=40, its=-1)
    try:
        for s in (a, b):
            s.set_stream(stream.cuda_stream)
        xa, xb = _view(lulesh, a).x, _view(lulesh, b).x
        a.step(1)
        assert window() == xa
        b.step(1)
        assert window() == xb
        a.set_graph_cycles(2)
        a.step(2)
        assert window() == xa
        b.run_graph(4)
        assert window() == xb
        b.close()
        assert window() is None
        a.set_graph_cycles(3)
        a.step(3)
        assert window() == xa
        a.sync()
    finally:
        a.close()
        b.close()
