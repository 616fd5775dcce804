"""Creating and closing sets touches no stream of the caller's: a capture of the
calling thread's default stream (cudaStreamPerThread, relaxed mode, as
lulesh_create allocates) goes on through it and stays empty (in a child
process, whose streams nothing else uses).  What is kept from closed sets goes
back to the driver on request."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_CHILD = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import lulesh_b200 as L
rt = ctypes.CDLL("libcudart.so.12")
PER_THREAD, RELAXED = ctypes.c_void_p(2), 2
def use():
    with L.LuleshSet(nx=12, its=-1) as s:
        s.step(3)
        s.sync()
use()
graph, nodes = ctypes.c_void_p(), ctypes.c_size_t(99)
assert rt.cudaStreamBeginCapture(PER_THREAD, RELAXED) == 0
use(); use()
assert rt.cudaStreamEndCapture(PER_THREAD, ctypes.byref(graph)) == 0
assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(nodes)) == 0
assert nodes.value == 0, nodes.value
use()
print("CAPTURE_OK")
"""


def test_capture_of_the_thread_stream_survives(lulesh):
    r = subprocess.run([sys.executable, "-c", _CHILD, lulesh.HERE], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "CAPTURE_OK" in r.stdout, r.stdout + r.stderr


def test_release_memory(lulesh):
    torch = pytest.importorskip("torch")
    size = lulesh.footprint_bytes([lulesh.JobSpec(70)])
    lulesh.release_memory()
    with lulesh.LuleshSet(nx=70, its=-1) as s:
        s.step(1)
        s.sync()
        used = torch.cuda.mem_get_info()[0]
    kept = torch.cuda.mem_get_info()[0]
    assert kept - used < 0.1 * size
    lulesh.release_memory()
    assert torch.cuda.mem_get_info()[0] - kept > 0.9 * size
