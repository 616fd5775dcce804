"""Sets from the memory of closed ones (csrc/block_cache.cu): the same results
whatever the blocks held before, blocks of very different sizes, several
threads at once, and a device reset between two sets (in a child process, whose
own context it ends)."""
import subprocess
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ["e", "p", "q", "v", "ss", "x", "xd", "nodalMass", "nodelist", "eosOrder", "fx_elem"]


def _run(lulesh, nx, **kw):
    with lulesh.LuleshSet(nx=nx, its=12, **kw) as s:
        first = [s.field(f) for f in FIELDS]
        assert s.run() == lulesh.OK
        return first + [s.field(f) for f in FIELDS], s.state()


@pytest.mark.parametrize("order", [(12, 12, 12), (20, 3, 19, 20), (1, 24, 1, 2)])
def test_reused_blocks(lulesh, order):
    want = {nx: _run(lulesh, nx) for nx in set(order)}
    kinds = ({}, {"tp": 2}, {"flags": lulesh.FLAG_MIXED}, {"flags": lulesh.FLAG_HOST_SETUP})
    for nx in order:
        for kw in kinds:  # leave other sets' data in the blocks
            with lulesh.LuleshSet(nx=max(1, nx // 2), its=2, **kw) as s:
                s.run()
        got = _run(lulesh, nx)
        assert got[1] == want[nx][1]
        for a, b in zip(got[0], want[nx][0]):
            assert np.array_equal(a, b)


def test_threads(lulesh):
    want = _run(lulesh, 9)
    bad = []

    def work():
        for _ in range(6):
            got = _run(lulesh, 9)
            if got[1] != want[1] or not all(np.array_equal(a, b) for a, b in zip(got[0], want[0])):
                bad.append(1)

    ts = [threading.Thread(target=work) for _ in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad


_CHILD = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import lulesh_b200 as L
rt = ctypes.CDLL("libcudart.so.12")
def energy():
    with L.LuleshSet(nx=10, its=8) as s:
        assert s.run() == L.OK
        return s.origin_energy()
a = energy(); b = energy()
assert rt.cudaDeviceReset() == 0
c = energy(); d = energy()
assert a == b == c == d, (a, b, c, d)
print("RESET_OK")
"""


def test_after_device_reset(lulesh):
    r = subprocess.run([sys.executable, "-c", _CHILD, lulesh.HERE], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "RESET_OK" in r.stdout, r.stdout + r.stderr
