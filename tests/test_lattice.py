"""lattice() (csrc/lulesh_dev.h): element and node numbers taken apart by a
multiplication, against integer division: every edge a domain can have (and the
node edge one above it), at the ends of every range of the quotient that could
round the wrong way."""
import ctypes
import os
import subprocess

import numpy as np

from conftest import PKG

LIB = os.path.join(PKG, "liblulesh_host.so")


def test_every_edge():
    if not os.path.exists(LIB):
        subprocess.run(["make", "-C", PKG, "liblulesh_host.so"], check=True)
    lib = ctypes.CDLL(LIB)
    lib.lulesh_host_lattice.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
    rng = np.random.default_rng(0)
    for d in range(1, 647):
        top = d ** 3 + 4096  # threads past the end compute it too
        k = np.concatenate([rng.integers(0, top // d + 1, 200), np.arange(min(50, top // d + 1)),
                            np.arange(max(0, top // d - 50), top // d + 1)])
        n = np.unique(np.clip(np.concatenate([k * d - 1, k * d, k * d + 1, [0, d ** 3 - 1, top]]), 0,
                              top)).astype(np.int32)
        if d == 1:
            n = np.zeros(1, np.int32)  # its one element
        out = np.empty((n.size, 3), np.int32)
        lib.lulesh_host_lattice(d, n.ctypes.data, n.size, out.ctypes.data)
        want = np.stack([n % d, n // d % d, n // d // d], axis=1)
        assert np.array_equal(out, want), d
