"""Host rules of a set that depend on a build switch, compiled here with the
switch on (nvcc, host code only is run; no GPU)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, REPO

_PROBE = r"""
#include <cstdio>
#include "set.hpp"
static int rule(int tp, int ndom, int nx)
{
    lulesh_set s;
    lulesh::DomDev D{};
    D.numNode = (nx + 1) * (nx + 1) * (nx + 1);
    s.tp = tp;
    s.ndom = ndom;
    s.hdoms.assign(ndom, D);
    return s.inline_increment();
}
int main()
{
    std::printf("%d%d %d%d %d%d %d%d %d%d\n", rule(1, 1, 6), rule(2, 8, 6), rule(1, 1, 66),
                rule(1, 1, 67), rule(2, 8, 24), rule(2, 8, 25), rule(3, 27, 15), rule(3, 27, 16),
                rule(1, 5, 28), rule(1, 6, 28));
    return 0;
}
"""


@pytest.mark.parametrize("flags,want", [
    ((), "11 10 10 10 10"), (("-DLULESH_FUSED_POSVEL_SYNC=1",), "10 10 00 00 10")])
def test_increment_inside_the_kernels(tmp_path, flags, want):
    """Which sets' kernels make the time increment: single domains to -s 66, sets
    of several domains to one wave.  The PosVel sync kernel gates on the time state that the increment inside
    the kernels commits only after it: a build with that kernel keeps the
    increment's own launch in subdomain sets."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "probe.cu", str(tmp_path / "probe")
    src.write_text(_PROBE)
    # the probe's set uses the cache's symbols in functions it does not call
    stub = tmp_path / "stub.cpp"
    stub.write_text('#include "block_cache.hpp"\nnamespace lulesh { void block_put(Block *) {} '
                    'void block_free(Block *) {} }\n')
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", *flags,
                    "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(REPO, "include"), "-o",
                    exe, str(src), str(stub)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.stdout.strip() == want, r.stdout + r.stderr
