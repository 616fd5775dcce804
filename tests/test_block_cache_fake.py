"""The memory kept from closed sets (csrc/block_cache.cu) over a fake runtime,
without a GPU: what is kept and how much, that every allocation which finds
the device full gets the kept blocks first, that the program can ask for
them, and that neither an unreadable context id nor a device reset loses or
reuses a block wrongly."""
import os
import subprocess

from conftest import PKG, REPO


def test_block_cache_over_a_fake_device(tmp_path):
    exe = str(tmp_path / "blocks")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-o", exe, "-x", "c++",
                    os.path.join(REPO, "tests", "fake_cudart.cpp"),
                    os.path.join(PKG, "csrc", "block_cache.cu"), "-I" + cuda,
                    "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(REPO, "include"),
                    "-lpthread"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "BLOCKS_OK" in r.stdout, r.stdout + r.stderr
