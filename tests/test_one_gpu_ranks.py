"""The sharded entry points with several ranks on one GPU: the ranks are threads whose all-gathers go through host memory
(tests/one_gpu_ranks), so that the code around the exchange runs as it is, with 4 and 8 ranks, where the machine has one GPU."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "one_gpu_ranks")


@pytest.fixture(scope="module")
def gather(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("ranks") / "libhostgather.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-soname,libnccl.so.2", os.path.join(HERE, "hostgather.cpp"), "-o", out,
                    "-I/usr/local/cuda/include", "-L/usr/local/cuda/lib64", "-lcudart", "-pthread"], check=True)
    return out


def run(*args):
    r = subprocess.run([sys.executable, os.path.join(HERE, "ranks.py"), *args], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-1000:] + r.stderr[-3000:]
    assert "ranks ok" in r.stdout


@pytest.mark.parametrize("world", [2, 4, 8])
def test_sharded_provers(gather, world):
    run(gather, str(world))


def test_damaged_share(gather):
    run(gather, "4", "damage")
