"""The cut of a contraction among the blocks of k_from_right_bytes (csrc/from_right_plan.hpp), walked on the CPU."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plan") / "libfromright.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", os.path.join(HERE, "hostmath", "from_right_plan_host.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    lib.zkf_walk.argtypes = [ctypes.c_uint64, ctypes.c_uint64, ctypes.c_int, ctypes.c_void_p]

    def call(lo_n, hi_n, sm):
        out = (ctypes.c_uint64 * 5)()
        return lib.zkf_walk(lo_n, hi_n, sm, out), list(out)

    return call


@pytest.mark.parametrize("sm", [148, 132, 3, 7])
def test_every_step_and_slot_once(walk, sm):
    crossed = 0
    for n in range(9, 25):
        for hi in range(9, n + 1):
            wrong, (groups, steps, per, blocks, slots) = walk(1 << (n - hi), 1 << hi, sm)
            assert wrong == 0, (n, hi, wrong)
            crossed += per % steps != 0 and steps % per != 0
    assert crossed  # pieces that cross from one column group to the next, or end inside one


@pytest.mark.parametrize("lo_n,hi_n", [(1, 513), (3, 1000), (17, 777), (33, 4097), (1000, 515), (4095, 8191)])
def test_ragged_shapes(walk, lo_n, hi_n):
    """Shapes that are no powers of two: the plan takes them all alike."""
    for sm in (148, 3):
        wrong, _ = walk(lo_n, hi_n, sm)
        assert wrong == 0


def test_largest_pieces(walk):
    """More steps than the blocks of a wave may take with exact sums: more blocks than places."""
    wrong, (_, steps, per, blocks, slots) = walk(1, 1 << 30, 148)
    assert wrong == 0 and per == 1024 and blocks > 296 and slots == steps // 1024
