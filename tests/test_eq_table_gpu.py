"""zk_eq_table at the sizes where its launch changes: below, at and above the stretch of entries one block makes, one stretch
per block, and several.  Entry x of the table is prod_j (x_j ? r_j : 1 - r_j) (util/poly.rs:573-618)."""
import ctypes
import random

import numpy as np
import pytest

import pyoracle as o
from zkes_b200._lib import ZK_MEM_HOST, check, lib
from zkes_b200.field import from_mont_array, to_mont_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [0, 1, 2, 5, 9, 10, 11, 12, 16, 18, 19, 20])
def test_eq_table(ctx, k):
    rnd = random.Random(k)
    point = [rnd.choice([0, 1, o.R_MOD - 1]) if rnd.random() < 0.1 else rnd.randrange(o.R_MOD) for _ in range(k)]
    pm = to_mont_array(point) if k else np.zeros((1, 4), dtype=np.uint64)
    out = np.zeros((1 << k, 4), dtype=np.uint64)
    check(lib.zk_eq_table(ctx.handle, k, ctypes.c_void_p(pm.ctypes.data), ctypes.c_void_p(out.ctypes.data), ZK_MEM_HOST), "zk_eq_table")
    size = 1 << k
    at = range(size) if size <= 4096 else sorted({0, 1, size - 1, size - 2, 1023, 1024, size // 2 - 1, size // 2} |
                                                 {rnd.randrange(size) for _ in range(3000)})
    got = from_mont_array(out[list(at)])
    for x, v in zip(at, got):
        want = 1
        for j, r in enumerate(point):
            want = want * (r if (x >> j) & 1 else 1 - r) % o.R_MOD
        assert v == want, x
