"""Lists of positions in pinned host memory, which the kernels read where they lie, against the same lists in pageable memory, which
are copied first: whole buffers, parts of one, lists of odd lengths, refused indices."""
import ctypes
import random

import numpy as np
import pytest
import torch

import pyoracle as o
from zkes_b200 import kzh
from zkes_b200._lib import check, lib
from zkes_b200.field import to_mont_array

pytestmark = pytest.mark.gpu
vp = ctypes.c_void_p
N = 9


@pytest.fixture(scope="module")
def srs(ctx):
    rnd = random.Random(4)
    return kzh.KZHSRS.setup(ctx, 2, N, o.G1_GEN, [rnd.randrange(1, 1 << 60) for _ in range(1 << (N // 2))],
                            [rnd.randrange(1, 1 << 60) for _ in range(1 << (N - N // 2))], alpha=7)


def pinned(values, before=0):
    whole = torch.zeros(before + len(values), dtype=torch.int64, pin_memory=True)
    whole[before:] = torch.from_numpy(values.view(np.int64))
    return whole, whole.data_ptr() + 8 * before


def opened(ctx, srs, ptr, count, point):
    out = np.zeros((1 << srs.y_log, 4), dtype=np.uint64)
    rc = lib.zk_sparse_kzh2_open(ctx.handle, srs.handle, count, vp(ptr), None, vp(point.ctypes.data), N, vp(out.ctypes.data))
    return rc, out


def committed(ctx, srs, ptr, count):
    c, dx = np.zeros((1, 8), dtype=np.uint64), np.zeros((1 << srs.x_log, 12), dtype=np.uint64)
    rc = lib.zk_sparse_kzh_commit(ctx.handle, srs.handle, count, vp(ptr), None, vp(c.ctypes.data), vp(dx.ctypes.data))
    return rc, c


def checked(ctx, terms, ptr, counts, weights, point):
    tr = lib.zk_transcript_new(b"p", 1)
    msgs, chal, fin = np.zeros((N * 4, 4), dtype=np.uint64), np.zeros((N, 4), dtype=np.uint64), np.zeros((1, 4), dtype=np.uint64)
    rc = lib.zk_sumcheck_sparse_bool_prove(ctx.handle, N, terms, vp(weights.ctypes.data), vp(ptr), vp(counts.ctypes.data), vp(point.ctypes.data),
                                           None, None, tr, vp(msgs.ctypes.data), vp(chal.ctypes.data), vp(fin.ctypes.data))
    lib.zk_transcript_free(tr)
    return rc, np.concatenate([msgs, chal, fin])


@pytest.mark.parametrize("count,before", [(1, 0), (31, 0), (33, 1), (256, 3), (257, 0), (512, 5)])
def test_same_results(ctx, srs, count, before):
    rnd = random.Random(count)
    values = np.array(rnd.sample(range(1 << N), count), dtype=np.uint64)
    point = to_mont_array([rnd.randrange(o.R_MOD) for _ in range(N)])
    weights = to_mont_array([rnd.randrange(o.R_MOD)])
    counts = np.array([count], dtype=np.uint64)
    keep, ptr = pinned(values, before)
    for call in (lambda p: opened(ctx, srs, p, count, point), lambda p: committed(ctx, srs, p, count),
                 lambda p: checked(ctx, 1, p, counts, weights, point)):
        rc, want = call(values.ctypes.data)
        check(rc, "pageable")
        rc, got = call(ptr)
        check(rc, "pinned")
        assert np.array_equal(got, want)
    del keep


@pytest.mark.parametrize("off", [1, 4, 7])
def test_lists_that_are_not_aligned_to_their_words(ctx, srs, off):
    """Copied whatever their address, as from pageable memory: no kernel reads them in place."""
    rnd = random.Random(off)
    values = np.array(rnd.sample(range(1 << N), 100), dtype=np.uint64)
    point, weights, counts = to_mont_array([rnd.randrange(o.R_MOD) for _ in range(N)]), to_mont_array([5]), np.array([100], dtype=np.uint64)
    keep = torch.zeros(off + values.nbytes, dtype=torch.uint8, pin_memory=True)
    keep[off:] = torch.from_numpy(values.view(np.uint8))
    ptr = keep.data_ptr() + off
    for call in (lambda p: opened(ctx, srs, p, 100, point), lambda p: committed(ctx, srs, p, 100),
                 lambda p: checked(ctx, 1, p, counts, weights, point)):
        rc, want = call(values.ctypes.data)
        check(rc, "aligned")
        rc, got = call(ptr)
        check(rc, "not aligned")
        assert np.array_equal(got, want)


def test_refused_indices(ctx, srs):
    point, weights = to_mont_array([3] * N), to_mont_array([5])
    values = np.array([1, 2, 1 << N], dtype=np.uint64)
    keep, ptr = pinned(values)
    assert opened(ctx, srs, ptr, 3, point)[0] != 0
    assert committed(ctx, srs, ptr, 3)[0] != 0
    assert checked(ctx, 1, ptr, np.array([3], dtype=np.uint64), weights, point)[0] != 0
    keep[2] = 2  # twice in one term
    assert checked(ctx, 1, ptr, np.array([3], dtype=np.uint64), weights, point)[0] != 0
    assert opened(ctx, srs, ptr, 3, point)[0] == 0
