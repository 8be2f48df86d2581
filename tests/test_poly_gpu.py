"""eq tables and fix_variables_from_right on the GPU against the oracle, with the closed forms of
tests/test_lagrange_basis.rs and tests/test_fix_variables.rs:278-307."""
import ctypes
import random

import numpy as np
import pytest

import pyoracle as o
from zkes_b200 import DenseMLPoly, evaluate_lagrange_basis, fix_variables_from_right
from zkes_b200._lib import ZK_MEM_HOST, check, lib
from zkes_b200.field import from_mont_array, to_mont_array

pytestmark = pytest.mark.gpu
M = o.R_MOD


def test_lagrange_basis_closed_forms(ctx):
    assert evaluate_lagrange_basis(ctx, []) == [1]  # test_lagrange_basis.rs:121-127
    r0, r1 = 3, 10
    assert evaluate_lagrange_basis(ctx, [r0]) == [(1 - r0) % M, r0]
    assert evaluate_lagrange_basis(ctx, [r0, r1]) == [(1 - r0) * (1 - r1) % M, r0 * (1 - r1) % M, (1 - r0) * r1 % M, r0 * r1 % M]
    assert evaluate_lagrange_basis(ctx, [1, 0, 1]) == [1 if i == 5 else 0 for i in range(8)]  # vertices :97-118


@pytest.mark.parametrize("k", [1, 4, 9, 10, 11, 14])
def test_lagrange_basis_random(ctx, k):
    rnd = random.Random(k)
    pt = [rnd.randrange(M) for _ in range(k)]
    got = evaluate_lagrange_basis(ctx, pt)
    assert got == o.evaluate_lagrange_basis(pt)
    assert sum(got) % M == 1  # partition of unity :66-73


def test_from_right_closed_form(ctx):
    f = DenseMLPoly.from_evaluations([1, 2, 3, 4])
    assert fix_variables_from_right(ctx, f, [0]).evaluations == [1, 2]
    assert fix_variables_from_right(ctx, f, [1]).evaluations == [3, 4]
    assert fix_variables_from_right(ctx, f, [7]).evaluations == [15, 16]
    assert fix_variables_from_right(ctx, f, []).evaluations == [1, 2, 3, 4]


@pytest.mark.parametrize("n,k", [(1, 1), (4, 2), (6, 6), (10, 3), (12, 6), (13, 12), (14, 2), (15, 8)])
def test_from_right_random(ctx, n, k):
    rnd = random.Random(100 * n + k)
    f = [rnd.randrange(M) for _ in range(1 << n)]
    pt = [rnd.randrange(M) for _ in range(k)]
    got = fix_variables_from_right(ctx, DenseMLPoly.from_evaluations(f), pt).evaluations
    assert got == o.fix_variables_from_right(f, pt)
    # the same polynomial: binding the low variables afterwards gives the full evaluation
    if n <= 12:
        lowpt = [rnd.randrange(M) for _ in range(n - k)]
        assert o.evaluate_multilinear_extension(got, lowpt) == o.evaluate_multilinear_extension(f, lowpt + pt)


@pytest.mark.parametrize("lo,hi", [(0, 4), (0, 8), (0, 9), (0, 11), (1, 9), (3, 8), (4, 9), (5, 8), (5, 9), (2, 10), (6, 4)])
@pytest.mark.parametrize("kind", ["largest", "random"])
def test_weighted_fold_edges(ctx, lo, hi, kind):
    """2^hi rows of 2^lo columns around the sizes where the byte products begin (512 rows) and a block's columns (16) end, its weights being
    held for 256 rows at a time, with the largest bytes that an element can have (p - 1 in memory) and random ones."""
    rnd = random.Random(100 * lo + hi)
    largest = (M - 1) * pow(1 << 256, -1, M) % M
    f = [largest if kind == "largest" else rnd.randrange(M) for _ in range(1 << (lo + hi))]
    w = [largest if kind == "largest" else rnd.choice([0, rnd.randrange(M)]) for _ in range(1 << hi)]
    fm, wm, out = to_mont_array(f), to_mont_array(w), np.zeros((1 << lo, 4), dtype=np.uint64)
    vp = ctypes.c_void_p
    check(lib.zk_weighted_fold_from_right(ctx.handle, lo + hi, vp(fm.ctypes.data), ZK_MEM_HOST, hi, vp(wm.ctypes.data), ZK_MEM_HOST,
                                          vp(out.ctypes.data), ZK_MEM_HOST), "zk_weighted_fold_from_right")
    assert list(from_mont_array(out)) == [sum(w[h] * f[(h << lo) + c] for h in range(1 << hi)) % M for c in range(1 << lo)]


@pytest.mark.parametrize("lo,hi", [(8, 13), (11, 9), (13, 9), (14, 9), (3, 16), (0, 19)])
def test_weighted_fold_pieces(ctx, lo, hi):
    """Shapes whose blocks take several steps of 32 rows, so that the sums go on from step to step, the slots of the stream and the weights'
    256 rows are used again, and pieces end inside a column group, cross into the next, or are a column's only ones.  The table
    has sixteen different elements, the largest (p - 1 in memory) and zero among them: out[c] = sum_e e sum_{h: f[h, c] = e} w[h], the
    inner sums exact in double precision by 16-bit limbs."""
    rnd = np.random.default_rng(100 * lo + hi)
    largest = (M - 1) * pow(1 << 256, -1, M) % M
    pool = [largest, 0] + [int.from_bytes(rnd.bytes(40), "little") % M for _ in range(14)]
    w = [largest if h % 3 == 0 else int.from_bytes(rnd.bytes(40), "little") % M for h in range(1 << hi)]
    which = rnd.integers(0, 16, size=(1 << hi, 1 << lo), dtype=np.uint8)
    which[:, 0] = 0  # a column of nothing but the largest
    f, wm, out = to_mont_array(pool)[which.reshape(-1)], to_mont_array(w), np.zeros((1 << lo, 4), dtype=np.uint64)
    vp = ctypes.c_void_p
    check(lib.zk_weighted_fold_from_right(ctx.handle, lo + hi, vp(f.ctypes.data), ZK_MEM_HOST, hi, vp(wm.ctypes.data), ZK_MEM_HOST,
                                          vp(out.ctypes.data), ZK_MEM_HOST), "zk_weighted_fold_from_right")
    limbs = np.frombuffer(b"".join(x.to_bytes(32, "little") for x in w), dtype="<u2").reshape(1 << hi, 16).astype(np.float64)
    want = [0] * (1 << lo)
    for e in range(16):
        if pool[e]:
            sums = (which == e).astype(np.float64).T @ limbs  # below 2^19 * 2^16
            want = [a + pool[e] * sum(int(x) << (16 * k) for k, x in enumerate(row)) for a, row in zip(want, sums.tolist())]
    assert list(from_mont_array(out)) == [x % M for x in want]


@pytest.mark.parametrize("n", [0, 1, 3, 8, 11, 15])
def test_evaluate_at_point(ctx, n):
    """DenseMLPoly::evaluate_at_point (poly.rs:788-791); test_kzh2.rs:149-175 relies on it."""
    rnd = random.Random(900 + n)
    f = [rnd.randrange(M) for _ in range(1 << n)]
    pt = [rnd.randrange(M) for _ in range(n)]
    assert DenseMLPoly.from_evaluations(f).evaluate_at_point(ctx, pt) == o.evaluate_multilinear_extension(f, pt)
    if n == 3:  # a vertex picks one table entry
        assert DenseMLPoly.from_evaluations(f).evaluate_at_point(ctx, [1, 0, 1]) == f[5]
