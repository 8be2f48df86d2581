"""The routes of the MSM pipeline at the sizes where they change: rows of small scalars by subset-sum tables, long buckets, and
the reduction of a window's buckets over several blocks.  The bases are known multiples of g, so that the expected point of any
row is one multiple of g."""
import ctypes
import random

import numpy as np
import pytest

import pyoracle as o
from zkes_b200 import curve
from zkes_b200._lib import ZK_MEM_DEVICE, ZK_MEM_HOST, check, lib
from zkes_b200.field import to_mont_array

pytestmark = pytest.mark.gpu
vp = ctypes.c_void_p


@pytest.fixture(scope="module")
def multiples():
    """k_i and k_i g; repeats, opposite points and infinity among them."""
    rnd = random.Random(9)
    ks = [rnd.randrange(1, 1 << 64) for _ in range(61)] + [0, 1, 1, 2, o.R_MOD - 1, o.R_MOD - 2, 3]
    return ks, [o.g1_mul(o.G1_GEN, k) if k else None for k in ks]


def of_g(k):
    k %= o.R_MOD
    return o.g1_mul(o.G1_GEN, k) if k else None


def values(rnd, lo, hi):
    return rnd.choice([lo, hi, 0, rnd.randint(lo, hi), rnd.randint(lo, hi)])


@pytest.mark.parametrize("rows,n,lo,hi", [(2, 1, -128, 127), (300, 1, -1, 0), (64, 2, 0, 1), (40, 13, -128, 127), (700, 12, -128, 128),
                                          (333, 25, -1, 1), (2050, 31, -32768, 32767), (97, 68, -(1 << 29), (1 << 29) - 1)])
def test_rows_of_small_scalars(ctx, multiples, rows, n, lo, hi):
    rnd = random.Random(rows * n)
    ks, pts = multiples
    mat = [[values(rnd, lo, hi) for _ in range(n)] for _ in range(rows)]
    mat[0] = [lo] * n
    mat[1] = [hi] * n
    got = curve.msm_batched(ctx, curve.affine_to_array(pts[-n:]), [[o.fr_from_int(v) for v in r] for r in mat])
    for r in list(range(0, rows, max(1, rows // 40))) + [1, rows - 1]:
        assert got[r] == of_g(sum(v * k for v, k in zip(mat[r], ks[-n:]))), r


def _device_msm(ctx, bases, scalars):
    import torch

    out = np.zeros((1, 12), dtype=np.uint64)
    torch.cuda.synchronize()
    check(lib.zk_msm_g1(ctx.handle, vp(bases.data_ptr()), ZK_MEM_DEVICE, vp(scalars.data_ptr()), ZK_MEM_DEVICE, bases.shape[0],
                        vp(out.ctypes.data), ZK_MEM_HOST), "zk_msm_g1")
    return curve.jacobian_to_affine_py(out)[0]


def _repeated(pool, picks):
    import torch

    return torch.from_numpy(pool.view(np.int64)).cuda()[torch.from_numpy(picks).cuda()].contiguous()


def test_rows_within_the_scratch_of_buckets(multiples):
    """256 rows of 2^18 four-bit values: the tables (0.65 GB at once) are made in slabs that take no more than the buckets' 0.5 GB."""
    import torch

    from zkes_b200 import Context

    ks, pts = multiples
    rows, n = 256, 1 << 18
    rng = np.random.default_rng(4)
    pick = rng.integers(0, len(ks), size=n)
    bases = _repeated(curve.affine_to_array(pts), pick)
    vals = torch.randint(-8, 8, (rows, n), dtype=torch.int8, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4))
    f = torch.from_numpy(to_mont_array([o.fr_from_int(v) for v in range(-8, 8)]).view(np.int64)).cuda()[(vals.reshape(-1).int() + 8)]
    out = np.zeros((rows, 12), dtype=np.uint64)
    torch.cuda.synchronize()
    c = Context(0)
    before = torch.cuda.mem_get_info()[0]
    check(lib.zk_msm_g1_batched(c.handle, vp(bases.data_ptr()), ZK_MEM_DEVICE, n, vp(f.data_ptr()), ZK_MEM_DEVICE, rows,
                                vp(out.ctypes.data), ZK_MEM_HOST), "zk_msm_g1_batched")
    taken = before - torch.cuda.mem_get_info()[0]
    c.close()
    buckets = 4 * rows * n + (rows * 8 + 2 * 148 * 4 * 128 * 12) * 128  # entries, bucket sums, pieces of chunks
    compact = 4 * rows * n
    assert taken <= buckets + compact + (64 << 20), taken  # with allocation granularity and the code loaded by the call
    for r in (0, 1, 131, rows - 1):
        per_base = np.bincount(pick, weights=vals[r].cpu().numpy(), minlength=len(ks))
        assert curve.jacobian_to_affine_py(out[r:r + 1])[0] == of_g(sum(int(v) * k for v, k in zip(per_base, ks))), r


@pytest.mark.parametrize("n", [1 << 21, 10_000_003])
@pytest.mark.parametrize("scalars", [[1, -1], [-128, 127, 5, 0, 1]])
def test_long_buckets_of_repeated_points(ctx, multiples, n, scalars):
    """Few buckets over millions of entries, and so few distinct points that equal, opposite and infinite operands meet at
    every step of the running sums."""
    ks, pts = multiples
    rng = np.random.default_rng(n)
    pick = rng.integers(0, len(ks), size=n)
    sel = rng.integers(0, len(scalars), size=n)
    counts = np.zeros((len(ks), len(scalars)), dtype=np.int64)
    np.add.at(counts, (pick, sel), 1)
    want = sum(int(counts[i, j]) * ks[i] * scalars[j] for i in range(len(ks)) for j in range(len(scalars)))
    bases = _repeated(curve.affine_to_array(pts), pick)
    sc = _repeated(to_mont_array([o.fr_from_int(v) for v in scalars]), sel)
    assert _device_msm(ctx, bases, sc) == of_g(want)


@pytest.mark.parametrize("n", [1 << 15, 100_003, (1 << 20) + 1])
def test_full_width_windows(ctx, multiples, n):
    """Full-width scalars: several blocks per window in the bucket reduction, a degenerate top window, and the
    combination on the host."""
    ks, pts = multiples
    rng = np.random.default_rng(n)
    rnd = random.Random(n)
    scalars = [o.R_MOD - 1, (o.R_MOD - 1) // 2, (o.R_MOD + 1) // 2, 1, 0] + [rnd.randrange(o.R_MOD) for _ in range(2043)]
    pick = rng.integers(0, len(ks), size=n)
    sel = rng.integers(0, len(scalars), size=n)
    per_scalar = [0] * len(scalars)
    for i, j in zip(pick.tolist(), sel.tolist()):
        per_scalar[j] += ks[i]
    want = sum(t * s for t, s in zip(per_scalar, scalars))
    assert _device_msm(ctx, _repeated(curve.affine_to_array(pts), pick), _repeated(to_mont_array(scalars), sel)) == of_g(want)


@pytest.mark.parametrize("rows,n", [(2, 5000), (40, 700), (700, 300)])
def test_full_width_rows(ctx, multiples, rows, n):
    """The combination of the windows on the host, by a warp per row and by a thread per row."""
    ks, pts = multiples
    rng = np.random.default_rng(rows)
    rnd = random.Random(rows)
    scalars = [o.R_MOD - 1, 0, 1] + [rnd.randrange(o.R_MOD) for _ in range(509)]
    pick = rng.integers(0, len(ks), size=n)
    sel = rng.integers(0, len(scalars), size=(rows, n))
    bases = np.ascontiguousarray(curve.affine_to_array(pts)[pick])
    sc = np.ascontiguousarray(to_mont_array(scalars)[sel.reshape(-1)])
    out = np.zeros((rows, 12), dtype=np.uint64)
    check(lib.zk_msm_g1_batched(ctx.handle, vp(bases.ctypes.data), ZK_MEM_HOST, n, vp(sc.ctypes.data), ZK_MEM_HOST, rows,
                                vp(out.ctypes.data), ZK_MEM_HOST), "zk_msm_g1_batched")
    for r in sorted({0, 1, rows // 2, rows - 1}):
        want = sum(ks[p] * scalars[s] for p, s in zip(pick.tolist(), sel[r].tolist()))
        assert curve.jacobian_to_affine_py(out[r:r + 1])[0] == of_g(want), r


@pytest.mark.parametrize("rows,n", [(31, 64), (32, 1), (32, 2), (32, 33), (33, 4097), (64, 128), (1500, 9)])
def test_full_width_rows_that_share_buckets(ctx, multiples, rows, n):
    """From 32 rows on the windows of a row share its buckets, over multiples of the bases; below they do not."""
    test_full_width_rows(ctx, multiples, rows, n)


@pytest.mark.parametrize("n", [1, 2, 5, 33, 1000])
@pytest.mark.parametrize("rows", [1, 33])
def test_scalars_at_the_ends_of_the_split(ctx, multiples, n, rows):
    """Scalars whose halves are zero, one, or the largest that occur, beside ones of 160 and 161 bits, where the split begins."""
    ks, pts = multiples
    rnd = random.Random(n * rows)
    lam = 0xb3c4d79d41a917585bfc41088d8daaa78b17ea66b99c90dd
    assert (lam * lam + lam + 1) % o.R_MOD == 0
    half = (o.R_MOD - 1) // 2
    pool = [0, 1, o.R_MOD - 1, lam, o.R_MOD - lam, lam + 1, lam * lam % o.R_MOD, half, half + 1, (1 << 126) - 1, ((1 << 125) * lam) % o.R_MOD,
            (1 << 160) - 1, 1 << 160, (1 << 161) - 1] + [(rnd.randrange(1 << 126) + rnd.randrange(1 << 125) * lam) % o.R_MOD for _ in range(20)]
    mat = [[rnd.choice(pool) for _ in range(n)] for _ in range(rows)]
    mat[0][0] = half
    got = curve.msm_batched(ctx, curve.affine_to_array(pts[-n:] if n <= len(pts) else [pts[i % len(pts)] for i in range(n)]), mat)
    use = ks[-n:] if n <= len(ks) else [ks[i % len(ks)] for i in range(n)]
    for r in sorted({0, rows // 2, rows - 1}):
        assert got[r] == of_g(sum(v * k for v, k in zip(mat[r], use))), r


@pytest.mark.parametrize("rows,n", [(2, 30), (3, 100), (300, 130), (650, 255)])
def test_full_width_rows_of_few_buckets(ctx, multiples, rows, n):
    """Fewer than 256 bases a row: windows of three bits, whose four buckets are one thread's."""
    test_full_width_rows(ctx, multiples, rows, n)


@pytest.mark.parametrize("n", [70_001, 1 << 18, 3_000_000])
@pytest.mark.parametrize("top", [100, 3000])
def test_one_hot_bucket_among_many(ctx, multiples, n, top):
    """Digits of which nearly all are the same: the pieces of that bucket are shared by several blocks, the others' are not."""
    ks, pts = multiples
    rng = np.random.default_rng(n + top)
    pick = rng.integers(0, len(ks), size=n)
    vals = np.where(rng.random(n) < 0.99, top - 1, rng.integers(-top, top + 1, size=n))
    per_base = np.bincount(pick, weights=vals, minlength=len(ks))
    sc = _repeated(to_mont_array([o.fr_from_int(v) for v in range(-top, top + 1)]), vals + top)
    got = _device_msm(ctx, _repeated(curve.affine_to_array(pts), pick), sc)
    assert got == of_g(sum(int(v) * k for v, k in zip(per_base, ks)))


@pytest.mark.parametrize("n,hot,share", [(3_000_000, 5000, 1.0), (3_000_000, 1500, 0.3), (3_000_000, 1200, 1.0), (200_000, 600, 0.9), (1_500_000, 40, 0.5)])
def test_buckets_of_some_pieces(ctx, multiples, n, hot, share):
    """Thousands of buckets of nine to twenty-four pieces (a thread each), hundreds of them (a warp each), longer ones (a block
    each), and all kinds at once."""
    ks, pts = multiples
    rng = np.random.default_rng(n + hot)
    pick = rng.integers(0, len(ks), size=n)
    values = rng.choice(np.arange(1, 32769), size=hot, replace=False)
    vals = np.where(rng.random(n) < share, values[rng.integers(0, hot, size=n)], rng.integers(-32768, 32769, size=n))
    vals[0] = 32768
    per_base = np.bincount(pick, weights=vals, minlength=len(ks))
    sc = _repeated(to_mont_array([o.fr_from_int(v) for v in range(-32768, 32769)]), vals + 32768)
    got = _device_msm(ctx, _repeated(curve.affine_to_array(pts), pick), sc)
    assert got == of_g(sum(int(v) * k for v, k in zip(per_base, ks)))


@pytest.mark.parametrize("rows,n", [(1024, 1024), (1024, 1003), (4096, 1000)])
def test_rows_in_several_chains(ctx, multiples, rows, n):
    """Hundreds of groups in a few chains of several groups each, the last one shorter."""
    import torch

    ks, pts = multiples
    rng = np.random.default_rng(rows + n)
    pick = rng.integers(0, len(ks), size=n)
    vals = rng.integers(-128, 128, size=(rows, n))
    vals[1], vals[2] = -128, 127
    f = _repeated(to_mont_array([o.fr_from_int(v) for v in range(-128, 128)]), vals.reshape(-1) + 128)
    bases = _repeated(curve.affine_to_array(pts), pick)
    out = np.zeros((rows, 12), dtype=np.uint64)
    torch.cuda.synchronize()
    check(lib.zk_msm_g1_batched(ctx.handle, vp(bases.data_ptr()), ZK_MEM_DEVICE, n, vp(f.data_ptr()), ZK_MEM_DEVICE, rows,
                                vp(out.ctypes.data), ZK_MEM_HOST), "zk_msm_g1_batched")
    for r in sorted({0, 1, 2, rows // 3, rows - 2, rows - 1}):
        per_base = np.bincount(pick, weights=vals[r], minlength=len(ks))
        assert curve.jacobian_to_affine_py(out[r:r + 1])[0] == of_g(sum(int(v) * k for v, k in zip(per_base, ks))), r


def test_full_width_rows_with_32_lanes(ctx, multiples):
    """1720 items of 32 buckets: 32 lanes an item."""
    test_full_width_rows(ctx, multiples, 40, 2000)


def test_work_of_rows_by_subset_sums(ctx, multiples):
    """The reported entries are table look-ups, one per row, bit plane and group; the sums that make the tables are not among them."""
    _, pts = multiples
    rows, n = 700, 12
    rnd = random.Random(3)
    mat = [[o.fr_from_int(rnd.randint(-128, 127)) for _ in range(n)] for _ in range(rows)]
    mat[0][0] = o.fr_from_int(-128)
    calls, entries, buckets = ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_uint64()
    args = (ctypes.byref(calls), ctypes.byref(entries), ctypes.byref(buckets), 1)
    check(lib.zk_msm_work(ctx.handle, *args), "zk_msm_work")
    curve.msm_batched(ctx, curve.affine_to_array(pts[-n:]), mat)
    check(lib.zk_msm_work(ctx.handle, *args), "zk_msm_work")
    planes = 8
    assert calls.value == 1 and buckets.value == 0
    assert entries.value % (rows * planes) == 0 and 1 <= entries.value // (rows * planes) <= n // 2
