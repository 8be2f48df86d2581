"""The rules by which the MSM pipeline picks its route and cuts its work (zkes_b200/csrc/msm_plan.hpp), on the CPU."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SM = 148
FREE_SCRATCH = 256 << 20  # what the tables may take whatever the buckets would
# largest magnitude, largest of v and -v - 1
KINDS = {"bit": (1, 1), "minus": (1, 0), "sign": (1, 1), "int8": (128, 127), "int16": (32768, 32767), "int30": ((1 << 30) - 1, (1 << 30) - 1)}


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("plan") / "libmsmplan.so")
    subprocess.run(["g++", "-O2", "-shared", "-fPIC", "-std=c++17", os.path.join(HERE, "hostmath", "msm_plan_host.cpp"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    u64, u32, i = ctypes.c_uint64, ctypes.c_uint32, ctypes.c_int
    lib.zkp_buckets.argtypes = [u64, u32, i, i, i, ctypes.c_void_p]
    lib.zkp_windows.argtypes = [u64, u32, u32, ctypes.c_void_p]
    lib.zkp_merged.argtypes = [u64, ctypes.c_void_p]
    lib.zkp_merged_rows.argtypes = [u64, u32]
    lib.zkp_rows.argtypes = [u64, u32, u32, u64, i, i, i, u64, ctypes.c_void_p]

    lib.zkp_reduce_lanes.argtypes = [u32, u32, i]
    lib.zkp_reduce_lanes.restype = u32
    lib.zkp_fixup_groups.argtypes = [u32, u32, u64, u32]
    lib.zkp_chunk_entries.argtypes = [u32, i]
    lib.zkp_combine_by.argtypes = [u32, i, i, i]

    def call(name, n_out, *args):
        if n_out == 0:
            return getattr(lib, name)(*args)
        out = (u64 * n_out)()
        getattr(lib, name)(*args, out)
        return list(out)

    return call


def shapes(plan, rows, n, kind):
    mag, span = KINDS[kind]
    w, k = plan("zkp_windows", 2, n, rows, mag)
    buckets, scratch = plan("zkp_buckets", 2, n * rows, rows, w, k, SM)
    return span, w, k, buckets, scratch


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rows,n", [(1024, 1 << 20), (320, 1 << 18), (4096, 1 << 17), (1 << 14, 1 << 14), (1 << 22, 300), (2, 1 << 28), (1 << 24, 7)])
def test_subset_tables_take_no_more_scratch_than_buckets(plan, rows, n, kind):
    """A call whose buckets fit the memory is not refused for the tables' sake."""
    span, w, k, buckets, scratch = shapes(plan, rows, n, kind)
    if buckets >= 1 << 31:
        scratch = (1 << 64) - 1
    group, _, _, _, parts, need, pieces, slab = plan("zkp_rows", 8, n, rows, span, n * rows, w, k, SM, scratch)
    assert need <= max(scratch, FREE_SCRATCH) or not group
    assert pieces < 1 << 31
    assert 1 <= slab <= parts or not group


def test_tables_by_slabs(plan):
    """2^20 columns in 1024 rows of int8 values: 9 GB of tables at once, made in slabs that fit the buckets' 4.6 GB."""
    span, w, k, _, scratch = shapes(plan, 1024, 1 << 20, "int8")
    at_once = plan("zkp_rows", 8, 1 << 20, 1024, span, 1 << 30, w, k, SM, 1 << 60)
    held = plan("zkp_rows", 8, 1 << 20, 1024, span, 1 << 30, w, k, SM, scratch)
    assert at_once[7] == at_once[4] and at_once[5] > scratch
    assert held[:5] == at_once[:5] and 1 <= held[7] < held[4] and held[5] <= scratch


def test_chains_cover_every_group(plan):
    for rows, n, kind in [(4096, 4096, "int8"), (1024, 1024, "int8"), (3000, 777, "int16"), (1000, 5000, "bit"), (50, 6, "int8")]:
        span, w, k, _, _ = shapes(plan, rows, n, kind)
        group, planes, groups, seg, parts = plan("zkp_rows", 8, n, rows, span, n * rows, w, k, SM, 1 << 60)[:5]
        assert group
        assert (groups - 1) * group < n <= groups * group
        assert (parts - 1) * seg < groups <= parts * seg


@pytest.mark.parametrize("n", [1, 2, 3, 40, 2047, 2048, 1 << 14, (1 << 20) - 1, 1 << 20])
def test_shared_buckets_hold_every_digit_and_entry(plan, n):
    """Signed digits of 126 bits and a carry in the windows; a multiple's index beside the two flag bits of an entry."""
    w, windows, most, split_most = plan("zkp_merged", 4, n)
    assert w * windows >= 127 > w * (windows - 1)
    assert n <= most and windows * n < 1 << 30 and split_most < 1 << 30
    assert plan("zkp_buckets", 2, 2 * n * windows * 32, 32, w, 1, SM)[0] == 32 << (w - 1)


@pytest.mark.parametrize("n", [1, 1 << 14, 1 << 17, (1 << 18) - 1, 1 << 18, 1 << 19, 1 << 20, (1 << 20) + 1, 1 << 24, 1 << 40])
@pytest.mark.parametrize("rows", [1, 31, 32, 1 << 12])
def test_shared_buckets_have_bounded_tables(plan, n, rows):
    """The multiples of a call's bases (an affine and an XYZZ point and a coordinate each) stay below half a gigabyte, whatever the rows."""
    taken = bool(plan("zkp_merged_rows", 0, n, rows))
    assert taken == (rows >= 32 and n <= 1 << 18)
    if taken:
        _, windows, _, _ = plan("zkp_merged", 4, n)
        assert n * windows * (64 + 128 + 32) <= 512 << 20


# rows, columns, kind, share of zeros, subset sums: measured, both ways at least a tenth apart
ROUTES = [
    (4096, 4096, "int8", 0, True),     # 2.63 ms by sums, 4.06 by buckets
    (4096, 4096, "int8", .9, False),   # 2.61, 1.79
    (4096, 4096, "int16", .9, False),  # 4.27, 3.09
    (4096, 4096, "bit", 0, True),      # 1.11, 2.75
    (1024, 512, "int8", 0, True),      # 0.38, 0.59
    (4096, 8, "int16", 0, True),       # 0.33, 0.41
    (4096, 8, "int16", .995, True),    # 0.32, 2.26: hundreds of empty buckets between two entries
    (16, 16384, "bit", 0, False),      # 0.62, 0.29
    (16, 16384, "sign", .75, False),
    (4, 65536, "minus", .9, False),    # 2.71, 0.26
    (2, 65536, "int8", 0, False),
    (16, 16384, "int8", 0, False),     # 0.67, 0.43
]


@pytest.mark.parametrize("rows,n,kind,zeros,sums", ROUTES)
def test_rows_take_the_faster_route(plan, rows, n, kind, zeros, sums):
    span, w, k, _, scratch = shapes(plan, rows, n, kind)
    nonzero = int(rows * n * (1 - zeros) * {"bit": .5, "minus": .5, "sign": 2 / 3}.get(kind, 1))
    assert (plan("zkp_rows", 8, n, rows, span, nonzero, w, k, SM, scratch)[0] > 0) == sums


@pytest.mark.parametrize("half", [2, 4])
@pytest.mark.parametrize("items", [1, 85, 340, 1024, 174080])
def test_few_buckets_an_item_get_a_thread(plan, items, half):
    """A block per item would keep one thread of 128 busy; few items, of which most buckets are empty, get blocks all the same."""
    assert plan("zkp_reduce_lanes", 0, items, half, SM) == (1 if items >= 512 else 0)


@pytest.mark.parametrize("half", [8, 16, 128, 512, 32768])
@pytest.mark.parametrize("items", [1, 1023, 1024, 2000, 30000])
def test_lanes_divide_the_buckets(plan, items, half):
    lanes = plan("zkp_reduce_lanes", 0, items, half, SM)
    assert lanes in ((0,) if items < 1024 else (8, 16, 32)) and lanes <= half


def test_who_combines_the_windows(plan):
    host, warps, threads = 0, 1, 2
    by = lambda rows, w, k: plan("zkp_combine_by", 0, rows, w, k, SM)  # noqa: E731
    for rows in (1, 4, 5, 592, 593):
        assert by(rows, 9, 1) == threads  # one window: nothing to combine
    assert by(1, 14, 19) == by(4, 8, 4) == host
    assert by(5, 8, 4) == by(1, 3, 2) == by(592, 3, 85) == warps
    assert by(593, 3, 85) == threads


@pytest.mark.parametrize("buckets", [1, 128, 4096, 8192])
@pytest.mark.parametrize("n", [1, 4095, 1 << 16, 1 << 18, 3_000_000, 1 << 24])
def test_equal_digits_are_no_long_chain(plan, buckets, n):
    """One window of n digits that all fall into one bucket: a thread adds 64 pieces at most, as with 2^18 digits in chunks of 32
    and a block of 128 threads, or the bucket has all the blocks that there are."""
    seg = plan("zkp_chunk_entries", 0, n, SM)
    chunks = (n + seg - 1) // seg
    groups = plan("zkp_fixup_groups", 0, buckets, chunks, n, seg)
    most = min(128, 16384 // buckets)
    assert 1 <= groups <= most
    assert (chunks + 1) / (128 * groups) <= 64 or groups == most
