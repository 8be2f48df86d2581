"""GPU parity of the sparse x dense product sumcheck against the oracle's dense prover on
[a.to_dense(), b] (the definition of this prover's output)."""
import random

import pytest

import pyoracle as o
from zkes_b200 import DenseMLPoly, SparseDenseSumcheckProver, Transcript
from zkes_b200._lib import ZkError
from zkes_b200.field import to_mont_array

pytestmark = pytest.mark.gpu


def run_case(ctx, n, nnz, seed, small_values=True):
    rnd = random.Random(seed)
    idx = sorted(rnd.sample(range(1 << n), nnz))
    if small_values:
        vals = [o.fr_from_int(rnd.randrange(-128, 128)) for _ in idx]  # int8 lifted, zeros allowed
    else:
        vals = [rnd.randrange(o.R_MOD) for _ in idx]
    dense = [rnd.randrange(o.R_MOD) for _ in range(1 << n)]
    t = Transcript(b"sd_sumcheck")
    prover = SparseDenseSumcheckProver(n, t)
    proof = prover.prove(ctx, idx, vals, DenseMLPoly.from_evaluations(dense), t)
    ot = o.Transcript(b"sd_sumcheck")
    oprover, oproof = o.sparse_dense_prove(n, idx, vals, dense, ot)
    assert proof.round_messages == oproof.round_messages
    assert prover.challenges == oprover.challenges
    assert proof.final_eval == oproof.final_eval
    assert [a[0] for a in prover.a_arrays] == [a[0] for a in oprover.a_arrays]
    assert t.challenge_scalar(b"after") == ot.challenge_scalar(b"after")
    # the restated verifier accepts with the true claimed sum
    claimed = sum(v * dense[i] for i, v in zip(idx, vals)) % o.R_MOD
    vt = o.Transcript(b"sd_sumcheck")
    ver = o.SumcheckVerifier(n, 2, vt)
    res, _ = ver.verify(vt, proof.round_messages, claimed)
    assert res == proof.final_eval


@pytest.mark.parametrize("n,nnz", [(0, 0), (0, 1), (1, 0), (1, 1), (1, 2), (3, 1), (4, 16), (6, 5), (8, 3), (10, 64),
                                   (12, 40), (12, 4096), (13, 700), (14, 1000), (16, 300)])
def test_sparse_dense_matches_dense_prover(ctx, n, nnz):
    run_case(ctx, n, nnz, seed=100 * n + nnz)


def test_full_width_values(ctx):
    run_case(ctx, 11, 200, seed=7, small_values=False)


def test_adjacent_runs(ctx):
    """Entries in consecutive runs exercise the even/odd pairing and the compaction."""
    n = 10
    idx = list(range(5, 40)) + list(range(511, 530)) + [1022, 1023]
    rnd = random.Random(3)
    vals = [rnd.randrange(1, o.R_MOD) for _ in idx]
    dense = [rnd.randrange(o.R_MOD) for _ in range(1 << n)]
    t = Transcript(b"sd")
    p = SparseDenseSumcheckProver(n, t)
    proof = p.prove(ctx, idx, vals, DenseMLPoly.from_evaluations(dense), t)
    ot = o.Transcript(b"sd")
    _, oproof = o.sparse_dense_prove(n, idx, vals, dense, ot)
    assert proof.round_messages == oproof.round_messages and proof.final_eval == oproof.final_eval


@pytest.mark.parametrize("n", [3, 4, 6, 7, 9])
@pytest.mark.parametrize("kind", ["largest", "mixed"])
def test_double_folds_of_extreme_tables(ctx, n, kind):
    """One entry keeps the prover in entry form, so the table is folded two variables at a time down to two elements: tiles of 32
    outputs whole and in part, with elements whose bytes make the largest sums (p - 1 in memory) beside zeros."""
    rnd = random.Random(n)
    largest = (o.R_MOD - 1) * pow(1 << 256, -1, o.R_MOD) % o.R_MOD  # its Montgomery form is p - 1
    dense = [largest if kind == "largest" else rnd.choice([0, largest, rnd.randrange(o.R_MOD)]) for _ in range(1 << n)]
    idx, vals = [rnd.randrange(1 << n)], [rnd.randrange(1, o.R_MOD)]
    t, ot = Transcript(b"sd"), o.Transcript(b"sd")
    proof = SparseDenseSumcheckProver(n, t).prove(ctx, idx, vals, DenseMLPoly.from_evaluations(dense), t)
    _, oproof = o.sparse_dense_prove(n, idx, vals, dense, ot)
    assert proof.round_messages == oproof.round_messages and proof.final_eval == oproof.final_eval


def test_rejects_unsorted_or_out_of_range(ctx):
    dense = DenseMLPoly.from_evaluations([1] * 16)
    for bad in ([3, 2], [1, 1], [5, 16]):
        t = Transcript(b"sd")
        p = SparseDenseSumcheckProver(4, t)
        with pytest.raises(ZkError):
            p.prove(ctx, bad, [1, 1], dense, t)


@pytest.mark.parametrize("vals_at", ["aligned", "eight bytes off", "pinned"])
@pytest.mark.parametrize("n,nnz", [(5, 1), (12, 40), (14, 1000)])
def test_device_inputs(ctx, n, nnz, vals_at):
    """Values in device memory are taken over by the launch that narrows the indices; unaligned or in other memory, by a copy."""
    import torch
    rnd = random.Random(n + nnz)
    idx = sorted(rnd.sample(range(1 << n), nnz))
    vals = [rnd.randrange(o.R_MOD) for _ in idx]
    dense = [rnd.randrange(o.R_MOD) for _ in range(1 << n)]

    def words(a):
        return torch.from_numpy(a.view("int64").reshape(-1).copy())

    d = words(DenseMLPoly.from_evaluations(dense).mont).cuda()
    i = torch.tensor(idx, dtype=torch.int64, device="cuda")
    v = words(to_mont_array(vals))
    off = 1 if vals_at == "eight bytes off" else 0
    buf = torch.zeros(v.numel() + 2, dtype=torch.int64)
    buf = buf.pin_memory() if vals_at == "pinned" else buf.cuda()
    buf[off:off + v.numel()] = v
    torch.cuda.synchronize()
    t, ot = Transcript(b"sd"), o.Transcript(b"sd")
    p = SparseDenseSumcheckProver(n, t)
    proof = p.prove(ctx, None, None, DenseMLPoly(n, device_ptr=d.data_ptr()), t, device_ptrs=(i.data_ptr(), buf.data_ptr() + 8 * off, nnz))
    _, oproof = o.sparse_dense_prove(n, idx, vals, dense, ot)
    assert proof.round_messages == oproof.round_messages and proof.final_eval == oproof.final_eval


def test_rejects_a_bad_order_on_the_device(ctx):
    """The word that the launch writes into host memory, once set and once not."""
    import torch
    d = torch.zeros(4 << 6, dtype=torch.int64, device="cuda")
    v = torch.zeros(8, dtype=torch.int64, device="cuda")
    dense = DenseMLPoly(6, device_ptr=d.data_ptr())
    for idx, ok in (([3, 2], False), ([2, 3], True), ([5, 5], False), ([5, 64], False), ([5, 1 << 40], False), ([5, 63], True)):
        i = torch.tensor(idx, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        t = Transcript(b"sd")
        p = SparseDenseSumcheckProver(6, t)
        if ok:
            assert p.prove(ctx, None, None, dense, t, device_ptrs=(i.data_ptr(), v.data_ptr(), 2)).final_eval == 0
        else:
            with pytest.raises(ZkError):
                p.prove(ctx, None, None, dense, t, device_ptrs=(i.data_ptr(), v.data_ptr(), 2))
