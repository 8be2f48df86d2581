"""The sharded entry points with their ranks as threads of this process, a context each, on one GPU: argv[1] is the stand-in for NCCL
(hostgather.cpp), argv[2] the number of ranks; with argv[3] one share of an all-gather is damaged."""
import ctypes
import os
import random
import sys
import threading

gather = ctypes.CDLL(sys.argv[1], mode=ctypes.RTLD_GLOBAL)  # before the library looks for libnccl.so.2, and torch stays out
ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
sys.path[:0] = [ROOT, os.path.join(ROOT, "oracle")]
import pyoracle as o
from zkes_b200 import Context, DenseMLPoly, Transcript
from zkes_b200 import dist as zd
from zkes_b200._lib import ZK_ERR_COMM, ZK_OPT_AHEAD_LOG, ZK_OPT_PEER_EXCHANGE, ZK_OPT_REPLICATE_LOG, ZkError, check, lib

M = o.R_MOD
WORLD = int(sys.argv[2])
LOG = zd.log2_exact(WORLD)


class Rank:
    pass


def start():
    uid = (ctypes.c_uint8 * 128)()
    check(lib.zk_comm_unique_id(uid), "zk_comm_unique_id")
    ranks = []
    for r in range(WORLD):
        k = Rank()
        k.ctx, k.rank, k.world = Context(0), r, WORLD
        k.ctx.set_option(ZK_OPT_PEER_EXCHANGE, 0)
        ranks.append(k)

    def join(k):
        k.handle = ctypes.c_void_p()
        check(lib.zk_comm_init(k.ctx.handle, k.rank, WORLD, uid, ctypes.byref(k.handle)), "zk_comm_init")
        assert not lib.zk_comm_peer_exchange(k.handle)

    on_all(ranks, join)
    return ranks


def on_all(ranks, work):
    got, wrong = [None] * WORLD, []

    def run(k):
        try:
            got[k.rank] = work(k)
        except BaseException as e:
            wrong.append(e)

    threads = [threading.Thread(target=run, args=(k,)) for k in ranks]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if wrong:
        raise wrong[0]
    return got


def linear(ranks, n, tables):
    def prove(k):
        t = Transcript(b"ranks")
        t.append_u64(b"num_var", n)
        t.append_u64(b"num_poly", len(tables))
        local = [DenseMLPoly.from_evaluations(zd.shard_dense(tb, k.rank, WORLD)) for tb in tables]
        return zd.sharded_linear_prove(k.ctx, k, n, local, t)

    ot = o.Transcript(b"ranks")
    op = o.LinearSumcheckProver(n, len(tables), ot)
    proof = op.prove(tables, ot)
    want = (proof.round_messages, op.challenges, [x[0] for x in op.a_arrays], proof.final_eval)
    for r, got in enumerate(on_all(ranks, prove)):
        assert tuple(got) == want, ("linear", n, len(tables), r)


def sparse(ranks, n, idx, vals, dense):
    def prove(k):
        t = Transcript(b"ranks")
        t.append_u64(b"num_var", n)
        t.append_u64(b"num_poly", 2)
        li, lv = zd.shard_sparse(idx, vals, k.rank, WORLD, n)
        return zd.sharded_sparse_dense_prove(k.ctx, k, n, li, lv, DenseMLPoly.from_evaluations(zd.shard_dense(dense, k.rank, WORLD)), t)

    ot = o.Transcript(b"ranks")
    op, proof = o.sparse_dense_prove(n, idx, vals, dense, ot)
    want = (proof.round_messages, op.challenges, [x[0] for x in op.a_arrays], proof.final_eval)
    for r, got in enumerate(on_all(ranks, prove)):
        assert tuple(got) == want, ("sparse", n, len(idx), r)


def healthy():
    ranks = start()
    rnd = random.Random(WORLD)
    for replicate_log, ahead_log in ((0, 14), (0, 0), (18, 14)):
        for k in ranks:
            k.ctx.set_option(ZK_OPT_REPLICATE_LOG, replicate_log)
            k.ctx.set_option(ZK_OPT_AHEAD_LOG, ahead_log)
        for n in (LOG, LOG + 1, LOG + 5):  # one entry of a table a rank, two, more
            for L in (1, 2, 3, 4):
                linear(ranks, n, [[rnd.randrange(M) for _ in range(1 << n)] for _ in range(L)])
            dense = [rnd.randrange(M) for _ in range(1 << n)]
            for nnz in (0, 1, min(1 << n, 40)):
                idx = sorted(rnd.sample(range(1 << n), nnz))
                sparse(ranks, n, idx, [rnd.randrange(M) for _ in idx], dense)


def damaged():
    """In the entry rounds s(1) is what the round before leaves for it, so a damaged share shows where the dense rounds begin and sum
    s(0) and s(1) again: whichever all-gather it was, no rank returns a proof, and the communicator stays retired."""
    rnd = random.Random(7)
    n = LOG + 9
    dense = [rnd.randrange(M) for _ in range(1 << n)]
    idx = [r << 9 | j for r in range(WORLD) for j in (3, 4, 77, 200, 201, 300, 411, 500)]  # eight entries a rank: rounds of 2^9 to 2^5 in entry form
    vals = [rnd.randrange(1, M) for _ in idx]
    for replicate_log in (0, 18):
        for first in (4, 5, 8, 9):  # two all-gathers of the start and one of the counts, then the rounds; 9: a round of the dense form or its table
            gather.hostgather_damage(0)
            ranks = start()
            for k in ranks:
                k.ctx.set_option(ZK_OPT_REPLICATE_LOG, replicate_log)

            def prove(k):
                t = Transcript(b"ranks")
                t.append_u64(b"num_var", n)
                t.append_u64(b"num_poly", 2)
                li, lv = zd.shard_sparse(idx, vals, k.rank, WORLD, n)
                try:
                    zd.sharded_sparse_dense_prove(k.ctx, k, n, li, lv, DenseMLPoly.from_evaluations(zd.shard_dense(dense, k.rank, WORLD)), t)
                except ZkError as e:
                    return e.code
                return 0

            gather.hostgather_damage(first)
            for again in range(2):
                assert on_all(ranks, prove) == [ZK_ERR_COMM] * WORLD, (replicate_log, first, again)
            for k in ranks:
                lib.zk_comm_free(k.ctx.handle, k.handle)
                k.ctx.close()


damaged() if len(sys.argv) > 3 else healthy()
print("ranks ok")
