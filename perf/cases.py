"""Workloads by which the speed of the proving path is followed.

Each case is one call, or one short run of calls, that a prover makes into the library: the sumcheck provers, the
commitments and their openings, a bare multi-scalar multiplication, and the table work of a node proof.  The calls go
through the C ABI on device-resident tables, as `bench.py` and `zkes_b200/gpt2_trace.py` make them; lists of positions
live in pinned host memory, where the library takes them from.  Results that a proof carries as projective points are
brought to affine form in the same pass (`zk_g1_normalize`), which is the form in which a proof is written out, and the
only one in which two correct computations agree byte for byte.
"""
from __future__ import annotations

import ctypes
import functools
import math
from ctypes import c_void_p as vp

import numpy as np
import torch

from zkes_b200 import Context, kzh
from zkes_b200._lib import ZK_MEM_DEVICE, ZK_MEM_HOST, check, lib
from zkes_b200.field import to_mont_array

G = (1368015179489954701390400359078579693043519447331113978918064868415326638035,
     9918110051302171585080402603319702774565515993150576347155970296011118125764)
FR = 32               # bytes of a field element
POINT = 64            # bytes of an affine point
LOOKUP_TABLE_LOG = 4  # a lookup's selection polynomial has 2^4 table rows per looked-up element


def listed():
    return [
        # the sumcheck of a layer norm's einsum: three tables over one sequence axis, over a hundred of them in a proof
        {"name": "linear_n7_l3", "kind": "linear", "n": 7, "polys": 3},
        # the dense prover at the size of the reference's own benchmark of it: two uniform tables
        {"name": "linear_n20_l2", "kind": "linear", "n": 20, "polys": 2},
        # quantised weights against a dense table: the headline workload
        {"name": "sparse_dense_n26", "kind": "sparse_dense", "n": 26, "nnz": 1 << 20},
        # commitment to a quantised weight matrix
        {"name": "kzh2_commit_n24_int8", "kind": "kzh2_commit", "n": 24, "bits": 8},
        # its opening
        {"name": "kzh2_open_n24", "kind": "kzh2_open", "n": 24, "bits": 8},
        # commitment and opening of a table whose slabs alternate between activations and full-width elements
        {"name": "kzh3_n22_mixed", "kind": "kzh3", "n": 22},
        # a multi-scalar multiplication with full-width scalars over a length that is no power of two
        {"name": "msm_100003_full", "kind": "msm", "count": 100003, "bits": 0},
        # commitment to the selection polynomial of a lookup over 2^18 elements, and its opening
        {"name": "selection_commit_2e18", "kind": "selection_commit", "log": 18, "entries": 1 << 18},
        {"name": "selection_open_2e18", "kind": "selection_open", "log": 18, "entries": 1 << 18},
        # the boolean check over the selection polynomials of one size
        {"name": "bool_check_16x2e17", "kind": "bool_check", "log": 17, "entries": 1 << 17, "terms": 16},
        # the proof of a matrix product in an MLP: inputs bound on their free variables, then the sumcheck
        {"name": "matmul_node_s7_d10_f12", "kind": "matmul_node", "seq": 7, "inner": 10, "outer": 12},
        # lookup preprocessing: one auxiliary polynomial of 2^17 elements scattered into a block of the table
        {"name": "range_aux_2e17", "kind": "range_aux", "log": 17, "table": 4},
    ]


def draw(rng):
    def count(lo, hi):  # spread over the logarithm
        return int(round(2 ** rng.uniform(lo, hi)))

    kind = rng.choice(["linear", "sparse_dense", "kzh2_commit", "kzh2_open", "kzh3", "msm", "selection_commit", "selection_open",
                       "bool_check", "matmul_node", "range_aux"])
    c = {"kind": kind}
    if kind == "linear":
        c.update(n=rng.randint(3, 20), polys=rng.choice([1, 2, 2, 3, 3, 4]))
    elif kind == "sparse_dense":
        n = rng.randint(12, 26)
        c.update(n=n, nnz=count(4, min(20, n - 3)))
    elif kind == "kzh2_commit":
        n = rng.randint(8, 24)
        c.update(n=n, bits=rng.choice([8, 8, 16] + ([0] if n <= 20 else [])))
    elif kind == "kzh2_open":
        c.update(n=rng.randint(8, 24), bits=rng.choice([8, 16, 0]))
    elif kind == "kzh3":
        c.update(n=rng.randint(9, 21))
    elif kind == "msm":
        c.update(count=count(4, 18), bits=rng.choice([8, 16, 0, 0]))
    elif kind in ("selection_commit", "selection_open"):
        log = rng.randint(10, 19)
        c.update(log=log, entries=count(log - 1, log))  # a padded tensor looks up fewer elements than its table has
    elif kind == "bool_check":
        log = rng.randint(8, 17)
        c.update(log=log, entries=count(log - 1, log), terms=rng.randint(1, 16))
    elif kind == "matmul_node":
        seq, inner, outer = rng.randint(4, 9), rng.randint(6, 11), rng.randint(6, 12)
        c.update(seq=seq, inner=inner, outer=min(outer, 22 - inner))
    else:
        c.update(log=rng.randint(8, 19), table=rng.choice([4, 4, 4, 8, 12, 16]))
    return c


# ---------------------------------------------------------------------------------------------- what a program keeps
@functools.lru_cache(maxsize=None)
def context():
    """A program makes one context per GPU and keeps it."""
    return Context(0)


class State(dict):
    """The inputs of a call, with the buffers and handles that the caller holds for it."""
    __getattr__ = dict.__getitem__


def _device(count, width=4):
    return torch.empty((count, width), dtype=torch.int64, device="cuda")


def _uniform(seed, stream, count):
    t = _device(count)
    torch.cuda.synchronize()
    check(lib.zk_gen_uniform_fr(context().handle, seed, stream, 0, count, vp(t.data_ptr())), "zk_gen_uniform_fr")
    return t


def _scalars(seed, stream, count, bits):
    """Signed integers of `bits` bits as field elements, or uniform field elements for bits = 0."""
    if not bits:
        return _uniform(seed, stream, count)
    t = _device(count)
    torch.cuda.synchronize()
    check(lib.zk_gen_small_fr(context().handle, seed, stream, 0, count, bits, vp(t.data_ptr())), "zk_gen_small_fr")
    return t


def _integers(seed, count):
    """int16 witness values as little-endian 128-bit integers."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    lo = torch.randint(-(1 << 15), 1 << 15, (count,), generator=g, device="cuda", dtype=torch.int64)
    return torch.stack([lo, lo >> 63], dim=1).contiguous()


def _host_fr(seed, stream, count):
    t = _uniform(seed, stream, max(count, 1))
    context().sync()
    return t[:count].cpu().numpy().view(np.uint64).copy()


def _srs(seed, dims, n):
    if dims == 2:
        logs = (n // 2, n - n // 2)
    else:
        k, r = divmod(n, 3)
        logs = (k + (r >= 1), k + (r == 2), k)
    rnd = np.random.default_rng(seed)
    taus = [[int(x) for x in rnd.integers(1, 1 << 62, size=1 << lg)] for lg in logs]
    return kzh.KZHSRS.setup(context(), dims, n, G, taus[0], taus[1], tau_z=taus[2] if dims == 3 else None,
                            alpha=12345 if dims == 2 else None)


def _pinned(values):
    t = torch.empty(values.shape, dtype=torch.int64, pin_memory=True)
    t.copy_(torch.from_numpy(values.view(np.int64)))
    return t


def _selection(seed, log, entries, terms=1):
    """One entry per looked-up element: position = table row << log | element."""
    rnd = np.random.default_rng(seed)
    rows = rnd.integers(0, 1 << LOOKUP_TABLE_LOG, size=(terms, entries), dtype=np.uint64)
    return (rows << np.uint64(log)) | np.arange(entries, dtype=np.uint64)


def _host(rows, width):
    return np.zeros((rows, width), dtype=np.uint64)


def prepare(case, seed):
    context()
    k = case["kind"]
    s = State(kind=k, case=case)
    if k == "linear":
        n, ell = case["n"], case["polys"]
        s.update(tables=[_uniform(seed, i, 1 << n) for i in range(ell)], msgs=_host(n * (ell + 1), 4), chal=_host(n, 4),
                 fin_t=_host(ell, 4), fin=_host(1, 4))
    elif k == "sparse_dense":
        n, nnz = case["n"], case["nnz"]
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        # distinct positions, ascending: the cumulative sums of random gaps that fit the domain
        gap = (1 << n) // nnz
        pos = torch.arange(nnz, device="cuda", dtype=torch.int64) * gap + torch.randint(0, gap, (nnz,), generator=g, device="cuda")
        s.update(idx=pos.contiguous(), val=_scalars(seed, 2, nnz, 8), dense=_uniform(seed, 0, 1 << n), msgs=_host(n * 3, 4),
                 chal=_host(n, 4), fin_t=_host(2, 4), fin=_host(1, 4))
    elif k == "kzh2_commit":
        n = case["n"]
        srs = _srs(seed, 2, n)
        s.update(srs=srs, f=_scalars(seed, 7, 1 << n, case["bits"]), c=_host(1, 8), dx=_host(1 << srs.x_log, 12),
                 dx_affine=_host(1 << srs.x_log, 8))
    elif k == "kzh2_open":
        n = case["n"]
        srs = _srs(seed, 2, n)
        s.update(srs=srs, f=_scalars(seed, 7, 1 << n, case["bits"]), point=_host_fr(seed, 9, n), f_star=_host(1 << srs.y_log, 4))
    elif k == "kzh3":
        n = case["n"]
        srs = _srs(seed, 3, n)
        f = _uniform(seed, 7, 1 << n).view(1 << srs.x_log, -1)
        slab = 1 << (n - srs.x_log)
        context().sync()
        for x in range(0, f.shape[0], 2):  # even slabs: activations round(N(0, 1) 2^8)
            check(lib.zk_gen_gauss_fr(context().handle, seed, 8, x * slab, slab, 8, vp(f[x].data_ptr())), "zk_gen_gauss_fr")
        rx, ry, rz = 1 << srs.x_log, 1 << srs.y_log, 1 << srs.z_log
        s.update(srs=srs, f=f, point=_host_fr(seed, 9, n), c=_host(1, 8), dx=_host(rx, 12), dy=_host(ry, 12), cy=_host(1, 8),
                 f_star=_host(rz, 4), dx_affine=_host(rx, 8), dy_affine=_host(ry, 8))
    elif k == "msm":
        m = case["count"]
        srs = _srs(seed, 2, max(2, (m - 1).bit_length()))  # its points serve as bases
        bases = _host(m, 8)
        check(lib.zk_kzh_srs_read(context().handle, srs.handle, 0, 0, m, vp(bases.ctypes.data)), "zk_kzh_srs_read")
        srs.close()
        s.update(bases=torch.from_numpy(bases.view(np.int64)).cuda(), f=_scalars(seed, 7, m, case["bits"]), jac=_host(1, 12),
                 affine=_host(1, 8))
    elif k in ("selection_commit", "selection_open"):
        log = case["log"]
        srs = _srs(seed, 2, log + LOOKUP_TABLE_LOG)
        s.update(srs=srs, pos=_pinned(_selection(seed, log, case["entries"])[0]), c=_host(1, 8), dx=_host(1 << srs.x_log, 12),
                 dx_affine=_host(1 << srs.x_log, 8), point=_host_fr(seed, 9, log + LOOKUP_TABLE_LOG), f_star=_host(1 << srs.y_log, 4))
    elif k == "bool_check":
        log, terms = case["log"], case["terms"]
        m = log + LOOKUP_TABLE_LOG
        s.update(pos=_pinned(_selection(seed, log, case["entries"], terms).reshape(-1)), counts=np.full(terms, case["entries"], dtype=np.uint64),
                 weights=_host_fr(seed, 5, terms), point=_host_fr(seed, 9, m), msgs=_host(m * 4, 4), chal=_host(m, 4), fin=_host(1, 4))
    elif k == "matmul_node":
        sq, inner, outer = case["seq"], case["inner"], case["outer"]
        s.update(x=_integers(seed, 1 << (sq + inner)), w=_integers(seed + 1, 1 << (inner + outer)), bias=_scalars(seed, 3, 1 << (sq + outer), 16),
                 xt=_device(1 << (sq + inner), 2), x_bound=_device(1 << inner), w_bound=_device(1 << inner), eq=_device(1 << inner),
                 point=_host_fr(seed, 9, sq + inner + outer), msgs=_host(inner * 4, 4), chal=_host(inner, 4), fin_t=_host(3, 4),
                 fin=_host(1, 4), at=_host(1, 4))
    else:
        log, table = case["log"], case["table"]
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        s.update(inputs=torch.arange(1 << log, dtype=torch.int64, device="cuda"),
                 rows=torch.randint(0, 1 << table, (1 << log,), generator=g, device="cuda", dtype=torch.int64),
                 point=_host_fr(seed, 9, log), weight=_host_fr(seed, 5, 1), acc=_uniform(seed, 6, 1 << table), sums=_device(1 << table),
                 middle=_host(1, 4))
    context().sync()
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------------------------- the calls
def _p(a):
    return vp(a.ctypes.data)


def _d(t):
    return vp(t.data_ptr())


def _transcript(n, polys):
    tr = lib.zk_transcript_new(b"proof", 5)
    lib.zk_transcript_append_u64(tr, b"num_var", 7, n)
    lib.zk_transcript_append_u64(tr, b"num_poly", 8, polys)
    return tr


def _linear(h, n, tables, s):
    ell = len(tables)
    tr = _transcript(n, ell)
    ptrs = (vp * ell)(*[_d(t) for t in tables])
    check(lib.zk_sumcheck_linear_prove(h, n, ell, ptrs, ZK_MEM_DEVICE, None, None, tr, _p(s.msgs), _p(s.chal), _p(s.fin_t), _p(s.fin)),
          "zk_sumcheck_linear_prove")
    lib.zk_transcript_free(tr)
    return [s.msgs, s.chal, s.fin_t, s.fin]


def _affine(h, jac, out):
    check(lib.zk_g1_normalize(h, _p(jac), ZK_MEM_HOST, jac.shape[0], _p(out), ZK_MEM_HOST), "zk_g1_normalize")
    return out


def run(state):
    s, h, case = state, context().handle, state.case
    k = s.kind
    if k == "linear":
        return _linear(h, case["n"], s.tables, s)
    if k == "sparse_dense":
        tr = _transcript(case["n"], 2)
        check(lib.zk_sumcheck_sparse_dense_prove(h, case["n"], case["nnz"], _d(s.idx), _d(s.val), _d(s.dense), ZK_MEM_DEVICE, None, None,
                                                 tr, _p(s.msgs), _p(s.chal), _p(s.fin_t), _p(s.fin)), "zk_sumcheck_sparse_dense_prove")
        lib.zk_transcript_free(tr)
        return [s.msgs, s.chal, s.fin_t, s.fin]
    if k == "kzh2_commit":
        check(lib.zk_kzh_commit(h, s.srs.handle, case["n"], _d(s.f), ZK_MEM_DEVICE, _p(s.c), _p(s.dx)), "zk_kzh_commit")
        return [s.c, _affine(h, s.dx, s.dx_affine)]
    if k == "kzh2_open":
        check(lib.zk_kzh2_open(h, s.srs.handle, case["n"], _d(s.f), ZK_MEM_DEVICE, _p(s.point), case["n"], _p(s.f_star)), "zk_kzh2_open")
        return s.f_star
    if k == "kzh3":
        check(lib.zk_kzh_commit(h, s.srs.handle, case["n"], _d(s.f), ZK_MEM_DEVICE, _p(s.c), _p(s.dx)), "zk_kzh_commit")
        check(lib.zk_kzh3_open(h, s.srs.handle, case["n"], _d(s.f), ZK_MEM_DEVICE, _p(s.point), case["n"], _p(s.dx), _p(s.dy), _p(s.cy),
                               _p(s.f_star)), "zk_kzh3_open")
        return [s.c, _affine(h, s.dx, s.dx_affine), _affine(h, s.dy, s.dy_affine), s.cy, s.f_star]
    if k == "msm":
        check(lib.zk_msm_g1(h, _d(s.bases), ZK_MEM_DEVICE, _d(s.f), ZK_MEM_DEVICE, case["count"], _p(s.jac), ZK_MEM_HOST), "zk_msm_g1")
        return _affine(h, s.jac, s.affine)
    if k == "selection_commit":
        check(lib.zk_sparse_kzh_commit(h, s.srs.handle, case["entries"], _d(s.pos), None, _p(s.c), _p(s.dx)), "zk_sparse_kzh_commit")
        return [s.c, _affine(h, s.dx, s.dx_affine)]
    if k == "selection_open":
        check(lib.zk_sparse_kzh2_open(h, s.srs.handle, case["entries"], _d(s.pos), None, _p(s.point), case["log"] + LOOKUP_TABLE_LOG,
                                      _p(s.f_star)), "zk_sparse_kzh2_open")
        return s.f_star
    if k == "bool_check":
        m = case["log"] + LOOKUP_TABLE_LOG
        tr = _transcript(m, 3)
        check(lib.zk_sumcheck_sparse_bool_prove(h, m, case["terms"], _p(s.weights), _d(s.pos), _p(s.counts), _p(s.point), None, None, tr,
                                                _p(s.msgs), _p(s.chal), _p(s.fin)), "zk_sumcheck_sparse_bool_prove")
        lib.zk_transcript_free(tr)
        return [s.msgs, s.chal, s.fin]
    if k == "matmul_node":
        sq, inner, outer = case["seq"], case["inner"], case["outer"]
        # out[s, f] = sum_i x[s, i] w[i, f]: x is brought to the layout that has its sequence axis in the low variables,
        # both inputs are bound at the claim's point, and the sumcheck runs over the inner axis
        ranges = np.array([inner, inner + sq, 0, inner], dtype=np.uint64)
        check(lib.zk_permute_by_ranges(h, sq + inner, 16, _d(s.x), ZK_MEM_DEVICE, 2, _p(ranges), _d(s.xt), ZK_MEM_DEVICE),
              "zk_permute_by_ranges")
        check(lib.zk_fix_variables_int(h, sq + inner, _d(s.xt), ZK_MEM_DEVICE, sq, _p(s.point), _d(s.x_bound), ZK_MEM_DEVICE),
              "zk_fix_variables_int")
        check(lib.zk_fix_variables_int(h, inner + outer, _d(s.w), ZK_MEM_DEVICE, outer, _p(s.point[sq:]), _d(s.w_bound), ZK_MEM_DEVICE),
              "zk_fix_variables_int")
        check(lib.zk_eq_table(h, inner, _p(s.point[sq + outer:]), _d(s.eq), ZK_MEM_DEVICE), "zk_eq_table")
        out = _linear(h, inner, [s.x_bound, s.w_bound, s.eq], s)
        check(lib.zk_mle_eval(h, sq + outer, _d(s.bias), ZK_MEM_DEVICE, _p(s.point), _p(s.at)), "zk_mle_eval")
        return out + [s.x_bound, s.w_bound, s.at]
    s.sums.copy_(s.acc)  # the running sums over the auxiliary polynomials; this pass adds one to them
    torch.cuda.current_stream().synchronize()
    check(lib.zk_range_aux_accumulate(h, case["log"], _p(s.point), 1 << case["log"], _d(s.inputs), _d(s.rows), ZK_MEM_DEVICE, _p(s.weight),
                                      case["table"], _d(s.sums), ZK_MEM_DEVICE, _p(s.middle)), "zk_range_aux_accumulate")
    return [s.sums, s.middle]


# ---------------------------------------------------------------------------------------------- what a pass needs
MUL = 2 * 136         # a 256-bit modular product is 136 multiply-adds of 32 x 32 bits, two operations each
ADD = 6 * MUL         # an addition of points: five products and a square, the inversion shared among many


def _msm_additions(count, bits):
    """Additions of the bucket method with the cheapest window: every window adds each base once and reduces its buckets."""
    width = 254 if not bits else bits
    return min(math.ceil(width / w) * (count + (1 << w)) for w in range(2, 18))


def work(case):
    k = case["kind"]
    if k == "linear":
        ell, size = case["polys"], 1 << case["n"]
        # per pair of entries and round: the folds of the tables and ell + 1 values of the message
        return {"bytes": FR * ell * size, "flops": MUL * size * (ell + (ell + 1) * max(ell - 1, 0))}
    if k == "sparse_dense":
        size, nnz = 1 << case["n"], case["nnz"]
        return {"bytes": FR * size + (8 + FR) * nnz, "flops": MUL * (size + 3 * nnz)}
    if k == "kzh2_commit":
        size = 1 << case["n"]
        return {"bytes": (FR + POINT) * size, "flops": ADD * 2 * _msm_additions(size, case["bits"])}
    if k == "kzh2_open":
        return {"bytes": FR * (1 << case["n"]), "flops": MUL * (1 << case["n"])}
    if k == "kzh3":
        half = 1 << (case["n"] - 1)
        return {"bytes": 2 * FR * 2 * half + POINT * 2 * half,
                "flops": ADD * 2 * (_msm_additions(half, 10) + _msm_additions(half, 0)) + MUL * 2 * half}
    if k == "msm":
        return {"bytes": (FR + POINT) * case["count"], "flops": ADD * _msm_additions(case["count"], case["bits"])}
    if k == "selection_commit":
        nnz = case["entries"]
        return {"bytes": (8 + POINT) * nnz, "flops": ADD * 2 * nnz}
    if k == "selection_open":
        return {"bytes": 8 * case["entries"], "flops": 0}
    if k == "bool_check":
        nnz = case["terms"] * case["entries"]
        return {"bytes": 8 * nnz + FR * (1 << (case["log"] + LOOKUP_TABLE_LOG)), "flops": MUL * 4 * 2 * nnz}
    if k == "matmul_node":
        x, w, b = 1 << (case["seq"] + case["inner"]), 1 << (case["inner"] + case["outer"]), 1 << (case["seq"] + case["outer"])
        return {"bytes": 16 * (3 * x + w) + FR * b, "flops": MUL * (x + w) // 16 + MUL * (b + 11 * (1 << case["inner"]))}
    nnz = 1 << case["log"]
    return {"bytes": 16 * nnz + 3 * FR * (1 << case["table"]), "flops": MUL * (nnz + 2 * (1 << case["table"]))}


def tolerance(case):
    """Field elements and points in affine form are whole numbers: there is one right answer."""
    return "exact"
