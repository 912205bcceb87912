"""The work that users of this package have it do, as cases that can be timed.

Every case goes through the public entry points of ``trident_b200.ops`` with
operands on the GPU.  The kinds, and what each stands for in a program that
uses the package:

* ``spgemm``    one plain product C = A·B (LocalMatrix::spgemm): the local tile
                product of a SUMMA stage, or a whole product on one GPU
* ``plan``      the numeric half of a product whose pattern is kept
                (structure reuse: new values, same pattern)
* ``galerkin``  the AMG coarse operator R·(A·P) as two products
* ``batch``     many independent products of uneven sizes in one run
* ``mma``       C_out = C_in + A·B, the accumulate of a SUMMA stage
* ``spadd``     the merge of two partial C tiles
* ``exchange``  one stage of the sparsity-aware exchange: stage mask, both
                tiles packed by it, unpacked, and A' turned from CSC to CSR
* ``coo``       COO coordinates to CSR / CSC, the tile build
* ``transpose`` CSC <-> CSR of a whole matrix
* ``mcl``       one Markov-clustering iteration: expand, inflate, prune

Inputs are made on the GPU: R-MAT (.57, .19, .19, .05) with duplicates merged,
rows of uniform-random columns (fixed or Poisson lengths) and 27- or 7-point
stencils.  A case has one pattern of its own; the seed draws the values and
relabels the rows and columns by a cyclic shift, so that inputs of another
seed are other matrices whose results have the same sizes.
"""
from __future__ import annotations

import functools
import json
import math
import os
import zlib

import torch

from trident_b200 import ops
from trident_b200._lib import TSPG_COLS, TSPG_ROWS
from trident_b200.csr import DeviceCSR

_DEV = "cuda"
_TUNING = os.path.join(os.path.dirname(os.path.abspath(ops.__file__)), "tuning")


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest call: 1024 x 1024, 16 uniform columns and the diagonal
        # per row, int32 offsets (a tile of a small run; latency counts)
        dict(name="spgemm_uniform_1k", kind="spgemm", matrix="uniform", n=1024, k=16, val=64, ptr=32, tuning=""),
        # a stage tile of the unchanged <int32, float> drivers, odd order
        dict(name="spgemm_rmat_20k_f32", kind="spgemm", matrix="rmat", n=20011, k=8, val=32, ptr=32, tuning=""),
        # the large graph square with its committed row binning
        dict(name="spgemm_rmat_2e18", kind="spgemm", matrix="rmat", n=1 << 18, k=16, val=64, ptr=64, tuning="rmat"),
        # structure reuse: a 27-point stencil squared again with new values
        dict(name="plan_stencil_63", kind="plan", matrix="stencil", n=63, k=27, val=64, ptr=32, tuning=""),
        # AMG set-up on a 128^3 grid, 3^3 aggregates
        dict(name="galerkin_128", kind="galerkin", n=128, k=27, agg=3, val=64, ptr=64, tuning="rap"),
        # independent products of 1k to 200k rows, Poisson row lengths
        dict(name="batch_poisson_20", kind="batch", count=20, rows_lo=1000, rows_hi=200000, lam_lo=8.0, lam_hi=32.0,
             val=64, ptr=64, tuning="batched"),
        # a late SUMMA stage: a full accumulator and one more tile product
        dict(name="mma_stage_2e17", kind="mma", n=1 << 17, k=4, kc=64, val=64, ptr=32, tuning=""),
        # partial C tiles of a hub-heavy graph
        dict(name="spadd_rmat_2e18", kind="spadd", matrix="rmat", n=1 << 18, k=64, val=64, ptr=64),
        # the exchange of one stage of a 4 x 4 grid over a scale-19 graph
        dict(name="exchange_tile_2e17", kind="exchange", n=1 << 17, k=6, val=64, ptr=32),
        # the tile build from shuffled coordinates of the scale-20 graph
        dict(name="coo_rmat_2e20", kind="coo", n=1 << 20, k=16, major="rows", val=64, ptr=64),
        # CSC -> CSR of short, even segments (the stencil operator), FP32
        dict(name="transpose_stencil_100", kind="transpose", matrix="stencil", n=100, k=27, val=32, ptr=32),
        # clustering of a mid-size graph
        dict(name="mcl_rmat_30k", kind="mcl", n=30011, k=8, power=2.0, tol=1.1e-4, val=64, ptr=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spgemm", "spgemm", "spgemm", "plan", "galerkin", "batch", "mma", "spadd", "exchange", "coo",
                       "transpose", "mcl"])
    val, ptr = rng.choice([64, 64, 32]), rng.choice([32, 64])
    if kind == "spgemm":
        matrix = rng.choice(["uniform", "poisson", "rmat", "rmat"])
        n = _log(rng, 700, 150000)
        k = rng.randint(4, 30 if matrix != "rmat" else 14)
        return dict(kind=kind, matrix=matrix, n=n, k=k, val=val, ptr=ptr,
                    tuning=rng.choice(["", "rmat"]) if matrix == "rmat" else "")
    if kind == "plan":
        matrix = rng.choice(["stencil", "uniform", "rmat"])
        n = _log(rng, 10, 70) if matrix == "stencil" else _log(rng, 700, 100000)
        k = rng.choice([7, 27]) if matrix == "stencil" else rng.randint(4, 12)
        return dict(kind=kind, matrix=matrix, n=n, k=k, val=val, ptr=ptr, tuning="")
    if kind == "galerkin":
        return dict(kind=kind, n=_log(rng, 12, 120), k=rng.choice([7, 27]), agg=rng.choice([2, 3]), val=64, ptr=ptr,
                    tuning=rng.choice(["", "rap"]))
    if kind == "batch":
        lo = _log(rng, 300, 3000)
        return dict(kind=kind, count=rng.randint(2, 20), rows_lo=lo, rows_hi=_log(rng, 2 * lo, 150000), lam_lo=4.0,
                    lam_hi=round(rng.uniform(8.0, 32.0), 1), val=val, ptr=ptr, tuning=rng.choice(["", "batched"]))
    if kind == "mma":
        return dict(kind=kind, n=_log(rng, 3000, 130000), k=rng.randint(3, 6), kc=_log(rng, 2, 64), val=val, ptr=ptr,
                    tuning="")
    if kind == "spadd":
        matrix = rng.choice(["rmat", "rmat", "poisson", "stencil"])
        n = _log(rng, 10, 100) if matrix == "stencil" else _log(rng, 1000, 250000)
        k = rng.choice([7, 27]) if matrix == "stencil" else _log(rng, 4, 64)
        return dict(kind=kind, matrix=matrix, n=n, k=k, val=val, ptr=ptr)
    if kind == "exchange":
        return dict(kind=kind, n=_log(rng, 2000, 260000), k=rng.randint(2, 8), val=val, ptr=ptr)
    if kind == "coo":
        return dict(kind=kind, n=_log(rng, 2000, 1000000), k=rng.randint(4, 16), major=rng.choice(["rows", "cols"]),
                    val=val, ptr=ptr)
    if kind == "transpose":
        matrix = rng.choice(["rmat", "poisson", "stencil"])
        n = _log(rng, 10, 110) if matrix == "stencil" else _log(rng, 1000, 600000)
        k = rng.choice([7, 27]) if matrix == "stencil" else rng.randint(4, 24)
        return dict(kind=kind, matrix=matrix, n=n, k=k, val=val, ptr=ptr)
    return dict(kind="mcl", n=_log(rng, 2000, 40000), k=rng.randint(3, 8), power=rng.choice([1.5, 2.0]),
                tol=rng.choice([1.1e-5, 1.1e-4, 1.1e-3]), val=64, ptr=ptr)


# ---------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=_DEV).manual_seed(seed)


def _pattern_gen(case):
    """The generator of the case's pattern: the same for every seed."""
    text = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    return _gen(zlib.crc32(text.encode()))


def _shifted(keys, n, seed):
    """Sorted keys row * n + col with rows and columns relabelled v + shift mod n."""
    shift = (seed * 7919 + 13) % n
    row = torch.div(keys, n, rounding_mode="floor")
    col = (keys - row * n + shift) % n
    return torch.sort((row + shift) % n * n + col).values


def _val_dtype(case):
    return torch.float64 if case["val"] == 64 else torch.float32


def _csr(keys, nrows, ncols, val, ptr_bits):
    """CSR of the sorted distinct keys row * ncols + col."""
    row = torch.div(keys, ncols, rounding_mode="floor")
    rowptr = torch.zeros(nrows + 1, dtype=torch.int64, device=_DEV)
    rowptr[1:] = torch.cumsum(torch.bincount(row, minlength=nrows), 0)
    col = (keys - row * ncols).to(torch.int32)
    return DeviceCSR(nrows, ncols, rowptr.to(torch.int32) if ptr_bits == 32 else rowptr, col, val, nnz=keys.numel())


def _uniform_values(g, n, dtype):
    return (torch.rand(n, generator=g, device=_DEV, dtype=torch.float64) * 2 - 1).to(dtype)


def _rmat_keys(g, n, k):
    """Distinct R-MAT coordinates below n (row * n + col), k draws per row of
    the enclosing power of two."""
    scale = max(1, (n - 1).bit_length())
    m = k << scale
    row = torch.zeros(m, dtype=torch.int64, device=_DEV)
    col = torch.zeros(m, dtype=torch.int64, device=_DEV)
    for _ in range(scale):
        u = torch.rand(m, generator=g, device=_DEV)
        row = 2 * row + (u >= 0.76).long()
        col = 2 * col + (((u >= 0.57) & (u < 0.76)) | (u >= 0.95)).long()
    keep = (row < n) & (col < n)
    return torch.unique(row[keep] * n + col[keep])


def _stencil_keys(n, pts):
    """Keys of the 27- or 7-point stencil on an n^3 grid, x fastest."""
    i = torch.arange(n ** 3, device=_DEV)
    x, y, z = i % n, (i // n) % n, i // (n * n)
    keys = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if pts == 7 and abs(dx) + abs(dy) + abs(dz) > 1:
                    continue
                ok = ((x + dx >= 0) & (x + dx < n) & (y + dy >= 0) & (y + dy < n) & (z + dz >= 0) & (z + dz < n))
                keys.append(torch.where(ok, i * n ** 3 + i + dx + n * (dy + n * dz), -1))
    keys = torch.stack(keys, 1).reshape(-1)
    return keys[keys >= 0]


def _stencil(g, n, pts, dtype, ptr):
    keys = _stencil_keys(n, pts)
    N = n ** 3
    v = -(0.5 + torch.rand(keys.numel(), generator=g, device=_DEV, dtype=torch.float64))
    v = torch.where(keys % (N + 1) == 0, -(pts - 1.0) * v, v)  # the diagonal: row * N + row
    return _csr(keys, N, N, v.to(dtype), ptr)


def _matrix(pg, g, case, seed, k=None, matrix=None):
    """A square operand of the case's kind: pattern from pg, values from g."""
    matrix, n, k = matrix or case["matrix"], case["n"], k or case["k"]
    dt, ptr = _val_dtype(case), case["ptr"]
    if matrix == "stencil":
        return _stencil(g, n, k, dt, ptr)
    if matrix == "rmat":
        keys = _rmat_keys(pg, n, k)
    else:
        keys = _random_keys(pg, n, k, matrix == "poisson", diag=matrix == "uniform")
    keys = _shifted(keys, n, seed)
    return _csr(keys, n, n, _uniform_values(g, keys.numel(), dt), ptr)


def _random_keys(g, n, k, poisson, diag):
    i = torch.arange(n, device=_DEV)
    if poisson:
        lens = torch.poisson(torch.full((n,), float(k), device=_DEV), generator=g).long().clamp_(max=n)
        row = torch.repeat_interleave(i, lens)
    else:
        row = i.repeat_interleave(k)
    keys = row * n + torch.randint(0, n, (row.numel(),), generator=g, device=_DEV)
    return torch.unique(torch.cat([keys, i * (n + 1)]) if diag else keys)


def _galerkin(g, case):
    """(R, A, P): the stencil, a prolongator on its pattern (row i reaches the
    agg^3 aggregates of its neighbours) and R = P^T."""
    n, pts, agg, ptr = case["n"], case["k"], case["agg"], case["ptr"]
    A = _stencil(g, n, pts, torch.float64, ptr)
    N, nc = n ** 3, -(-n // agg)
    keys = _stencil_keys(n, pts)
    row = torch.div(keys, N, rounding_mode="floor")
    j = keys - row * N
    c = ((j // (n * n)) // agg * nc + ((j // n) % n) // agg) * nc + (j % n) // agg
    pk = torch.unique(row * nc ** 3 + c)
    pv = torch.rand(pk.numel(), generator=g, device=_DEV, dtype=torch.float64)
    P = _csr(pk, N, nc ** 3, pv, ptr)
    prow = torch.div(pk, nc ** 3, rounding_mode="floor")
    rk, order = torch.sort((pk - prow * nc ** 3) * N + prow)
    return _csr(rk, nc ** 3, N, pv[order], ptr), A, P


def _batch_operands(pg, g, case, seed):
    out = []
    rel = torch.rand(case["count"], 2, generator=pg, device=_DEV, dtype=torch.float64).tolist()
    for u, v in rel:
        n = round(case["rows_lo"] * (case["rows_hi"] / case["rows_lo"]) ** u)
        lam = case["lam_lo"] + v * (case["lam_hi"] - case["lam_lo"])
        c = dict(case, n=n, k=lam, matrix="poisson")
        out.append((_matrix(pg, g, c, seed), _matrix(pg, g, c, seed)))
    return out


@functools.lru_cache(maxsize=None)
def _context(tuning):
    """One library context per row binning, as a program keeps them."""
    ctx = ops.Context(0)
    if tuning:
        with open(os.path.join(_TUNING, tuning + ".json")) as fh:
            ctx.set_tuning(json.load(fh)["tuning"])
    return ctx


def _inputs(case, seed):
    pg, g, kind = _pattern_gen(case), _gen(seed), case["kind"]
    if kind in ("spgemm", "plan", "transpose"):
        return dict(A=_matrix(pg, g, case, seed))
    if kind == "galerkin":
        R, A, P = _galerkin(g, case)
        return dict(R=R, A=A, P=P)
    if kind == "batch":
        return dict(pairs=_batch_operands(pg, g, case, seed))
    if kind == "mma":
        return dict(A=_matrix(pg, g, case, seed, matrix="rmat"), B=_matrix(pg, g, case, seed, matrix="rmat"),
                    C=_matrix(pg, g, case, seed, k=case["kc"], matrix="rmat"))
    if kind == "spadd":
        return dict(A=_matrix(pg, g, case, seed), B=_matrix(pg, g, case, seed))
    if kind == "exchange":
        # tiles whose columns and rows are partly empty, as R-MAT tiles are
        return dict(A=_matrix(pg, g, case, seed, matrix="rmat"), B=_matrix(pg, g, case, seed, matrix="rmat"))
    if kind == "coo":
        n = case["n"]
        keys = _shifted(_rmat_keys(pg, n, case["k"]), n, seed)
        keys = keys[torch.randperm(keys.numel(), generator=g, device=_DEV)]
        row = torch.div(keys, n, rounding_mode="floor")
        return dict(n=n, row=row.to(torch.int32), col=(keys - row * n).to(torch.int32),
                    val=_uniform_values(g, keys.numel(), _val_dtype(case)))
    # mcl: a row-stochastic matrix, self-loops added, every neighbour of a
    # vertex alike (the usual start); what is pruned depends on the values, so
    # the seed only relabels the vertices
    n = case["n"]
    i = torch.arange(n, device=_DEV)
    keys = _shifted(torch.unique(torch.cat([_rmat_keys(pg, n, case["k"]), i * (n + 1)])), n, seed)
    M = _csr(keys, n, n, None, case["ptr"])
    lens = M.rowptr[1:].long() - M.rowptr[:-1].long()
    M.val = (1.0 / lens.double()).repeat_interleave(lens)
    return dict(A=M)


def prepare(case, seed):
    st = _inputs(case, seed)
    ctx = _context(case.get("tuning", ""))
    st["case"], st["ctx"] = case, ctx
    if case["kind"] == "plan":
        A = st["A"]
        st["plan"] = ops.Plan(ctx, A, A)
        v = _uniform_values(_gen(seed + 1), A.nnz, A.val.dtype)
        st["A"] = DeviceCSR(A.nrows, A.ncols, A.rowptr, A.col, v, nnz=A.nnz)
    elif case["kind"] == "batch":
        st["batch"] = ops.Batch(ctx)
        for A, B in st["pairs"]:
            st["batch"].add(A, B)
    elif case["kind"] == "exchange":
        st["A_csc"] = ops.transpose(ctx, st["A"], rowptr_bits=case["ptr"])
    return st


def _out(M):
    return {"rowptr": M.rowptr, "col": M.col[:M.nnz], "val": M.val[:M.nnz]}


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind, ptr = case["kind"], case["ptr"]
    if kind == "spgemm":
        return _out(ops.spgemm(ctx, state["A"], state["A"], rowptr_bits=ptr))
    if kind == "plan":
        return _out(state["plan"].numeric(state["A"], state["A"], rowptr_bits=ptr))
    if kind == "galerkin":
        AP = ops.spgemm(ctx, state["A"], state["P"], rowptr_bits=ptr)
        return {"ap": _out(AP), "rap": _out(ops.spgemm(ctx, state["R"], AP, rowptr_bits=ptr))}
    if kind == "batch":
        state["batch"].run()
        results = [state["batch"].result(i) for i in range(case["count"])]
        for M in results:  # views of the batch's output slab: it lives as long as they do
            M.rowptr.owner = state["batch"]
        return [_out(M) for M in results]
    if kind == "mma":
        return _out(ops.sp_mma(ctx, state["A"], state["B"], state["C"], rowptr_bits=ptr))
    if kind == "spadd":
        return _out(ops.spadd(ctx, state["A"], state["B"], rowptr_bits=ptr))
    if kind == "exchange":
        A, B, Acsc = state["A"], state["B"], state["A_csc"]
        mask, mults, upper = ops.spgemm_count_mask(ctx, A, B)
        abuf, akept = ops.compress(ctx, Acsc, mask, TSPG_ROWS)
        Ap = ops.unpack(abuf, Acsc.nrows, Acsc.ncols, akept, TSPG_ROWS, case["val"], ptr)
        Ap = ops.csc_to_csr(ctx, Ap, rowptr_bits=ptr)
        bbuf, bkept = ops.compress(ctx, B, mask, TSPG_ROWS)
        Bp = ops.unpack(bbuf, B.nrows, B.ncols, bkept, TSPG_ROWS, case["val"], ptr)
        return {"mask": mask, "mults": mults, "upper": upper, "a": _out(Ap), "b": _out(Bp)}
    if kind == "coo":
        n, major = state["n"], TSPG_ROWS if case["major"] == "rows" else TSPG_COLS
        return _out(ops.coo_to_csx(ctx, n, n, state["row"], state["col"], state["val"], major, rowptr_bits=ptr))
    if kind == "transpose":
        return _out(ops.transpose(ctx, state["A"], rowptr_bits=ptr))
    C = ops.spgemm(ctx, state["A"], state["A"], rowptr_bits=ptr)
    ops.mcl_inflate(ctx, C, case["power"])
    return {"expanded": _out(C), "pruned": _out(ops.mcl_prune(ctx, C, case["tol"], rowptr_bits=ptr))}


# ---------------------------------------------------------------- work

def _nbytes(*objs):
    total = 0
    for o in objs:
        if isinstance(o, DeviceCSR):
            total += _nbytes(o.rowptr, o.col[:o.nnz], o.val[:o.nnz])
        elif isinstance(o, torch.Tensor):
            total += o.numel() * o.element_size()
        elif isinstance(o, dict):
            total += _nbytes(*o.values())
        elif isinstance(o, (list, tuple)):
            total += _nbytes(*o)
    return total


def work(case):
    """Every operand read once and every result written once; two operations
    per product of a multiplication, one per entry of a merge or an update."""
    st = prepare(case, 1)
    out, kind, ctx = run(st), case["kind"], st["ctx"]
    if kind == "batch":
        st["batch"].run()
        ins = [M for pair in st["pairs"] for M in pair]
        flops = 2 * sum(c[0] for c in st["batch"].count())
    elif kind == "galerkin":
        ap = out["ap"]
        AP = DeviceCSR(st["A"].nrows, st["P"].ncols, ap["rowptr"], ap["col"], ap["val"], nnz=ap["col"].numel())
        ins = [st["A"], st["P"], st["R"], AP]
        flops = 2 * (ops.spgemm_count(ctx, st["A"], st["P"])[0] + ops.spgemm_count(ctx, st["R"], AP)[0])
    elif kind in ("spgemm", "plan", "mcl"):
        ins = [st["A"]]
        flops = 2 * ops.spgemm_count(ctx, st["A"], st["A"])[0]
        if kind == "mcl":  # the inflation reads the product again, the pruning the inflated values
            ins.append([out["expanded"], out["expanded"]["val"]])
            flops += 3 * out["expanded"]["val"].numel()
    elif kind == "mma":
        ins = [st["A"], st["B"], st["C"]]
        flops = 2 * ops.spgemm_count(ctx, st["A"], st["B"])[0] + st["C"].nnz
    elif kind == "exchange":
        ins = [st["A"].rowptr, st["A"].col, st["A_csc"], st["B"], out["a"]]
        flops = st["A"].nnz
    elif kind == "coo":
        ins, flops = [st["row"], st["col"], st["val"]], st["val"].numel()
    else:
        ins = [st["A"]] + ([st["B"]] if kind == "spadd" else [])
        flops = sum(M.nnz for M in ins)
    return {"bytes": _nbytes(ins, out), "flops": flops}


# ---------------------------------------------------------------- 64-bit values

def _coo64(M):
    lens = M.rowptr[1:].long() - M.rowptr[:-1].long()
    row = torch.arange(M.nrows, device=_DEV).repeat_interleave(lens)
    return row, M.col[:M.nnz].long(), M.val[:M.nnz].double()


def _product64(A, B, addend=None, chunk=150_000_000):
    """Sorted keys and FP64 values of A·B (+ addend): all products of a chunk
    of rows expanded, sorted by (row, column) and summed."""
    ra, ca, va = _coo64(A)
    bp = B.rowptr.long()
    vb = B.val[:B.nnz].double()
    blen = (bp[1:] - bp[:-1])[ca]
    csum = torch.zeros(ra.numel() + 1, dtype=torch.int64, device=_DEV)
    csum[1:] = torch.cumsum(blen, 0)
    ap = A.rowptr.long()
    done = csum[ap]  # products before each row
    keys, vals, r0 = [], [], 0
    while r0 < A.nrows:
        r1 = int(torch.searchsorted(done, done[r0] + chunk, right=True)) - 1
        r1 = min(A.nrows, max(r1, r0 + 1))
        e0, e1 = int(ap[r0]), int(ap[r1])
        ent = torch.arange(e0, e1, device=_DEV).repeat_interleave(blen[e0:e1])
        q = bp[ca[ent]] + torch.arange(ent.numel(), device=_DEV) - (csum[ent] - csum[e0])
        k, v = ra[ent] * B.ncols + B.col[q].long(), va[ent] * vb[q]
        del ent, q
        if addend is not None:
            rc, cc, vc = _coo64(addend)
            m = (rc >= r0) & (rc < r1)
            k, v = torch.cat([k, (rc * B.ncols + cc)[m]]), torch.cat([v, vc[m]])
        k, order = torch.sort(k)
        v = v[order]
        del order
        k, cnt = torch.unique_consecutive(k, return_counts=True)
        keys.append(k)
        vals.append(torch.segment_reduce(v, "sum", lengths=cnt))
        r0 = r1
    return torch.cat(keys), torch.cat(vals)


def _vals(v):
    return {"rowptr": None, "col": None, "val": v}


def exact(case, seed):
    st, kind = _inputs(case, seed), case["kind"]
    if kind == "spgemm":
        return _vals(_product64(st["A"], st["A"])[1])
    if kind == "plan":
        A = st["A"]
        A.val = _uniform_values(_gen(seed + 1), A.nnz, A.val.dtype)
        return _vals(_product64(A, A)[1])
    if kind == "galerkin":
        R, A, P = st["R"], st["A"], st["P"]
        keys, v = _product64(A, P)
        AP = _csr(keys, A.nrows, P.ncols, v, 64)
        return {"ap": _vals(v), "rap": _vals(_product64(R, AP)[1])}
    if kind == "batch":
        return [_vals(_product64(A, B)[1]) for A, B in st["pairs"]]
    if kind == "mma":
        return _vals(_product64(st["A"], st["B"], st["C"])[1])
    if kind == "spadd":
        (ra, ca, va), (rb, cb, vb) = _coo64(st["A"]), _coo64(st["B"])
        k, order = torch.sort(torch.cat([ra * st["A"].ncols + ca, rb * st["A"].ncols + cb]))
        _, cnt = torch.unique_consecutive(k, return_counts=True)
        return _vals(torch.segment_reduce(torch.cat([va, vb])[order], "sum", lengths=cnt))
    if kind == "exchange":
        A, B = st["A"], st["B"]
        (_, ca, va), (rb, _, vb) = _coo64(A), _coo64(B)
        used = torch.zeros(A.ncols, dtype=torch.bool, device=_DEV)
        full = torch.zeros(A.ncols, dtype=torch.bool, device=_DEV)
        used[ca] = True
        full[rb] = True
        keep = used & full
        return {"mask": None, "mults": None, "upper": None, "a": _vals(va[keep[ca]]), "b": _vals(vb[keep[rb]])}
    if kind == "coo":
        maj, mnr = (st["row"], st["col"]) if case["major"] == "rows" else (st["col"], st["row"])
        order = torch.argsort(maj.long() * st["n"] + mnr.long(), stable=True)
        return _vals(st["val"].double()[order])
    if kind == "transpose":
        r, c, v = _coo64(st["A"])
        return _vals(v[torch.argsort(c * st["A"].nrows + r, stable=True)])
    A = st["A"]
    keys, v = _product64(A, A)
    row = torch.div(keys, A.ncols, rounding_mode="floor")
    v = v ** case["power"]
    lens = torch.bincount(row, minlength=A.nrows)
    v = v / torch.segment_reduce(v, "sum", lengths=lens)[row]
    return {"expanded": _vals(v), "pruned": _vals(v[v.abs() > case["tol"]])}
