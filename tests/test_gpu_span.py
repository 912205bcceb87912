"""GPU: rows whose column span lies in a shared-memory bitmap — sizes at the
edges of its words, units, tiles and register-held products, both phases."""
import numpy as np
import pytest

import oracle
from helpers import TOL32, TOL64, check_product, check_sum
from trident_b200 import ops
from trident_b200._lib import TSPG_F_ACC_FUSE
from trident_b200.csr import HostCSR

pytestmark = pytest.mark.gpu


def _rows(lens, n, rng, dup=False, sort=True):
    rp = np.zeros(len(lens) + 1, np.int64)
    rp[1:] = np.cumsum(lens)
    cols = [rng.choice(n, size=k, replace=dup) for k in lens]
    cols = np.concatenate([np.sort(c) if sort else c for c in cols]).astype(np.int32)
    return HostCSR(len(lens), n, rp, cols, rng.uniform(-1, 1, cols.size))


def _pair(n, dup, seed):
    """A rows of 1 ... 1100 entries (staging rounds of 128 / 256 / 512) over B
    rows of 0, 1, 31 ... 33, 127 ... 129 and 400 entries; the first and last
    columns are hit."""
    rng = np.random.default_rng(seed)
    blens = np.minimum(rng.choice([0, 1, 1, 2, 5, 31, 32, 33, 127, 128, 129, 400], size=1200), n)
    blens[:3] = [1, 2, 1]
    B = _rows(blens, n, rng, dup=dup, sort=not dup)
    B.col[0], B.col[-1] = n - 1, 0
    alens = [0, 1, 2, 3, 7, 15, 16, 17, 31, 32, 33, 64, 127, 128, 129, 255, 256, 257, 511, 513, 1100] * 3
    return _rows(alens, 1200, rng), B


@pytest.mark.parametrize("dup", [False, True])
@pytest.mark.parametrize("n", [700, 1023, 1024, 1025, 4097, 33000, 150000])
def test_span_rows_match_the_oracle(ctx, n, dup):
    A, B = _pair(n, dup, seed=n)
    dA, dB = A.to_device(rowptr_bits=32), B.to_device(rowptr_bits=32)
    check_product(ops.spgemm(ctx, dA, dB), A, B, tol=TOL64)
    plan = ops.Plan(ctx, dA, dB)  # new values of the same pattern
    A2 = HostCSR(A.nrows, A.ncols, A.rowptr, A.col, A.val[::-1].copy())
    check_product(plan.numeric(A2.to_device(rowptr_bits=32), dB), A2, B)
    plan.close()


@pytest.mark.parametrize("n", [1025, 33000])
def test_span_rows_fp32_wide_offsets(ctx, n):
    A, B = _pair(n, False, seed=5 * n)
    A, B = (HostCSR(M.nrows, M.ncols, M.rowptr, M.col, M.val.astype(np.float32).astype(np.float64))
            for M in (A, B))
    check_product(ops.spgemm(ctx, A.to_device(rowptr_bits=64, val_bits=32), B.to_device(rowptr_bits=64, val_bits=32)),
                  A, B, tol=TOL32)


@pytest.mark.parametrize("n", [64, 65, 16384, 16385, 32704, 32767, 32768, 32769])
def test_warp_rows_over_the_whole_span(ctx, n):
    # rows of 65 ... 190 products; first and last column, and columns on both
    # sides of every unit boundary up to the slice's last unit
    rng = np.random.default_rng(n)
    edges = np.unique(np.clip(np.concatenate([np.arange(64, n + 1, 64), np.arange(63, n + 1, 64), [0, n - 1]]), 0, n - 1))
    lens = np.minimum(rng.integers(4, 24, size=600), edges.size)
    rp = np.zeros(601, np.int64)
    rp[1:] = np.cumsum(lens)
    col = np.concatenate([np.sort(rng.choice(edges, size=k, replace=False)) for k in lens]).astype(np.int32)
    B = HostCSR(600, n, rp, col, rng.uniform(-1, 1, col.size))
    A = _rows(rng.integers(4, 9, size=3000), 600, rng)
    dA, dB = A.to_device(rowptr_bits=32), B.to_device(rowptr_bits=32)
    check_product(ops.spgemm(ctx, dA, dB), A, B, tol=TOL64)


def test_span_rows_with_an_addend(ctx):
    A, B = _pair(4097, False, seed=11)
    E = _rows(np.tile([0, 300, 1500], 21), 4097, np.random.default_rng(3))
    C = ops.sp_mma(ctx, A.to_device(), B.to_device(), E.to_device(), flags=TSPG_F_ACC_FUSE)
    rp, cj, cx, _ = oracle.spgemm(A, B)
    check_sum(C, HostCSR(A.nrows, B.ncols, rp, cj, cx), E)


def test_dense_rows_two_ctas_per_sm():
    # more DENSE rows than 16 per SM, their outputs on both sides of the slots
    # that fit shared memory
    c = ops.Context(0)
    c.set_tuning({"num_lim": [256, 1024, 2048, 2048]})
    rng = np.random.default_rng(7)
    B = _rows(np.full(600, 900), 60000, rng)
    A = _rows(rng.choice([5, 40], size=2600), 600, rng)
    check_product(ops.spgemm(c, A.to_device(rowptr_bits=64), B.to_device(rowptr_bits=64)), A, B)
    c.close()


@pytest.mark.parametrize("val_bits", [64, 32])
def test_kept_bitmaps(val_bits):
    # a one-shot product of 65,536 rows or more keeps the bitmaps of its heavy
    # DENSE rows for the numeric phase: 1,500 of them (f ~36,000, c ~27,000)
    # among rows of 3 products and rows on both sides of the register-held ones
    c = ops.Context(0)
    c.set_tuning({"sym_lim": [512, 2048, 4096, 4096], "num_lim": [256, 1024, 2048, 2048]})
    rng = np.random.default_rng(9)
    B = _rows(np.concatenate([np.full(600, 900), np.full(100, 3)]), 60000, rng)
    lens = np.ones(66000, np.int64)
    heavy = rng.choice(66000, size=1800, replace=False)
    lens[heavy] = np.where(np.arange(1800) < 1500, 40, 9)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(600, size=k, replace=False)) if k > 1 else [600 + i % 100]
                          for i, k in enumerate(lens)]).astype(np.int32)
    A = HostCSR(66000, 700, rp, col, rng.uniform(-1, 1, col.size))
    if val_bits == 32:
        A, B = (HostCSR(M.nrows, M.ncols, M.rowptr, M.col, M.val.astype(np.float32).astype(np.float64))
                for M in (A, B))
    dA, dB = (M.to_device(rowptr_bits=64, val_bits=val_bits) for M in (A, B))
    check_product(ops.spgemm(c, dA, dB), A, B, tol=TOL64 if val_bits == 64 else TOL32)
    c.close()


def test_overlapped_kernels_of_a_large_batch_and_product(ctx):
    # rows of every class in one product, launched to overlap, several times
    rng = np.random.default_rng(21)
    B = _rows(rng.choice([1, 8, 60, 400], size=3000), 30000, rng)
    A = _rows(rng.choice([1, 3, 10, 40, 150], size=4000), 3000, rng)
    dA, dB = A.to_device(), B.to_device()
    for _ in range(5):
        C = ops.spgemm(ctx, dA, dB)
    check_product(C, A, B)
    b = ops.Batch(ctx)
    for _ in range(2):
        b.add(dA, dB)
    for _ in range(3):
        b.run()
    for i in range(2):
        check_product(b.result(i), A, B)
    b.close()


@pytest.mark.parametrize("val_bits", [64, 32])
def test_lane_rows(val_bits):
    # numeric rows of 1 ... 32 outputs, 32 to a warp (even rows of 30 products
    # first, then uneven ones that a warp takes one by one), 33 past the slots;
    # a plan run twice, and a batch whose rows alternate between two products
    rng = np.random.default_rng(5)
    B = _rows(np.concatenate([np.full(400, 5), rng.choice([0, 1, 3, 33, 200], size=400)]), 50000, rng)
    even = [np.sort(rng.choice(400, size=6, replace=False)) for _ in range(40000)]
    mixed = [np.sort(rng.choice(800, size=k, replace=False)) for k in rng.choice([1, 2, 6, 7], size=20000)]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in even + mixed])]).astype(np.int64)
    A = HostCSR(60000, 800, rp, np.concatenate(even + mixed).astype(np.int32), rng.uniform(-1, 1, rp[-1]))
    tol = TOL64 if val_bits == 64 else TOL32
    if val_bits == 32:
        A, B = (HostCSR(M.nrows, M.ncols, M.rowptr, M.col, M.val.astype(np.float32).astype(np.float64))
                for M in (A, B))
    c = ops.Context(0)
    dA, dB = A.to_device(val_bits=val_bits), B.to_device(val_bits=val_bits)
    plan = ops.Plan(c, dA, dB)
    for _ in range(2):
        check_product(plan.numeric(dA, dB), A, B, tol=tol)
    plan.close()
    b = ops.Batch(c)
    b.add(dA, dB)
    b.add(dA, dB)
    b.run()
    for i in range(2):
        check_product(b.result(i), A, B, tol=tol)
    b.close()
    c.close()


@pytest.mark.parametrize("m", [3000, 66000])
def test_short_rows_of_many_a_entries(ctx, m):
    # A rows of 1 ... 700 entries whose B rows are mostly empty: few products,
    # by lanes where the rows of a warp are alike, else one by one
    rng = np.random.default_rng(m)
    bl = np.zeros(2000, np.int64)
    bl[rng.choice(2000, size=60, replace=False)] = rng.choice([1, 2, 3], size=60)
    B = _rows(bl, 9000, rng)
    lens = np.full(m, 4)
    lens[: m // 3] = rng.choice([1, 31, 32, 33, 64], size=m // 3)
    at = rng.choice(m, size=200, replace=False)
    lens[at] = rng.choice([255, 256, 257, 300, 700], size=200)
    lens[m // 2: m // 2 + 64] = 700  # whole warps of them
    A = _rows(lens, 2000, rng)
    dA, dB = A.to_device(), B.to_device()
    check_product(ops.spgemm(ctx, dA, dB), A, B)
    plan = ops.Plan(ctx, dA, dB)
    check_product(plan.numeric(dA, dB), A, B)
    plan.close()
    b = ops.Batch(ctx)
    b.add(dA, dB)
    b.run()
    check_product(b.result(0), A, B)
    b.close()


def _common_columns(m, groups, na, cols, val_bits, rng):
    """A (m rows of `na` entries) and B such that row i's products meet `na`
    times in each of `cols` columns, and the exact values (m, cols)."""
    B = HostCSR(groups * na, groups * cols, np.arange(groups * na + 1, dtype=np.int64) * cols,
                (np.repeat(np.arange(groups), na * cols) * cols + np.tile(np.arange(cols), groups * na)).astype(np.int32),
                rng.uniform(0.1, 1, groups * na * cols))
    g = np.arange(m) % groups
    A = HostCSR(m, groups * na, np.arange(m + 1, dtype=np.int64) * na,
                (g[:, None] * na + np.arange(na)).ravel().astype(np.int32), rng.uniform(-1, 1, m * na))
    if val_bits == 32:
        for M in (A, B):
            M.val = M.val.astype(np.float32).astype(np.float64)
    a = A.val.reshape(m, na).astype(np.longdouble)
    b = B.val.reshape(groups, na, cols).astype(np.longdouble)
    exact = np.zeros((m, cols), np.longdouble)
    for t in range(na):
        exact += a[:, t, None] * b[g, t, :]
    return A, B, exact


@pytest.mark.parametrize("val_bits", [64, 32])
@pytest.mark.parametrize("m,cols", [(66000, 12), (66000, 27)])
def test_lane_rows_lose_nothing_to_their_order(val_bits, m, cols):
    # 100 products an output by one lane.  Rounding each result alone, correctly,
    # is an error of at most u in the norm; a running sum of these is 4 u off.
    A, B, exact = _common_columns(m, 50, 100, cols, val_bits, np.random.default_rng(cols))
    c = ops.Context(0)
    dA, dB = A.to_device(val_bits=val_bits), B.to_device(val_bits=val_bits)
    u = 2.0 ** -53 if val_bits == 64 else 2.0 ** -24
    plan = ops.Plan(c, dA, dB)
    for C in (ops.spgemm(c, dA, dB), plan.numeric(dA, dB)):
        H = C.to_host()
        np.testing.assert_array_equal(H.rowptr, np.arange(m + 1) * cols)
        d = H.val.reshape(m, cols).astype(np.longdouble) - exact
        assert float(np.sqrt((d * d).sum() / (exact * exact).sum())) <= u
    plan.close()
    c.close()


def test_lane_rows_at_the_ends_of_the_number_range():
    # sums that overflow, infinite and NaN operands, values whose rounding
    # errors lie below the smallest number: as plain sums give them
    m, na = 5000, 4
    A, B, _ = _common_columns(m, 50, na, 6, 64, np.random.default_rng(1))
    a, b = A.val.reshape(m, na), B.val.reshape(50, na, 6)
    b[:] = 1.0
    a[0::8] = 1e308
    a[1::8] = [np.inf, 1, 2, 3]
    a[2::8] = [1, np.inf, -np.inf, 1]
    a[3::8] = [1, np.nan, 2, 3]
    a[4::8] = 1e-310
    a[5::8] = [1e300, 1.0, -1e300, 1.0]
    a[6::8] = -0.0
    a[7::8] = [1e308, 1e308, -1e308, -1e308]
    A.val, B.val = a.ravel(), b.ravel()
    c = ops.Context(0)
    dA, dB = A.to_device(), B.to_device()
    plan = ops.Plan(c, dA, dB)
    got = plan.numeric(dA, dB).to_host().val.reshape(m, 6)
    assert np.all(got[0::8] == np.inf) and np.all(got[1::8] == np.inf)
    assert np.all(np.isnan(got[2::8])) and np.all(np.isnan(got[3::8]))
    assert np.all(got[4::8] == 4e-310)
    assert np.all(np.isin(got[5::8], [0.0, 1.0, 2.0]))
    assert np.all(got[6::8] == 0.0)
    assert not np.any(np.isfinite(got[7::8]) & (got[7::8] != 0.0))
    plan.close()
    c.close()


def test_plan_whose_b_rows_change_their_order(ctx):
    # the same pattern, B's rows in another order at each call: a form that takes
    # a row's span from the ends of its B rows must not be kept from a call before
    n, rng = 40000, np.random.default_rng(17)
    col = np.sort(np.clip(np.arange(n), 24, n - 25)[:, None] + np.arange(-8, 9) * 3, axis=1)
    rp = np.arange(n + 1, dtype=np.int64) * 17
    A = HostCSR(n, n, rp, col.ravel().astype(np.int32), rng.uniform(-1, 1, col.size))
    dA = A.to_device()
    plan = ops.Plan(ctx, dA, dA)
    check_product(plan.numeric(dA, dA), A, A)
    for _ in range(2):
        o = np.argsort(rng.random(col.shape), axis=1)
        U = HostCSR(n, n, rp, np.take_along_axis(col, o, 1).ravel().astype(np.int32),
                    np.take_along_axis(A.val.reshape(n, 17), o, 1).ravel())
        check_product(plan.numeric(dA, U.to_device()), A, A)
        check_product(plan.numeric(U.to_device(), dA), A, A)
        check_product(plan.numeric(dA, dA), A, A)
    plan.close()


def _heavy_product(rng):
    """A product that keeps bitmaps: 66,000 rows, 1,500 of them DENSE."""
    B = _rows(np.concatenate([np.full(600, 900), np.full(100, 3)]), 60000, rng)
    lens = np.ones(66000, np.int64)
    lens[rng.choice(66000, size=1500, replace=False)] = 40
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    col = np.concatenate([np.sort(rng.choice(600, size=k, replace=False)) if k > 1 else [600 + i % 100]
                          for i, k in enumerate(lens)]).astype(np.int32)
    return HostCSR(66000, 700, rp, col, rng.uniform(-1, 1, col.size)), B


HEAVY = {"sym_lim": [512, 2048, 4096, 4096], "num_lim": [256, 1024, 2048, 2048]}


@pytest.mark.parametrize("refuse", [(0,), (1,), (1, 2)])
def test_output_refused_beside_kept_bitmaps(refuse):
    # the allocator refuses a request: the pool's free blocks, then the bitmaps
    # are given back, and only what is missing is asked for again
    import ctypes as C

    import torch

    from trident_b200._lib import ALLOC_FN, TspgCsrOut, check, lib
    from trident_b200.csr import DeviceCSR
    A, B = _heavy_product(np.random.default_rng(9))
    dA, dB = A.to_device(rowptr_bits=64), B.to_device(rowptr_bits=64)
    c = ops.Context(0)
    c.set_tuning(HEAVY)
    asked, blocks = [], {}

    def alloc(user, nbytes, stream):
        asked.append(nbytes)
        if len(asked) - 1 in refuse:
            return None
        t = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        blocks[t.data_ptr()] = t
        return t.data_ptr()

    rp = torch.empty(A.nrows + 1, dtype=torch.int64, device="cuda")
    o = TspgCsrOut()
    o.nrows, o.ncols, o.rowptr, o.rowptr_bits, o.val_bits = A.nrows, B.ncols, rp.data_ptr(), 64, 64
    o.alloc = ALLOC_FN(alloc)
    a, b = dA.abi(), dB.abi()
    check(lib.tspg_spgemm(c.h, torch.cuda.current_stream().cuda_stream, C.byref(a), C.byref(b), C.byref(o), 0),
          "tspg_spgemm")
    nnz = int(o.nnz)
    assert asked == [k * nnz for k in {(0,): [4, 4, 8], (1,): [4, 8, 8], (1, 2): [4, 8, 8, 8]}[refuse]]
    check_product(DeviceCSR(A.nrows, B.ncols, rp, blocks[o.col].view(torch.int32), blocks[o.val].view(torch.float64),
                            nnz=nnz), A, B)
    c.close()


@pytest.mark.parametrize("n,keeps", [(60_000, True), (1_000_000, False)])
def test_bitmaps_are_kept_only_where_they_are_filled(n, keeps):
    # at 1M columns the symbolic DENSE rows are no span rows: no room for bitmaps
    # (125 KB a row) is taken.  1,500 rows' bitmaps are the larger part at 60,000.
    A, B = _heavy_product(np.random.default_rng(9))
    B = HostCSR(B.nrows, n, B.rowptr, (B.col.astype(np.int64) * (n // 60_000)).astype(np.int32), B.val)
    c = ops.Context(0)
    c.set_tuning(HEAVY)
    C = ops.spgemm(c, A.to_device(rowptr_bits=64), B.to_device(rowptr_bits=64))
    if n == 60_000:
        check_product(C, A, B)
    bits = 1500 * ((n + 1023) // 1024) * 128
    rows = 66_000 * (28 + 4) + 12 * 32 * 66_000  # row arrays, slots, one-pass scratch
    assert (c.mem()[1] >= bits) == keeps and c.mem()[1] < (bits if keeps else 0) + rows + (1 << 20)
    c.close()


def test_budget_goes_to_the_cursors_before_the_kept_bitmaps():
    # one A row longer than the cursors in shared memory: its buffer comes after
    # the bitmaps were taken, and a budget that holds either must do
    rng = np.random.default_rng(19)
    A, B = _heavy_product(rng)
    k = 8200
    B = HostCSR(700 + k, 60000, np.concatenate([B.rowptr, np.full(k, B.rowptr[-1])]), B.col, B.val)
    lens = np.diff(A.rowptr)
    lens[-1] = k
    A = HostCSR(66000, 700 + k, np.concatenate([[0], np.cumsum(lens)]).astype(np.int64),
                np.concatenate([A.col[:A.rowptr[-2]], np.arange(700, 700 + k, dtype=np.int32)]),
                rng.uniform(-1, 1, int(lens.sum())))
    dA, dB = A.to_device(rowptr_bits=64), B.to_device(rowptr_bits=64)
    c = ops.Context(0)
    c.set_tuning(HEAVY)
    check_product(ops.spgemm(c, dA, dB), A, B)
    need, cursors = c.mem()[1], 2 * 148 * k * 4
    bits, slots = 1500 * ((60000 + 1023) // 1024) * 128, -(-66000 * 4 // 256) * 256
    assert need > bits + cursors
    for budget in (need, need - 512, need - cursors, need - cursors - 512, need - bits - 256, need - bits - slots):
        t = ops.Context(0, budget)
        t.set_tuning(HEAVY)
        check_product(ops.spgemm(t, dA, dB), A, B)
        t.close()
    c.close()


@pytest.mark.parametrize("na", [23, 24])
@pytest.mark.parametrize("cols", [28, 32, 33, 48, 50, 64, 98, 99, 128, 190])
def test_warp_rows_of_many_products_an_output(na, cols):
    # both sides of the rule between the hash and the span form of a warp row
    from test_gpu_tuning import _alike_rows
    A, B = _alike_rows(4500, na, cols)
    c = ops.Context(0)
    plan = ops.Plan(c, A.to_device(), B.to_device())
    check_product(plan.numeric(A.to_device(), B.to_device()), A, B)
    plan.close()
    c.close()


@pytest.mark.parametrize("cols", [26, 27, 28, 31, 32, 33, 200])
@pytest.mark.parametrize("late", [False, True])
def test_one_pass_rows_at_the_lanes_and_the_warps_bound(cols, late):
    # one-pass rows that a lane, a warp or neither holds, their columns in every B
    # row or spread over them; counted at once (table and products that fit) or
    # later; every fourth stretch of rows is short, so warps change their mind
    m, groups, na, rng = 66000, 40, 12, np.random.default_rng(cols)
    width = 200
    B_rows, per = [], -(-cols // na) + 3
    for g in range(groups):
        mine = np.sort(rng.choice(width, size=cols if g % 4 else 9, replace=False))
        for t in range(na):
            part = mine if not late or g % 4 == 0 else np.unique(np.r_[mine[:3], np.roll(mine, -t * (cols // na + 1))[:per]])
            B_rows.append(g * width + np.sort(part))
    rp = np.concatenate([[0], np.cumsum([len(r) for r in B_rows])]).astype(np.int64)
    B = HostCSR(groups * na, groups * width, rp, np.concatenate(B_rows).astype(np.int32), rng.uniform(-1, 1, rp[-1]))
    g = np.arange(m) * groups // m
    A = HostCSR(m, groups * na, np.arange(m + 1, dtype=np.int64) * na,
                (g[:, None] * na + np.arange(na)).ravel().astype(np.int32), rng.uniform(-1, 1, m * na))
    c = ops.Context(0)
    check_product(ops.spgemm(c, A.to_device(), B.to_device()), A, B)
    c.close()



@pytest.mark.parametrize("na", [23, 24])
@pytest.mark.parametrize("cols,rows", [(300, 888), (1200, 444), (3000, 148)])
@pytest.mark.parametrize("less", [0, 1])
def test_classes_of_many_products_an_output(na, cols, rows, less):
    # 128-, 256- and 512-thread rows on both sides of the rule between the forms
    from test_gpu_tuning import _alike_rows
    A, B = _alike_rows(rows - less, na, cols, groups=10)
    c = ops.Context(0)
    plan = ops.Plan(c, A.to_device(), B.to_device())
    for _ in range(2):
        check_product(plan.numeric(A.to_device(), B.to_device()), A, B)
    plan.close()
    c.close()
