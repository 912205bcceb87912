"""GPU: the row binning changes speed only — results equal the oracle's under
non-default tunings, invalid tunings are refused, batches re-capture."""
import pytest

from helpers import check_product, random_csr
from trident_b200 import ops, tune, workloads
from trident_b200._lib import TSPG_EINVAL, TspgError

pytestmark = pytest.mark.gpu

TUNINGS = [
    {"sym_lim": [128, 1024, 2048, 8192], "num_lim": [128, 512, 1024, 4096], "hash_load": 4, "dense_win_log2": 17, "dense_win_fill_log2": 4, "dense_win_cluster": 0},
    {"sym_lim": [512, 512, 512, 512], "num_lim": [256, 256, 256, 256], "hash_load": 2, "dense_win_log2": 0, "dense_win_fill_log2": 4, "dense_win_cluster": 0},
    {"sym_lim": [1, 1, 1, 1], "num_lim": [1, 1, 1, 1], "hash_load": 8, "dense_win_log2": 10, "dense_win_fill_log2": 12, "dense_win_cluster": 2},
]


@pytest.fixture
def tctx():
    c = ops.Context(0)
    yield c
    c.close()


def test_invalid_tuning_refused(tctx):
    for bad in ({"num_lim": [1024, 1024, 2048, 8192]}, {"sym_lim": [512, 256, 4096, 24576]},
                {"hash_load": 3}, {"num_lim": [0, 1024, 2048, 8192]}, {"dense_win_log2": 9}):
        with pytest.raises(TspgError) as e:
            tctx.set_tuning(bad)
        assert e.value.status == TSPG_EINVAL
    assert tctx.get_tuning() == tune.default_tuning()


@pytest.mark.parametrize("t", TUNINGS)
def test_results_do_not_depend_on_tuning(tctx, t):
    tctx.set_tuning(t)
    assert tctx.get_tuning() == t
    R = workloads.rmat(scale=12, edge_factor=16, seed=3)
    check_product(ops.spgemm(tctx, R.to_device(), R.to_device()), R, R)
    A = random_csr(3000, 2500, per_row=14, seed=8)
    B = random_csr(2500, 4000, per_row=9, seed=9)
    check_product(ops.spgemm(tctx, A.to_device(), B.to_device()), A, B)


def test_batch_recaptures_on_tuning_change(tctx):
    specs = workloads.batched_specs(count=6, seed=9, rows_lo=300, rows_hi=8000)
    hosts, keep = [], []
    b = ops.Batch(tctx)
    for spec in specs:
        A, B = workloads.batched_product(spec)
        dA, dB = A.to_device(), B.to_device()
        hosts.append((A, B))
        keep.append((dA, dB))
        b.add(dA, dB)
    n0 = b.run()
    tctx.set_tuning(TUNINGS[0])
    assert b.run() == n0
    for i, (A, B) in enumerate(hosts):
        check_product(b.result(i), A, B)
    b.close()


@pytest.mark.parametrize("t", TUNINGS[1:])
def test_batch_results_do_not_depend_on_tuning(tctx, t):
    """Products of different shapes in one batch, with most rows (or all) in
    the DENSE forms: the rank-form kernel takes rows of several products,
    each with its own column count."""
    tctx.set_tuning(t)
    specs = workloads.batched_specs(count=5, seed=21, rows_lo=200, rows_hi=5000)
    hosts, keep = [], []
    b = ops.Batch(tctx)
    for spec in specs:
        A, B = workloads.batched_product(spec)
        dA, dB = A.to_device(), B.to_device()
        hosts.append((A, B))
        keep.append((dA, dB))
        b.add(dA, dB)
    b.run()
    for i, (A, B) in enumerate(hosts):
        check_product(b.result(i), A, B)
    b.close()


def test_plan_numeric_with_dense_rows(tctx):
    """The plan API's numeric re-runs (new values, same structure) with every
    row above 256 outputs in the DENSE forms."""
    tctx.set_tuning(TUNINGS[1])
    R = workloads.rmat(scale=12, edge_factor=16, seed=5)
    dR = R.to_device()
    plan = ops.Plan(tctx, dR, dR)
    try:
        check_product(plan.numeric(dR, dR), R, R)
        R.val[:] = R.val * -0.5 + 0.25
        dR2 = R.to_device()
        check_product(plan.numeric(dR2, dR2), R, R)
    finally:
        plan.close()


def _poisoned_numeric(plan, A, B):
    """The numeric call of a plan into arrays filled with values no result has."""
    import ctypes as C

    import torch

    from trident_b200._lib import TspgCsrOut, check, lib
    from trident_b200.csr import DeviceCSR
    m, n = plan.shape
    rp = torch.full((m + 1,), -3, dtype=torch.int64, device="cuda")
    col = torch.full((plan.c_nnz,), -7, dtype=torch.int32, device="cuda")
    val = torch.full((plan.c_nnz,), float("nan"), dtype=torch.float64, device="cuda")
    o = TspgCsrOut()
    o.nrows, o.ncols, o.rowptr, o.rowptr_bits, o.val_bits = m, n, rp.data_ptr(), 64, 64
    o.col, o.val, o.capacity = col.data_ptr(), val.data_ptr(), plan.c_nnz
    a, b = A.abi(), B.abi()
    check(lib.tspg_spgemm_numeric(plan.ctx.h, torch.cuda.current_stream().cuda_stream, plan.h, C.byref(a),
                                  C.byref(b), C.byref(o)), "tspg_spgemm_numeric")
    return DeviceCSR(m, n, rp, col, val, nnz=plan.c_nnz)


NARROW = {"num_lim": [64, 256, 512, 2048]}
WINDOW = {"num_lim": [64, 256, 512, 2048], "dense_win_log2": 10, "dense_win_fill_log2": 12}
PAIRS = [({}, NARROW), (NARROW, {}), ({}, WINDOW), (WINDOW, {}), (WINDOW, dict(WINDOW, dense_win_cluster=2)),
         (dict(WINDOW, dense_win_cluster=2), {})]


@pytest.mark.parametrize("made,now", PAIRS)
def test_plan_keeps_the_tuning_it_was_made_with(tctx, made, now):
    # rows of every class; a tuning set after the symbolic call holds for later
    # calls, the plan's rows were classed with the one before it
    import numpy as np

    from trident_b200.csr import HostCSR
    rng = np.random.default_rng(31)

    def rows(lens, n):
        rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
        col = np.concatenate([np.sort(rng.choice(n, size=k, replace=False)) for k in lens]).astype(np.int32)
        return HostCSR(len(lens), n, rp, col, rng.uniform(-1, 1, col.size))

    B = rows(np.full(200, 400), 30000)
    A = rows(rng.choice([1, 2, 4, 8, 12, 20, 60], size=300), 200)
    dA, dB = A.to_device(), B.to_device()
    tctx.set_tuning(dict(tune.default_tuning(), **made))
    plan = ops.Plan(tctx, dA, dB)
    tctx.set_tuning(dict(tune.default_tuning(), **now))
    for _ in range(2):
        check_product(_poisoned_numeric(plan, dA, dB), A, B)
    plan.close()
    check_product(ops.spgemm(tctx, dA, dB), A, B)


@pytest.mark.parametrize("bounds,cls", [([256, 1024, 2048, 8192], 5), ([255, 1024, 2048, 8192], 6),
                                        ([200, 1024, 2048, 8192], 6), ([199, 1024, 2048, 8192], 5)])
def test_bounds_of_the_caller_hold(tctx, bounds, cls):
    # rows of 200 outputs: warp rows (class 6) up to the caller's bound; at the
    # default the library picks 192 for this width (class 5, 128 threads)
    import ctypes as C

    import numpy as np

    from trident_b200._lib import check, lib
    from trident_b200.csr import HostCSR
    rng = np.random.default_rng(2)
    col = np.concatenate([np.sort(rng.choice(3000, size=100, replace=False)) for _ in range(40)]).astype(np.int32)
    for i in range(0, 40, 2):  # rows 2i and 2i + 1 share no column
        both = np.sort(rng.choice(3000, size=200, replace=False)).astype(np.int32)
        col[i * 100:(i + 1) * 100], col[(i + 1) * 100:(i + 2) * 100] = both[::2], both[1::2]
    B = HostCSR(40, 3000, np.arange(41, dtype=np.int64) * 100, col, rng.uniform(-1, 1, col.size))
    acol = ((np.arange(2000) % 20)[:, None] * 2 + np.arange(2)).ravel().astype(np.int32)
    A = HostCSR(2000, 40, np.arange(2001, dtype=np.int64) * 2, acol, rng.uniform(-1, 1, 4000))
    tctx.set_tuning({"num_lim": bounds})
    check(lib.tspg_ctx_class_profile(tctx.h, 1), "tspg_ctx_class_profile")
    check_product(ops.spgemm(tctx, A.to_device(), B.to_device()), A, B)
    out = (C.c_uint64 * 64)()
    check(lib.tspg_ctx_class_cycles(tctx.h, out), "tspg_ctx_class_cycles")
    check(lib.tspg_ctx_class_profile(tctx.h, 0), "tspg_ctx_class_profile")
    assert [out[32 + 8 + c] for c in (5, 6)] == [2000 * (c == cls) for c in (5, 6)]


def _class_rows(ctx, run):
    """Numeric rows per class (DENSE0..2, G1024, G256, G128, G32, LANE) of a call."""
    import ctypes as C

    from trident_b200._lib import check, lib
    check(lib.tspg_ctx_class_profile(ctx.h, 1), "tspg_ctx_class_profile")
    run()
    out = (C.c_uint64 * 64)()
    check(lib.tspg_ctx_class_cycles(ctx.h, out), "tspg_ctx_class_cycles")
    check(lib.tspg_ctx_class_profile(ctx.h, 0), "tspg_ctx_class_profile")
    return [int(x) for x in out[40:48]]


def _alike_rows(m, na, cols, groups=20):
    """m rows of na * cols products on the same `cols` columns."""
    import numpy as np

    from trident_b200.csr import HostCSR
    rng = np.random.default_rng(m + na)
    base = np.sort(rng.choice(3 * cols, size=cols, replace=False))
    col = (np.repeat(np.arange(groups), na * cols) * 3 * cols + np.tile(base, groups * na)).astype(np.int32)
    B = HostCSR(groups * na, groups * 3 * cols, np.arange(groups * na + 1, dtype=np.int64) * cols, col,
                rng.uniform(-1, 1, col.size))
    g = np.arange(m) * groups // m
    A = HostCSR(m, groups * na, np.arange(m + 1, dtype=np.int64) * na,
                (g[:, None] * na + np.arange(na)).ravel().astype(np.int32), rng.uniform(-1, 1, m * na))
    return A, B


@pytest.mark.parametrize("m,na,cols,cls", [(3000, 24, 100, 5), (4000, 24, 100, 6), (1500, 25, 400, 4), (2000, 25, 400, 5),
                                           (300, 21, 100, 5), (300, 20, 100, 6)])
def test_wider_rows_only_where_the_others_do_not_cover_them(tctx, m, na, cols, cls):
    # rows of 2,400 and 10,000 products on 100 and 400 columns: as many as the chip
    # has warps (3,552) or 128-thread groups (1,776), or fewer
    A, B = _alike_rows(m, na, cols)
    rows = _class_rows(tctx, lambda: check_product(ops.spgemm(tctx, A.to_device(), B.to_device()), A, B))
    assert rows[cls] == m and sum(rows) == m


@pytest.mark.parametrize("m,na,cls", [(4000, 1, 7), (4000, 2, 6), (19_000, 9, 7), (19_000, 10, 6), (38_000, 60, 7)])
def test_lane_rows_want_warps_full_of_rows(tctx, m, na, cls):
    # rows of 20 products and more on 20 columns: by lanes while the rows to a
    # warp (of 2,368) make up for a lane's time a product
    A, B = _alike_rows(m, na, 20, groups=10)
    p = ops.Plan(tctx, A.to_device(), B.to_device())
    rows = _class_rows(tctx, lambda: check_product(p.numeric(A.to_device(), B.to_device()), A, B))
    p.close()
    assert rows[cls] == m and sum(rows) == m
