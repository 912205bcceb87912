"""GPU: the counting-sort passes behind the transpose and the COO builder, at
the edges of their digits (10 bits), tiles (2048 / 8192 entries) and windows."""
import numpy as np
import pytest
import torch

import oracle
from trident_b200 import ops
from trident_b200._lib import TSPG_COLS, TSPG_ROWS
from trident_b200.csr import DeviceCSR, HostCSR

pytestmark = pytest.mark.gpu


def _matrix(m, n, nnz, seed):
    """CSR with runs of empty rows and one long row; repeated columns too."""
    rng = np.random.default_rng(seed)
    lens = np.bincount(rng.choice(rng.integers(0, m, max(1, m // 3)), size=nnz - nnz // 3), minlength=m)
    lens[rng.integers(0, m)] += nnz // 3
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    return HostCSR(m, n, rp, rng.integers(0, n, nnz).astype(np.int32), rng.uniform(-1, 1, nnz))


@pytest.mark.parametrize("m,n,nnz", [(1, 1, 1), (1, 5, 33), (40, 1024, 2047), (40, 1025, 2048), (5000, 2, 2049),
                                     (70000, 1 << 20, 9000), (3, 1500000, 70), (900, 1 << 21, 400000),
                                     (200000, 30000, 2500000)])
@pytest.mark.parametrize("bits", [32, 64])
def test_transpose_is_stable(ctx, m, n, nnz, bits):
    M = _matrix(m, n, nnz, seed=nnz)
    T = ops.transpose(ctx, M.to_device(rowptr_bits=bits, val_bits=bits), rowptr_bits=bits).to_host()
    order = np.argsort(M.col, kind="stable")
    row = np.repeat(np.arange(m), np.diff(M.rowptr))
    np.testing.assert_array_equal(T.rowptr, np.concatenate([[0], np.cumsum(np.bincount(M.col, minlength=n))]))
    np.testing.assert_array_equal(T.col, row[order])
    np.testing.assert_array_equal(T.val, M.val.astype(np.float64 if bits == 64 else np.float32)[order])


def test_transpose_of_a_row_panel(ctx):
    # a view of rows [r0, r1): offsets that do not start at 0, the count an
    # upper bound
    M = _matrix(3000, 700, 50000, seed=5)
    D = M.to_device(rowptr_bits=64)
    r0, r1 = 1000, 1800
    V = DeviceCSR(r1 - r0, M.ncols, D.rowptr[r0:r1 + 1], D.col, D.val, nnz=int(M.rowptr[r1]))
    T = ops.transpose(ctx, V)
    a, b = M.rowptr[r0], M.rowptr[r1]
    order = np.argsort(M.col[a:b], kind="stable")
    row = np.repeat(np.arange(r1 - r0), np.diff(M.rowptr[r0:r1 + 1]))
    rp = T.rowptr.cpu().numpy()
    assert rp[-1] == b - a
    np.testing.assert_array_equal(T.col[:b - a].cpu().numpy(), row[order])
    np.testing.assert_array_equal(T.val[:b - a].cpu().numpy(), M.val[a:b][order])


def test_small_budget_takes_the_segment_sort():
    # 60,000 entries: the passes want about 1.5 MB and more for their table
    M = oracle_free(400, 3000, 60000)
    c = ops.Context(0, budget=400 << 10)
    T = ops.transpose(c, M.to_device()).to_host()
    rp, col, val = oracle.transpose(M)
    np.testing.assert_array_equal(T.rowptr.astype(np.int64), rp)
    np.testing.assert_array_equal(T.col, col)
    np.testing.assert_array_equal(T.val, val)
    torch.cuda.synchronize()
    c.close()


def oracle_free(m, n, nnz):
    """Distinct columns per row (the order of equal ones is the passes' own)."""
    rng = np.random.default_rng(3)
    per = nnz // m
    col = np.concatenate([np.sort(rng.choice(n, size=per, replace=False)) for _ in range(m)])
    return HostCSR(m, n, np.arange(m + 1, dtype=np.int64) * per, col.astype(np.int32), rng.uniform(-1, 1, m * per))


@pytest.mark.parametrize("nrows,ncols,nnz", [(1, 1, 5), (1025, 1024, 2049), (1 << 20, 3, 5000), (3, 1 << 21, 70000),
                                             (50000, 1 << 20, 1300000)])
@pytest.mark.parametrize("major", [TSPG_ROWS, TSPG_COLS])
def test_coo_is_stable(ctx, nrows, ncols, nnz, major):
    rng = np.random.default_rng(nnz)
    r, c = rng.integers(0, nrows, nnz).astype(np.int32), rng.integers(0, ncols, nnz).astype(np.int32)
    v = rng.uniform(-1, 1, nnz)
    dev = [torch.from_numpy(a).cuda() for a in (r, c, v)]
    M = ops.coo_to_csx(ctx, nrows, ncols, *dev, major=major).to_host()
    maj, mnr, nmaj = (r, c, nrows) if major == TSPG_ROWS else (c, r, ncols)
    order = np.lexsort((np.arange(nnz), mnr, maj))
    np.testing.assert_array_equal(M.rowptr, np.concatenate([[0], np.cumsum(np.bincount(maj, minlength=nmaj))]))
    np.testing.assert_array_equal(M.col, mnr[order])
    np.testing.assert_array_equal(M.val, v[order])
