"""GPU: output arrays from a caller's allocator that refuses some requests."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import check_product, check_sum, random_csr
from trident_b200 import ops
from trident_b200._lib import ALLOC_FN, TSPG_ENOMEM, TSPG_ROWS, TspgCsrOut, lib
from trident_b200.csr import DeviceCSR

pytestmark = pytest.mark.gpu


class Hook:
    """Refuses the requests numbered in `refuse`; notes sizes and the device's
    free memory at each request."""

    def __init__(self, refuse):
        self.refuse, self.asked, self.free, self.blocks = refuse, [], [], {}
        self.cb = ALLOC_FN(self._alloc)

    def _alloc(self, user, nbytes, stream):
        self.asked.append(nbytes)
        self.free.append(torch.cuda.mem_get_info()[0])
        if len(self.asked) - 1 in self.refuse:
            return None
        t = torch.empty(max(nbytes, 16), dtype=torch.uint8, device="cuda")
        self.blocks[t.data_ptr()] = t
        return t.data_ptr()

    def out(self, nrows, ncols):
        o = TspgCsrOut()
        self.rp = torch.empty(nrows + 1, dtype=torch.int64, device="cuda")
        o.nrows, o.ncols, o.rowptr, o.rowptr_bits, o.val_bits = nrows, ncols, self.rp.data_ptr(), 64, 64
        o.alloc = self.cb
        return o

    def result(self, o):
        return DeviceCSR(int(o.nrows), int(o.ncols), self.rp, self.blocks[o.col].view(torch.int32),
                         self.blocks[o.val].view(torch.float64), nnz=int(o.nnz))


def _calls(ctx, A, B):
    dA, dB = A.to_device(), B.to_device()
    a, b = dA.abi(), dB.abi()
    s = torch.cuda.current_stream().cuda_stream
    r = np.repeat(np.arange(A.nrows), np.diff(A.rowptr)).astype(np.int32)
    row, keep = torch.from_numpy(r).cuda(), (dA, dB)
    return keep, {
        "spgemm": (A.nrows, B.ncols, lambda o: lib.tspg_spgemm(ctx.h, s, C.byref(a), C.byref(b), C.byref(o), 0),
                   lambda M: check_product(M, A, B)),
        "spadd": (A.nrows, A.ncols, lambda o: lib.tspg_spadd(ctx.h, s, C.byref(a), C.byref(b), C.byref(o)),
                  lambda M: check_sum(M, A, B)),
        "prune": (A.nrows, A.ncols, lambda o: lib.tspg_mcl_prune(ctx.h, s, C.byref(a), 0.0, C.byref(o)),
                  lambda M: np.testing.assert_array_equal(M.to_host().col, A.col)),
        "transpose": (A.ncols, A.nrows, lambda o: lib.tspg_transpose(ctx.h, s, C.byref(a), C.byref(o)),
                      lambda M: np.testing.assert_array_equal(np.sort(M.to_host().val), np.sort(A.val))),
        "coo": (A.nrows, A.ncols,
                lambda o: lib.tspg_coo_to_csx(ctx.h, s, A.nrows, A.ncols, A.nnz, row.data_ptr(), dA.col.data_ptr(),
                                              dA.val.data_ptr(), 64, TSPG_ROWS, C.byref(o)),
                lambda M: np.testing.assert_array_equal(M.to_host().col, A.col)),
    }


@pytest.mark.parametrize("call", ["spgemm", "spadd", "prune", "transpose", "coo"])
@pytest.mark.parametrize("refuse", [(0,), (1,), (0, 2)])
def test_refused_once_and_asked_again(call, refuse):
    # the pool keeps 64 MB of an earlier call: at a refusal they go back to the
    # device, and only what is missing is asked for again
    ctx = ops.Context(0)
    big = random_csr(64, 60000, per_row=60000, seed=1)
    ops.transpose(ctx, big.to_device())  # workspace of 24 bytes an entry: 92 MB
    A, B = random_csr(900, 900, per_row=9, seed=2), random_csr(900, 900, per_row=11, seed=3)
    keep, calls = _calls(ctx, A, B)
    m, n, run, check = calls[call]
    hook = Hook(refuse)
    o = hook.out(m, n)
    status = run(o)
    nnz = int(o.nnz)
    want = {(0,): [4, 4, 8], (1,): [4, 8, 8], (0, 2): [4, 4, 8]}[refuse]
    assert hook.asked == [k * nnz for k in want]
    assert max(hook.free[1:]) >= hook.free[0] + (64 << 20)
    if refuse == (0, 2):
        assert status == TSPG_ENOMEM
    else:
        assert status == 0
        check(hook.result(o))
    ctx.close()


def test_transpose_output_does_not_wait_for_the_workspace():
    # an allocator with room for the output, but not beside 24 bytes an entry
    ctx = ops.Context(0)
    A = random_csr(500, 800, per_row=400, seed=4)
    keep, calls = _calls(ctx, A, A)
    m, n, run, check = calls["transpose"]

    class Tight(Hook):
        def _alloc(self, user, nbytes, stream):
            if ctx.mem()[0] > 8 * A.nnz:
                self.refuse = (len(self.asked),)
            return super()._alloc(user, nbytes, stream)

    hook = Tight(())
    o = hook.out(m, n)
    assert run(o) == 0
    check(hook.result(o))
    # and a budget that only the segment sort fits
    ref = hook.result(o).to_host()
    small = ops.Context(0, 12 * A.nnz)
    got = ops.transpose(small, A.to_device()).to_host()
    for x, y in ((got.rowptr, ref.rowptr), (got.col, ref.col), (got.val, ref.val)):
        np.testing.assert_array_equal(x, y)
    small.close()
    ctx.close()
