"""The native base of ``Tensor``: arguments by position and name, errors, lifetime - on graphs without a device."""
import ctypes as C

import numpy as np
import pytest

from ratchet_b200 import Tensor, capi
from ratchet_b200.capi import RatchetCudaError


class NoDevice:
    handle = True

    def __init__(self):
        self._lib = capi.lib()

    def check(self, st):
        if st != capi.OK:
            raise RatchetCudaError(st, "")


def leaf(*shape, dt=capi.F32):
    dev, h, d = NoDevice(), C.c_void_p(), capi.describe(dt, shape, 0x1000)
    assert dev._lib.rcu_lazy_wrap(None, C.byref(d), C.byref(h)) == capi.OK
    return Tensor(dev, h)


def test_builders_take_names_and_positions():
    x, w = leaf(2, 3, 8), leaf(16, 8)
    assert w.gemm(x, None, False, True, True).shape() == w.gemm(rhs=x, bias=None, trans_lhs=False, trans_rhs=True, trans_out=True).shape() == (2, 3, 16)
    assert x.view([6, 8]).matmul(rhs=w, trans_rhs=True).shape() == (6, 16)
    assert x.slice([(0, 2), (1, 3), (0, 4)]).shape() == x.slice([slice(None), slice(1, None), (0, 4)]).shape() == (2, 2, 4)
    assert x.permute([2, 0, 1]).shape() == x.permute(dims=(2, 0, 1)).shape() == (8, 2, 3)
    assert x.half().dt() == x.cast(dst_dt=capi.F16).dt() == capi.F16
    assert x.layer_norm(leaf(8), bias=None, eps=1e-5).softmax(dim=2).shape() == (2, 3, 8)
    assert x.rank() == 3 and x.resolved() and x.data_ptr() == 0x1000


@pytest.mark.parametrize("call, error", [
    (lambda x: x.view([5]), RatchetCudaError), (lambda x: x.view([1] * 9), RatchetCudaError), (lambda x: x.permute([0, 1]), RatchetCudaError),
    (lambda x: x.slice([(0, 1)]), RatchetCudaError), (lambda x: x.slice([(0, 3), (0, 3), (0, 8)]), RatchetCudaError), (lambda x: x.softmax(-1), RatchetCudaError),
    (lambda x: x.permute([0, 1.0, 2]), TypeError), (lambda x: x.view(6), TypeError), (lambda x: x.add(3), TypeError), (lambda x: x.matmul(), TypeError), (lambda x: x.matmul(x, trans=True), TypeError), (lambda x: x.add(x, other=x), TypeError),
])
def test_refusals(call, error):
    with pytest.raises(error):
        call(leaf(2, 3, 8))


def test_a_handle_is_one_reference():
    x = leaf(4, 4)
    y, z = x.clone(), x.gelu()
    assert x.strong_count() == 3
    del y, z
    assert x.strong_count() == 1
    x.consume()
    x.consume()
    assert x._h is None and x.shape() == ()
    with pytest.raises(RatchetCudaError):
        x.gelu()


def test_a_sequence_that_changes_while_it_is_read():
    x, shape = leaf(2, 3, 8), []

    class Entry:
        def __int__(self):
            shape.clear()
            return 6

    shape += [Entry(), 8]
    assert x.view(shape).shape() == (6, 8)
    assert x.view(np.array([6, 8])).shape() == (6, 8)
