"""The native base of ``Tensor``: arguments by position and name, errors, lifetime - on graphs without a device."""
import ctypes as C
import os
import shutil
import subprocess
import sys
import sysconfig

import numpy as np
import pytest

from ratchet_b200 import Tensor, _build, capi
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


def run(code, folder=None, **env):
    return subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env={**os.environ, **env}, timeout=300,
                          cwd=folder or os.path.join(_build.HERE, ".."))


def test_no_tensor_before_the_library_is_loaded():
    p = run("from ratchet_b200 import Tensor\ntry: Tensor(None, 16)\nexcept RuntimeError as e: print(e)")
    assert p.returncode == 0 and "has not been loaded" in p.stdout, p.stderr


@pytest.fixture
def checkout(tmp_path):
    """The package's sources without anything built."""
    pkg = tmp_path / "ratchet_b200"
    shutil.copytree(_build.HERE, pkg, ignore=shutil.ignore_patterns("*.so", "_obj", "__pycache__"))
    shutil.copytree(os.path.join(_build.HERE, "..", "include"), tmp_path / "include")
    return tmp_path


def test_importing_needs_no_compiler(checkout):
    code = "import ratchet_b200 as r\nfrom ratchet_b200 import gguf, nn, callers, models\n" \
           "assert r.__file__.startswith(%r)\ntry: r.Tensor(None, 16)\nexcept r.RatchetCudaError as e: print(e)" % str(checkout)
    p = run(code, checkout, CC="no-such-compiler")
    assert p.returncode == 0 and "could not be built" in p.stdout, p.stderr


def test_the_module_is_as_new_as_its_source(checkout):
    """Built on the first import under this interpreter's name, left alone by the second, built again after a change of the header."""
    built = checkout / "ratchet_b200" / ("_graph" + sysconfig.get_config_var("EXT_SUFFIX"))
    code = "import ratchet_b200 as r; assert r.__file__.startswith(%r) and r.Tensor.__base__.__module__ == 'ratchet_b200._graph'" % str(checkout)
    assert os.path.basename(_build.GRAPH_LIB) == built.name
    for change, again in ((False, True), (False, False), (True, True)):
        if built.exists():
            os.utime(built, (1e9, 1e9))
        for f in (checkout / "include" / "ratchet_cuda.h", checkout / "ratchet_b200" / "csrc" / "pygraph.c"):
            os.utime(f, (1e9 - 10, 1e9 + 10 if change else 1e9 - 10))
        p = run(code, checkout)
        assert p.returncode == 0, p.stderr
        assert (os.path.getmtime(built) != 1e9) == again
