"""Attention of an f32 block in one pass over split operands, against a float64 evaluation and the same graph with one kernel per op.

Bound: both are f32-level, their errors against float64 come from scores that are off by a few 2^-24 and sums that are; the fused path may be
off by no more than the chain of split-TF32 products, plus the rounding of the comparison itself (2^-24 of the values)."""
import numpy as np
import pytest

from ratchet_b200 import callers, nn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from ratchet_b200 import Device
    d = Device(0)
    yield d
    d.close()


class Same:
    def schedule(self, x):
        return x


# beside the tiles of 64 keys and 128 queries, one and two query tiles, one and several runs of keys, heads narrower than a 64-column plane
@pytest.mark.parametrize("T,H,D", [(2, 1, 64), (63, 2, 64), (64, 1, 32), (65, 2, 64), (128, 1, 48), (129, 3, 64), (256, 1, 4), (257, 6, 64), (501, 6, 64),
                                   (1500, 6, 64), (300, 2, 20), (700, 40, 64)])
def test_against_64_bits_and_the_unfused_graph(dev, T, H, D):
    from ratchet_b200 import Tensor
    g = np.random.Generator(np.random.PCG64(T + D))
    d = H * D
    t = lambda a: Tensor.from_data(np.ascontiguousarray(a, np.float32), device=dev)
    x = g.standard_normal((1, T, d)).astype(np.float32)
    ws = [(g.standard_normal((d, d)) * 1.5 / np.sqrt(d)).astype(np.float32) for _ in range(3)]
    dk = np.float32(float(D) ** -0.25)

    def run(**debug):
        mha = callers.WhisperMHA(*[nn.Linear(t(w)) for w in ws], Same(), H, t(np.array([dk])))
        out = mha.schedule(t(x))
        dev.set_debug(profile=True, **debug)
        try:
            dev.profile_report()
            out.resolve()
            names = dev.profile_report()
        finally:
            dev.set_debug()
        return out.to_numpy().astype(np.float64), names

    (got, names), (chain, names0) = run(), run(no_reuse=True)
    assert "attention" in names and "softmax" not in names and "softmax" in names0
    # from the projections as the device has them, so that only the attention's own error is seen
    q, k, v = (nn.Linear(t(w)).schedule(t(x)).resolve().to_numpy().astype(np.float64).reshape(T, H, D).transpose(1, 0, 2) for w in ws[:3])
    z = (q * dk) @ (k * dk).transpose(0, 2, 1)
    p = np.exp(z - z.max(-1, keepdims=True))
    want = ((p / p.sum(-1, keepdims=True)) @ v).transpose(1, 0, 2).reshape(1, T, d)
    n = np.linalg.norm(want)
    err, err0 = np.linalg.norm(got - want) / n, np.linalg.norm(chain - want) / n
    assert err <= err0 + 2.0 ** -24, (err, err0)


def test_infinities_and_nan(dev):
    """An overflowing score and NaN in a value reach the rows they reach with one kernel per op."""
    from ratchet_b200 import Tensor
    T, D = 300, 64
    g = np.random.Generator(np.random.PCG64(2))
    x = g.standard_normal((1, T, D)).astype(np.float32)
    x[0, 7] *= 1e25                                     # its own score overflows
    eye = np.eye(D, dtype=np.float32)
    t = lambda a: Tensor.from_data(np.ascontiguousarray(a, np.float32), device=dev)
    res = []
    for no_reuse in (False, True):
        dev.set_debug(no_reuse=no_reuse)
        try:
            res.append(callers.WhisperMHA(*[nn.Linear(t(eye)) for _ in range(4)], 1, t(np.array([0.3]))).schedule(t(x)).resolve().to_numpy())
        finally:
            dev.set_debug()
    assert np.array_equal(np.isfinite(res[0]), np.isfinite(res[1])) and not np.isfinite(res[1]).all()


@pytest.mark.parametrize("T", [2, 20, 31])
def test_infinite_operands_as_in_f32(dev, T):
    """Few positions: a key that no query can see (a score of minus infinity has no weight), one that takes everything (NaN), infinite values."""
    from ratchet_b200 import Tensor
    D, L = 64, 200
    g = np.random.Generator(np.random.PCG64(T))
    q, k, v = (g.standard_normal((1, 1, n, D)).astype(np.float32) for n in (T, L, L))
    q[..., 0] = np.abs(q[..., 0]) + 0.5
    q[0, 0, 1, 0] *= -1                                  # to this query the second key is plus infinity
    k[0, 0, 1, 0], v[0, 0, 5, 7], v[0, 0, 6, 8] = -np.inf, np.inf, -np.inf
    t = lambda a: Tensor.from_data(np.ascontiguousarray(a, np.float32), device=dev)
    one = t(np.array([1.0]))
    heads = lambda a: t(a.transpose(0, 2, 1, 3))
    a, b = heads(q).permute([0, 2, 1, 3]).mul(one), heads(k).permute([0, 2, 3, 1]).mul(one)
    dev.set_debug(profile=True)
    try:
        dev.profile_report()
        got = a.matmul(b).softmax(3).matmul(heads(v).permute([0, 2, 1, 3])).permute([0, 2, 1, 3])
        del a, b
        got = got.resolve().to_numpy()[0, :, 0].astype(np.float64)
        assert "attention" in dev.profile_report()
    finally:
        dev.set_debug()
    with np.errstate(invalid="ignore"):
        s = q[0, 0].astype(np.float64) @ k[0, 0].astype(np.float64).T
        p = np.exp(s - s.max(-1, keepdims=True))
        want = (p / p.sum(-1, keepdims=True)) @ v[0, 0].astype(np.float64)
    assert np.isnan(want[1]).all() and np.isfinite(np.delete(want[0], [7, 8])).all() and want[0, 7] == np.inf and want[0, 8] == -np.inf
    fine = np.isfinite(want)
    assert np.array_equal(got[~fine], want[~fine], equal_nan=True)
    got, want = (np.where(fine, a, 0) for a in (got, want))
    assert np.linalg.norm(got - want) < 1e-5 * np.linalg.norm(want)


def test_the_switch_that_keeps_f32_off_the_tensor_cores():
    import os
    import subprocess
    import sys
    code = """
import numpy as np
from ratchet_b200 import Device, Tensor
dev = Device(0)
q, k, v = (Tensor.from_data(np.ones((1, 40, 1, 64), np.float32), device=dev) for _ in range(3))
s = Tensor.from_data(np.ones(1, np.float32), device=dev)
o = q.permute([0, 2, 1, 3]).mul(s).matmul(k.permute([0, 2, 3, 1]).mul(s)).softmax(3).matmul(v.permute([0, 2, 1, 3])).permute([0, 2, 1, 3])
dev.set_debug(profile=True)
assert np.abs(o.resolve().to_numpy() - 1).max() < 1e-5
print("attention" in dev.profile_report())
"""
    for switch, fused in (("1", "True"), ("0", "False")):
        p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, env={**os.environ, "RCU_GEMM_F32_TC": switch})
        assert p.returncode == 0 and p.stdout.strip() == fused, (switch, p.stdout, p.stderr)
