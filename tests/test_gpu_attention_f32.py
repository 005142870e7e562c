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
    print(f"T={T} H={H} D={D}: {err:.2e}, one kernel per op {err0:.2e}")
    assert err <= err0 + 2.0 ** -24


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
