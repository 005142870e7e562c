"""f32 products over operands in three bf16 parts, against float64.

Bound: partial products below 2^-23 are left out, and the leading parts meet sixteen truncating additions (2^-23 each at most, half of it on
average) before their sums are rounded like any f32 sum: 2^-23 + 16 * 2^-24 of the result's norm."""
import numpy as np
import pytest

from ratchet_b200 import nn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from ratchet_b200 import Device
    d = Device(0)
    yield d
    d.close()


def tensor(dev, a):
    from ratchet_b200 import Tensor
    return Tensor.from_data(np.ascontiguousarray(a, np.float32), device=dev)


# beside the tiles of 16, 32 and 64 tokens and 128 features, units of 64 and sums restarted at 256 of K, whole tiles and runs across tiles
@pytest.mark.parametrize("M", [2, 15, 16, 17, 32, 33, 64, 65, 129])
@pytest.mark.parametrize("N,K", [(64, 32), (100, 36), (128, 64), (129, 256), (127, 260), (300, 1028), (640, 2560), (64, 8192), (4000, 320)])
def test_linear_f32(dev, M, N, K):
    g = np.random.Generator(np.random.PCG64(M * N + K))
    x, w, b = g.standard_normal((1, M, K)), g.standard_normal((N, K)) * 0.05, g.standard_normal(N)
    x, w, b = (a.astype(np.float32) for a in (x, w, b))
    got = nn.Linear(tensor(dev, w), tensor(dev, b)).schedule(tensor(dev, x)).resolve().to_numpy()[0].astype(np.float64)
    want = x[0].astype(np.float64) @ w.astype(np.float64).T + b
    assert np.linalg.norm(got - want) <= (2.0 ** -23 + 16 * 2.0 ** -24) * np.linalg.norm(want)


@pytest.mark.parametrize("B,M,N,K", [(3, 40, 72, 64), (2, 100, 64, 300), (5, 17, 128, 36)])
def test_batched_f32(dev, B, M, N, K):
    g = np.random.Generator(np.random.PCG64(B))
    a, b = (g.standard_normal(s).astype(np.float32) for s in ((1, B, M, K), (1, B, N, K)))
    got = tensor(dev, a).matmul(tensor(dev, b), False, True).resolve().to_numpy().astype(np.float64)
    want = a.astype(np.float64) @ b.astype(np.float64).transpose(0, 1, 3, 2)
    assert np.linalg.norm(got - want) <= (2.0 ** -23 + 16 * 2.0 ** -24) * np.linalg.norm(want)


def test_large_values_and_nan(dev):
    """Values near the type's largest stay finite; infinities and NaN reach the tokens and features that they meet."""
    w, x = np.zeros((64, 64), np.float32), np.ones((1, 20, 64), np.float32)
    np.fill_diagonal(w, 1.0)
    w[3, 3], x[0, 5, 7], x[0, 6, 8] = 3.4e38, np.nan, np.inf
    got = nn.Linear(tensor(dev, w)).schedule(tensor(dev, x)).resolve().to_numpy()[0]
    fine = np.ones(20, bool)
    fine[5:7] = False
    assert np.isfinite(got[fine]).all() and abs(got[0, 3] / 3.4e38 - 1) < 1e-6 and not np.isfinite(got[5, 7]) and not np.isfinite(got[6, 8])
