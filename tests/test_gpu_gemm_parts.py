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


# more tiles than SMs and rows that do not start on four features: as exact as where there are few (and as the FMA pipe)
@pytest.mark.parametrize("M,N,K", [(450, 2501, 10240), (129, 9999, 260), (600, 2050, 64)])
def test_many_tiles_of_odd_features(dev, M, N, K):
    g = np.random.Generator(np.random.PCG64(N))
    x, w, b = g.standard_normal((1, M, K), np.float32), g.standard_normal((N, K), np.float32) * np.float32(0.05), g.standard_normal(N, np.float32)
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


# token rows that the FMA pipe, and that split TF32 took before; one tile per CTA and tiles that are cut
@pytest.mark.parametrize("M,N,K", [(2, 64, 64), (20, 100, 300), (31, 128, 2560), (64, 128, 512), (200, 72, 256)])
def test_infinities_and_nan_as_in_f32(dev, M, N, K):
    """Values near the type's largest stay finite; infinities and NaN give what f32 arithmetic gives, sign by sign, and only where they meet."""
    g = np.random.Generator(np.random.PCG64(M + K))
    # whole numbers and halves, many of whose remainders are zero, beside numbers of 24 bits
    x, w = (np.where(g.random(s) < 0.5, g.integers(1, 5, s) * g.choice([-0.5, 0.5], s), g.standard_normal(s)).astype(np.float32) for s in ((1, M, K), (N, K)))
    x[0, 0, 3], x[0, 1, 5], w[7, 9], w[8, 2] = np.inf, -np.inf, np.inf, np.nan
    w[11, 3] = 0.0
    w.view(np.uint32)[9, 1] = 0x7f800001                     # NaN in the bits that no leading part holds
    w[20], x[0, :, 30] = 0.0, 1.0
    w[20, 30] = 3.4e38
    with np.errstate(invalid="ignore"):
        want = x[0].astype(np.float64) @ w.astype(np.float64).T
        want[:, 9] = np.nan
    got = nn.Linear(tensor(dev, w)).schedule(tensor(dev, x)).resolve().to_numpy()[0].astype(np.float64)
    fine = np.isfinite(want)
    assert np.isinf(want).sum() > N and np.isnan(want).sum() > 2 * M - 2
    assert np.array_equal(got[~fine], want[~fine], equal_nan=True)
    got, want = (np.where(fine, a, 0) for a in (got, want))
    assert np.linalg.norm((got - want)[:, :20]) <= (2.0 ** -23 + 16 * 2.0 ** -24) * np.linalg.norm(want[:, :20])
    assert np.abs(got[2:, 20] / np.float64(np.float32(3.4e38)) - 1).max(initial=0) < 1e-6
