"""Quantised weights that the CTA-pair GEMM converts on the way: bit for bit what the product over the converted matrix gives (the same
f16 weights in the same order of sums), at the edges of its tiles, steps and rings, with each epilogue."""
import numpy as np
import pytest

from ratchet_b200 import Tensor, capi, nn

pytestmark = pytest.mark.gpu

F16 = np.float16


@pytest.fixture(scope="module")
def dev():
    from ratchet_b200 import Device
    d = Device(0)
    yield d
    d.close()


def codes(g, kind, n, k):
    """W [n, k] of random codes and scales in ratchet's layout."""
    dt = capi.Q8_0H if kind == "q8_0h" else capi.Q4_KH
    at, raw = capi.dtype_segments(dt, n * k), np.zeros(capi.dtype_nbytes(dt, n * k), np.uint8)
    if kind == "q8_0h":
        raw[:n * k] = g.integers(0, 256, n * k)
        d = (g.random(n * k // 32) * 4e-4).astype(F16)
        raw[at[1]:at[1] + d.nbytes] = d.view(np.uint8)
    else:
        raw[:n * k // 2] = g.integers(0, 256, n * k // 2)
        raw[at[1]:at[1] + n * k // 256 * 12] = g.integers(0, 256, n * k // 256 * 12)
        for i in (2, 3):
            d = (g.random(n * k // 256) * 1e-4).astype(F16)
            raw[at[i]:at[i] + d.nbytes] = d.view(np.uint8)
    return raw, dt


# the rule, and the pair kernel at sizes that the rule leaves to the others: None and "2" of RCU_GEMM_FUSED
ROUTES = [None, "2"]


def force(monkeypatch, route):
    monkeypatch.delenv("RCU_GEMM_FUSED", raising=False)
    if route is not None:
        monkeypatch.setenv("RCU_GEMM_FUSED", route)


# one group of steps, rings that wrap, one tile per pair and several; ragged rows, columns and columns that are no multiple of four; three
# rows of tiles, and the other side of the rule: too few columns for the rounds, a K of other than whole groups (converted both times)
SIZES = [("q8_0h", 257, 5120, 256), ("q8_0h", 512, 5125, 512), ("q8_0h", 300, 16384, 3072), ("q8_0h", 400, 40000, 768), ("q8_0h", 700, 16384, 256), ("q8_0h", 700, 9728, 512), ("q8_0h", 300, 4992, 288),
         ("q4_kh", 257, 6400, 256), ("q4_kh", 512, 6501, 512), ("q4_kh", 512, 5001, 512), ("q4_kh", 300, 16384, 3072), ("q4_kh", 512, 8192, 1280), ("q4_kh", 333, 40002, 768)]


@pytest.mark.parametrize("kind,M,N,K", SIZES)
@pytest.mark.parametrize("route", ROUTES)
def test_equals_the_product_over_the_converted_matrix(dev, monkeypatch, kind, M, N, K, route):
    g = np.random.Generator(np.random.PCG64(M + N + K))
    raw, dt = codes(g, kind, N, K)
    w, x, b = dev.from_quantized(raw, dt, (N, K)), dev.from_numpy(g.standard_normal((M, K)).astype(F16)), dev.from_numpy(g.standard_normal(N).astype(F16))
    force(monkeypatch, route)
    launches = dev.launches
    got = dev.matmul(w, x, b, False, True, True).to_numpy()
    if route == "2":
        assert dev.launches - launches == 1                # no conversion in front
    force(monkeypatch, "0")
    want = dev.matmul(w, x, b, False, True, True).to_numpy()
    assert np.isfinite(want).all() and np.array_equal(got.view(np.uint16), want.view(np.uint16))


# one row of tiles: the first and last rows of a CTA of the pair, none in the second; against the one-CTA kernel that converts, which does not cut K at
# these sizes either (the last two are on the other side of the rule) but for 18944 columns: 148 tiles of 128, two slices of K.  There f32 sums of K products
# come in another order (2^-24 each, random signs), and an output may round to f16's neighbour.
@pytest.mark.parametrize("kind", ["q8_0h", "q4_kh"])
@pytest.mark.parametrize("route", ROUTES)
@pytest.mark.parametrize("M,N,K", [(129, 5120, 2048), (256, 4801, 2304), (200, 16384, 256), (33, 9728, 2048), (128, 18944, 2048), (128, 19200, 2048), (256, 8192, 1024)])
def test_one_row_of_tiles(dev, monkeypatch, kind, M, N, K, route):
    g = np.random.Generator(np.random.PCG64(M + N + K))
    raw, dt = codes(g, kind, N, K)
    w, x, b = dev.from_quantized(raw, dt, (N, K)), dev.from_numpy(g.standard_normal((M, K)).astype(F16)), dev.from_numpy(g.standard_normal(N).astype(F16))
    force(monkeypatch, route)
    got = dev.matmul(w, x, b, False, True, True).to_numpy()
    force(monkeypatch, "1")
    want = dev.matmul(w, x, b, False, True, True).to_numpy()
    assert np.isfinite(want).all()
    if N == 18944:
        got, want = got.astype(np.float64), want.astype(np.float64)
        assert (np.abs(got - want) <= 2.0 ** -10 * np.abs(want) + 4 * 2.0 ** -24 * np.sqrt(K) * np.sqrt((want ** 2).mean())).all()
    else:
        assert np.array_equal(got.view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("kind,M,F,K", [("q8_0h", 500, 2608, 512), ("q4_kh", 470, 4912, 768), ("q8_0h", 200, 5120, 2048), ("q4_kh", 130, 5600, 2048)])
@pytest.mark.parametrize("what", ["gate", "gelu", "resid"])
@pytest.mark.parametrize("route", ROUTES)
def test_epilogues(dev, monkeypatch, kind, M, F, K, what, route):
    g = np.random.Generator(np.random.PCG64(F))
    raw, dt = codes(g, kind, 2 * F, K)
    x, r = g.standard_normal((1, M, K)).astype(F16), g.standard_normal((1, M, 2 * F)).astype(F16)

    def run():
        h = nn.Linear(Tensor.from_quantized(raw, dt, (2 * F, K), dev)).schedule(Tensor.from_data(x, device=dev))
        if what == "gelu":
            return h.full().gelu().cast(capi.F16).resolve().to_numpy()
        if what == "resid":
            return h.add(Tensor.from_data(r, device=dev)).resolve().to_numpy()
        return h.slice([(0, 1), (0, M), (F, 2 * F)]).mul(h.slice([(0, 1), (0, M), (0, F)]).full().silu().cast(capi.F16)).resolve().to_numpy()

    force(monkeypatch, route)
    got = run()
    force(monkeypatch, "0")
    assert np.array_equal(got.view(np.uint16), run().view(np.uint16))
