"""Linears over few token rows, with any number of output features: the register kernel (2 to 32 rows; Q8_0F weights under f16
activations at any number) and the element-wise stores of the tcgen05 kernels, against a float64 product of the oracle's dequantised weights.

Bound: f32 sums of K f16 products (K * 2^-24 of the absolute sum at most; 2^-21 for the sizes here, as errors average) and one
rounding to f16 (2^-11 of the result)."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    from ratchet_b200 import Device
    d = Device(0)
    yield d
    d.close()


def weights(g, kind, N, K):
    """(stored form, dtype, float64 values)"""
    from ratchet_b200 import capi
    w = g.standard_normal((N, K)) * 0.05
    if kind == "f32":
        return w.astype(np.float32), capi.F32, w.astype(np.float32).astype(np.float64)
    if kind == "f16":
        return w.astype(np.float16), capi.F16, w.astype(np.float16).astype(np.float64)
    if kind == "q8_0h":
        buf = orc.quantize_q8(w.astype(np.float16))
        return buf, capi.Q8_0H, orc.dequantize_q8(buf, (N, K), True).astype(np.float64)
    if kind == "q8_0f":
        buf = orc.quantize_q8(w.astype(np.float32))
        return buf, capi.Q8_0F, orc.dequantize_q8(buf, (N, K), False).astype(np.float64)
    buf = orc.quantize_q4k(w.astype(np.float32), True)
    return buf, capi.Q4_KH, orc.dequantize_q4k(buf, (N, K), True).astype(np.float64)


def run(dev, kind, M, N, K, with_bias):
    g = np.random.Generator(np.random.PCG64(M * 3 + N * 5 + K))
    stored, dt, w = weights(g, kind, N, K)
    act = np.float32 if kind == "f32" else np.float16
    x, b = g.standard_normal((M, K)).astype(act), g.standard_normal(N).astype(act)
    dw = dev.from_numpy(stored) if kind in ("f16", "f32") else dev.from_quantized(stored, dt, (N, K))
    y = dev.matmul(dw, dev.from_numpy(x), dev.from_numpy(b) if with_bias else None, False, True, True)
    x64 = x.astype(np.float64)
    ref = x64 @ w.T + (b.astype(np.float64) if with_bias else 0.0)
    size = np.abs(x64) @ np.abs(w).T + 1.0
    out = 2.0 ** -11 * np.abs(ref) if act == np.float16 else 0.0
    bad = np.abs(y.to_numpy().astype(np.float64) - ref) > out + 2.0 ** -20 * size
    assert y.shape == (M, N) and not bad.any(), f"{kind} {M}x{N}x{K}: {bad.sum()} of {bad.size}"


# rows: one, two and four tiles of eight tokens, whole and ragged; K: less than the eight warps' first chunks, half a chunk at the end,
# more chunks than the warps hold ahead; N: less than a tile, odd, beside a tile's edge
@pytest.mark.parametrize("kind", ["f16", "q8_0h", "q8_0f", "q4_kh"])
@pytest.mark.parametrize("M,N,K", [(2, 16, 256), (7, 5, 512), (8, 33, 768), (9, 31, 1024), (16, 130, 2560), (17, 64, 256), (32, 257, 3072)])
def test_few_rows(dev, kind, M, N, K):
    run(dev, kind, M, N, K, with_bias=N % 2 == 1)


@pytest.mark.parametrize("kind,M,N,K", [("q8_0h", 3, 40, 96), ("q8_0f", 12, 40, 32), ("f16", 5, 24, 72), ("f16", 20, 24, 40),
                                        # enough weight rows for the wide tile
                                        ("f16", 4, 14239, 128), ("q8_0h", 13, 14240, 96), ("q4_kh", 25, 14241, 256), ("q8_0f", 31, 14249, 64)])
def test_few_rows_edges(dev, kind, M, N, K):
    run(dev, kind, M, N, K, with_bias=False)


@pytest.mark.parametrize("M,N,K", [(33, 47, 96), (64, 129, 1024), (100, 31, 160), (129, 300, 512)])
def test_q8_0f_at_any_number_of_rows(dev, M, N, K):
    run(dev, "q8_0f", M, N, K, with_bias=True)


@pytest.mark.parametrize("kind,M,N,K", [("f16", 33, 65, 128), ("f16", 130, 129, 512), ("q8_0h", 40, 67, 256), ("q4_kh", 300, 130, 256), ("f16", 1030, 2499, 128),
                                        ("f32", 2, 64, 32), ("f32", 31, 67, 128), ("f32", 65, 130, 2048), ("f32", 200, 129, 96)])
def test_any_number_of_features(dev, kind, M, N, K):
    run(dev, kind, M, N, K, with_bias=True)


# the promise is about matrix-vector products: a matrix written right before it is multiplied by a few rows is read as written
@pytest.mark.parametrize("kind,M", [("f16", 8), ("f16", 2), ("q8_0f", 20), ("q8_0f", 100)])
def test_weights_that_were_just_written_under_constant_weights(dev, kind, M):
    from ratchet_b200 import capi
    N, K = 2048, 1024
    g = np.random.Generator(np.random.PCG64(M))
    x = dev.from_numpy(g.standard_normal((M, K)).astype(np.float16))
    dense = [(g.standard_normal((N, K)) * 0.05).astype(np.float32) for _ in range(2)]
    if kind == "f16":
        sources = [dev.from_quantized(orc.quantize_q8(d.astype(np.float16)), capi.Q8_0H, (N, K)) for d in dense]
        w, write = dev.empty(capi.F16, (N, K)), dev.dequantize
    else:
        sources = [dev.from_numpy(d) for d in dense]
        w, write = dev.empty(capi.Q8_0F, (N, K)), dev.quantize
    want = []
    for s in sources:
        write(s, w)
        want.append(dev.matmul(w, x, None, False, True, True).to_numpy())
    assert not np.array_equal(*want)
    dev.set_constant_weights(True)
    try:
        for i in range(60):
            write(sources[i % 2], w)
            assert np.array_equal(dev.matmul(w, x, None, False, True, True).to_numpy(), want[i % 2])
    finally:
        dev.set_constant_weights(False)
