"""Linears over the same rows in one launch: bit for bit what each gives by itself, at the edges of the tiles, with and without biases, and where a
member must stay apart."""
import numpy as np
import pytest

from ratchet_b200 import Device, Tensor, capi, nn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    d = Device(0)
    yield d
    d.close()


def resolved_apart(ws, bs, x):
    return [nn.Linear(w, b).schedule(x).resolve().to_numpy() for w, b in zip(ws, bs)]


# rows on either side of a tile of 64 or 128, one and several tiles of columns, ragged ones; K of one step up to the longest, and beyond it; products
# that fill the device (apart)
@pytest.mark.parametrize("dt", [np.float16, np.float32])
@pytest.mark.parametrize("M,N,K", [(65, 64, 64), (129, 72, 136), (501, 384, 384), (1500, 384, 384), (700, 200, 512), (90, 136, 1096), (2000, 1536, 256)])
@pytest.mark.parametrize("n", [2, 3, 4])
def test_equals_the_products_by_themselves(dev, dt, M, N, K, n):
    g = np.random.Generator(np.random.PCG64(M + N + K + n))
    tensor = lambda a: Tensor.from_data(a, device=dev)
    x = tensor(g.standard_normal((1, M, K)).astype(dt))
    ws = [tensor((g.standard_normal((N, K)) * 0.05).astype(dt)) for _ in range(n)]
    # the second without a bias, the third's to be rounded from 32 bits
    bs = [None if i == 1 else tensor(g.standard_normal(N).astype(np.float32 if i == 2 else dt)) for i in range(n)]
    cast = lambda i: bs[i].cast(capi.F16) if bs[i] is not None and i == 2 and dt == np.float16 else bs[i]
    want = resolved_apart(ws, [cast(i) for i in range(n)], x)
    ys = [nn.Linear(w, cast(i)).schedule(x) for i, w in enumerate(ws)]
    total = ys[-1]                               # from the right: the products come one after another in the order
    for y in ys[-2::-1]:
        total = y.add(total)
    launches = dev.launches
    total = total.resolve().to_numpy()
    launches = dev.launches - launches
    if n == 3 and (M, N, K) == (1500 if dt == np.float32 else 501, 384, 384):
        assert launches == 3                     # one for the products, two additions
    for y, z in zip(ys, want):
        assert np.array_equal(y.to_numpy(), z)
    sums = want[-1]
    for z in want[-2::-1]:
        sums = (sums.astype(np.float32) + z).astype(dt)
    assert np.array_equal(total, sums)


def test_an_output_that_takes_over_a_members_input_stays_apart(dev):
    """The first product's bias is a temporary that ends with it, so the second's output may be planned into its place."""
    g = np.random.Generator(np.random.PCG64(2))
    M, N, K = 300, 128, 128
    tensor = lambda a: Tensor.from_data(a, device=dev)
    x = tensor(g.standard_normal((1, M, K)).astype(np.float32))
    ws = [tensor((g.standard_normal((N, K)) * 0.05).astype(np.float32)) for _ in range(3)]
    b = [tensor(g.standard_normal(N).astype(np.float32)) for _ in range(2)]
    want = resolved_apart(ws, [b[0].add(b[1]).resolve(), None, None], x)
    y = nn.Linear(ws[0], b[0].add(b[1])).schedule(x).mul(nn.Linear(ws[1]).schedule(x).mul(nn.Linear(ws[2]).schedule(x)))
    assert np.array_equal(y.resolve().to_numpy(), want[0] * (want[1] * want[2]))


# an f32 product and the addition behind it: whole tiles of 32 and of 64 tokens, tiles that are cut into runs, one row too few or many; a product that
# another kernel runs (apart); whole tiles of 64 tokens with short K, and with a longer one (apart)
@pytest.mark.parametrize("M,N,K", [(16, 136, 256), (33, 128, 512), (64, 2560, 2048), (65, 260, 96), (1500, 384, 384), (1501, 384, 1536), (70, 61, 128), (1500, 1536, 384), (2, 64, 64),
                                   (65, 9216, 256), (1500, 512, 512), (750, 768, 768)])
@pytest.mark.parametrize("left", [False, True])
@pytest.mark.parametrize("quantised", [False, True])
def test_the_addition_behind_an_f32_product(dev, M, N, K, left, quantised):
    from oracle import oracle as orc
    g = np.random.Generator(np.random.PCG64(M + N + K))
    w, x, r = (g.standard_normal((N, K)) * 0.05).astype(np.float32), g.standard_normal((1, M, K)).astype(np.float32), g.standard_normal((1, M, N)).astype(np.float32)
    x[0, 0, 0], r[0, M - 1, N - 1] = np.inf, np.nan
    w = Tensor.from_quantized(orc.quantize_q8(w), capi.Q8_0F, (N, K), dev) if quantised else Tensor.from_data(w, device=dev)
    x, r = Tensor.from_data(x, device=dev), Tensor.from_data(r, device=dev)
    b = None if left else Tensor.from_data(g.standard_normal(N).astype(np.float32), device=dev)
    lin = nn.Linear(w, b)
    want = lin.schedule(x).resolve().to_numpy() + r.to_numpy()
    got = r.add(lin.schedule(x)) if left else lin.schedule(x).add(r)
    launches = dev.launches
    got = got.resolve()
    if not quantised and N >= 512:
        assert dev.launches - launches == (1 if M > 64 and K <= 512 and N != 1536 else 3 if M == 64 else 2)        # 64 tokens: cut into runs
    assert np.array_equal(got.to_numpy(), want, equal_nan=True)


# an activation, a permute, positions and a cast in one kernel, against the ops by themselves (each result held): pieces of 32 in both directions, ragged
# in the last two, many pieces that are mostly empty (apart)
@pytest.mark.parametrize("T,C", [(501, 384), (32, 64), (33, 31), (2, 1), (100, 97), (2, 131105), (131105, 3)])
@pytest.mark.parametrize("act", ["gelu", "silu"])
@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("left", [False, True])
def test_a_convolutions_output_to_rows(dev, T, C, act, half, left):
    g = np.random.Generator(np.random.PCG64(T + C))
    x = Tensor.from_data((g.standard_normal((1, C, T)) * 2).astype(np.float32), device=dev)
    e = Tensor.from_data(g.standard_normal((1, T, C) if left else (T, C)).astype(np.float32), device=dev)

    def schedule(keep):
        a = getattr(x, act)()
        p = a.permute([0, 2, 1])
        s = e.add(p) if left else p.add(e)
        keep.extend([a, p, s])
        return s.cast(capi.F16) if half else s

    held = []
    want = schedule(held).resolve().to_numpy()
    launches = dev.launches
    handles = []
    out = schedule(handles)
    handles.clear()                              # nothing holds the ops between
    got = out.resolve().to_numpy()
    assert dev.launches - launches == (1 if T * C < 1 << 18 else 4 if half else 3)
    assert got.dtype == (np.float16 if half else np.float32) and np.array_equal(got, want)
