"""What an f16 graph has behind a Linear, in the product's epilogue, against the same graph with one kernel per op.  Same products, same roundings: the
same bits."""
import numpy as np
import pytest

from ratchet_b200 import capi, nn
from ratchet_b200.capi import RatchetCudaError

pytestmark = pytest.mark.gpu
F16 = np.float16


@pytest.fixture(scope="module")
def dev():
    from ratchet_b200 import Device
    d = Device(0)
    yield d
    d.close()


def both(dev, build):
    """(result, kernels) fused and with one kernel per op"""
    res = []
    for no_reuse in (False, True):
        out = build()
        dev.set_debug(no_reuse=no_reuse, profile=True)
        try:
            dev.profile_report()
            out.resolve()
            names = [ln.rsplit(None, 4)[0] for ln in dev.profile_report().splitlines()[1:]]
        finally:
            dev.set_debug()
        res.append((out.to_numpy(), names))
    return res


def tensor(dev, a):
    from ratchet_b200 import Tensor
    return Tensor.from_data(np.ascontiguousarray(a), device=dev)


def weight(dev, g, dt, n, k):
    from oracle import oracle as orc
    from ratchet_b200 import Tensor
    w = (g.standard_normal((n, k)) / np.sqrt(k)).astype(F16)
    return tensor(dev, w) if dt == "f16" else Tensor.from_quantized(orc.quantize_q8(w), capi.Q8_0H, (n, k), dev)


# few and many tiles, K in slices (1024 and more), rows beside the tiles of 128 and 256, the pair kernel, converted and fused quantised weights
@pytest.mark.parametrize("dt,M,N,K", [("f16", 33, 64, 64), ("f16", 129, 384, 1536), ("f16", 501, 1536, 384), ("f16", 600, 4104, 256), ("f16", 2049, 1280, 96),
                                      ("q8_0h", 40, 384, 384), ("q8_0h", 255, 136, 1024), ("q8_0h", 501, 384, 384), ("q8_0h", 1000, 3072, 512)])
@pytest.mark.parametrize("what", ["bias", "bias+gelu", "silu", "bias+resid", "resid first"])
def test_linear_and_what_follows(dev, dt, M, N, K, what):
    g = np.random.Generator(np.random.PCG64(M + N))
    x, r, b = g.standard_normal((1, M, K)).astype(F16), g.standard_normal((1, M, N)).astype(F16), g.standard_normal(N).astype(np.float32)
    x[0, 0, 0], r[0, 1, 2] = np.inf, np.nan
    w = weight(dev, g, dt, N, K)

    def build():
        h = nn.Linear(w, tensor(dev, b) if "bias" in what else None).schedule(tensor(dev, x))
        if "gelu" in what:
            return h.full().gelu().cast(capi.F16)
        if "silu" in what:
            return h.full().silu().cast(capi.F16)
        if "resid" in what:
            return tensor(dev, r).add(h) if "first" in what else h.add(tensor(dev, r))
        return h

    (got, names), (want, names0) = both(dev, build)
    assert any(n.startswith("linear chain") for n in names) or "lu" in what, names
    assert not any(n.startswith(("binary", "unary")) for n in names), names
    assert any(n.startswith("matmul") for n in names0)
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.parametrize("dt,M,F,K", [("f16", 256, 4736, 64), ("f16", 1000, 1288, 512), ("q8_0h", 700, 1600, 512), ("bf16", 600, 1544, 256), ("bf16", 2049, 640, 128)])
def test_product_of_a_gate(dev, dt, M, F, K):
    """Gate and up columns beside the tiles of 128."""
    from ratchet_b200 import Tensor
    g = np.random.Generator(np.random.PCG64(M + F))
    x = g.standard_normal((1, M, K)).astype(np.float32)
    if dt == "bf16":
        w = Tensor.from_data(capi.to_bf16((g.standard_normal((2 * F, K)) / np.sqrt(K)).astype(np.float32)), device=dev, dt=capi.BF16)
        build = lambda: w.linear(tensor(dev, x[0]).cast(capi.BF16)).glu("gelu").full()
    else:
        w = weight(dev, g, dt, 2 * F, K)

        def build():
            h = nn.Linear(w).schedule(tensor(dev, x.astype(F16)))
            return h.slice([(0, 1), (0, M), (F, 2 * F)]).mul(h.slice([(0, 1), (0, M), (0, F)]).full().silu().cast(capi.F16))

    (got, names), (want, _) = both(dev, build)
    assert any(n.startswith("linear chain") for n in names) and not any(n.startswith(("matmul", "linear b", "glu")) for n in names), names
    assert np.array_equal(got, want, equal_nan=True)


def test_a_product_that_is_kept_is_computed(dev):
    """A caller's handle on the product, or a second consumer, leaves the ops apart."""
    g = np.random.Generator(np.random.PCG64(3))
    w, x = weight(dev, g, "f16", 128, 128), tensor(dev, g.standard_normal((1, 64, 128)).astype(F16))
    h = nn.Linear(w).schedule(x)
    y = h.add(x).resolve().to_numpy()
    assert h.resolved() and np.array_equal(y, (h.to_numpy().astype(np.float32) + x.to_numpy()).astype(F16))
    h = nn.Linear(w).schedule(x)
    z = h.full().gelu().cast(capi.F16).add(h)
    del h
    assert np.isfinite(z.resolve().to_numpy()).all()


# rows on either side of the rule that the switch overrides, as many columns as the pair kernel wants
@pytest.mark.parametrize("fused", ["0", "1"])
@pytest.mark.parametrize("M,F,K", [(256, 4752, 64), (600, 1600, 512)])
@pytest.mark.parametrize("what", ["gate", "gelu", "resid"])
def test_with_the_conversion_forced(dev, monkeypatch, fused, M, F, K, what):
    monkeypatch.setenv("RCU_GEMM_FUSED", fused)
    g = np.random.Generator(np.random.PCG64(M))
    w, x, r = weight(dev, g, "q8_0h", 2 * F, K), g.standard_normal((1, M, K)).astype(F16), g.standard_normal((1, M, 2 * F)).astype(F16)

    def build():
        h = nn.Linear(w).schedule(tensor(dev, x))
        if what == "gelu":
            return h.full().gelu().cast(capi.F16)
        if what == "resid":
            return h.add(tensor(dev, r))
        return h.slice([(0, 1), (0, M), (F, 2 * F)]).mul(h.slice([(0, 1), (0, M), (0, F)]).full().silu().cast(capi.F16))

    (got, _), (want, _) = both(dev, build)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("M", [20, 64, 600])
@pytest.mark.parametrize("what", ["alone", "gelu", "resid"])
def test_a_bias_of_another_type_is_refused(dev, M, what):
    g = np.random.Generator(np.random.PCG64(M))
    N, K = 3328, 128
    w, x = weight(dev, g, "f16", N, K), tensor(dev, g.standard_normal((1, M, K)).astype(F16))
    h = w.gemm(x, tensor(dev, g.standard_normal(N).astype(np.float32)), False, True, True)
    if what == "gelu":
        h = h.full().gelu().cast(capi.F16)
    if what == "resid":
        h = h.add(tensor(dev, g.standard_normal((1, M, N)).astype(F16)))
    with pytest.raises(RatchetCudaError, match="DType mismatch: bias"):
        h.resolve()


@pytest.mark.parametrize("kw", [{"act_cols": 3096}, {"act": "softcap", "act_cols": 0}])
def test_what_linear_refuses_is_refused_in_front_of_a_gate(dev, kw):
    """More activated columns than there are; a softcap without its parameter."""
    from ratchet_b200 import Tensor
    g = np.random.Generator(np.random.PCG64(5))
    w = Tensor.from_data(capi.to_bf16(g.standard_normal((3088, 256)).astype(np.float32)), device=dev, dt=capi.BF16)
    x = tensor(dev, g.standard_normal((1000, 256)).astype(np.float32)).cast(capi.BF16)
    with pytest.raises(RatchetCudaError, match="linear: "):
        w.linear(x, **kw).glu("gelu").resolve()
