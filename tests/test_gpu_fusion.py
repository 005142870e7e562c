"""Subgraphs of an f16 prompt that the resolver runs as one kernel, against the same graph with one kernel per op (the debug switch that
gives every tensor its own buffer) and, for attention, against a float64 evaluation.

Bounds: norms, activations, gates, rotations and copies are the same arithmetic, so the same bits - except where the compiler contracts
a product and a sum of the f32 norm, one ulp of f32 before the rounding to f16 (one ulp of f16 at most, rarely).  Attention: the graph
rounds scores and weights to f16 (2^-11 each); with scores up to about 8 that is 8 * 2^-11 in the exponent."""
import numpy as np
import pytest

from ratchet_b200 import callers, capi, nn
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
    """(fused result, names of its kernels, result with one kernel per op); build() makes the graph and returns (output, caches)."""
    res = []
    for no_reuse in (False, True):
        out, caches = build()
        dev.set_debug(no_reuse=no_reuse, profile=True)
        try:
            dev.profile_report()
            out.resolve()
            names = [ln.rsplit(None, 4)[0] for ln in dev.profile_report().splitlines()[1:]]
        finally:
            dev.set_debug()
        res.append((out.to_numpy().astype(np.float64), [c.to_numpy() for c in caches], names))
    return res


def tensor(dev, a):
    from ratchet_b200 import Tensor
    return Tensor.from_data(np.ascontiguousarray(a), device=dev)


def close(got, want, what, tol=1e-2):
    scale = np.sqrt(np.mean(want * want)) + 1e-30
    assert np.abs(got - want).max() < tol * (scale + np.abs(want)).max(), (what, np.abs(got - want).max(), scale)


def causal(T, L):
    return np.triu(np.full((T, L), -65504.0, F16), 1 + L - T)


# positions beside the tiles of 128 queries and 64 keys, one and two query tiles, rows of an odd length (padded mask), head sizes of one and two
# 64-column blocks with and without a remainder
@pytest.mark.parametrize("T,prior,H,D", [(2, 0, 2, 64), (3, 4, 1, 96), (63, 0, 2, 16), (64, 1, 2, 128), (65, 0, 3, 96), (128, 0, 2, 80), (129, 7, 2, 96),
                                         (200, 0, 2, 64), (256, 0, 2, 96), (257, 0, 2, 96), (300, 33, 2, 48), (520, 0, 2, 96)])
def test_attention_over_a_cache_with_mask(dev, T, prior, H, D):
    g = np.random.Generator(np.random.PCG64(T * 5 + D))
    d, L = H * D, T + prior
    rd = D // 16 * 16
    x = g.standard_normal((1, T, d)).astype(F16)
    wqkv, wo = (g.standard_normal((3 * d, d)) * 2 / np.sqrt(d)).astype(F16), np.eye(d, dtype=F16)
    kc, vc = np.zeros((1, H, L + 9, D), F16), np.zeros((1, H, L + 9, D), F16)
    kc[:, :, :prior], vc[:, :, :prior] = g.standard_normal((1, H, prior, D)), g.standard_normal((1, H, prior, D))
    mask = causal(T, L)
    if T > 100:
        mask[5] = -65504.0                       # nothing to see: the average of all values

    def build():
        k, v = tensor(dev, kc), tensor(dev, vc)
        attn = callers.Phi3SelfAttention(nn.Linear(tensor(dev, wqkv)), nn.Linear(tensor(dev, wo)), nn.RotaryEmbedding(rd, False, 10000.0, 1.0), H, H,
                                         tensor(dev, np.array([D ** -0.5], np.float32)))
        return attn.schedule(tensor(dev, x), tensor(dev, mask), nn.KVEntry(k, v, prior)), (k, v)

    (got, caches, names), (want, caches0, names0) = both(dev, build)
    assert any(n.startswith("attention") for n in names) and not any(n.startswith("softmax") for n in names), names
    assert any(n.startswith("softmax") for n in names0)
    close(got, want, (T, prior, H, D))
    for a, b in zip(caches, caches0):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("T,H,D", [(2, 2, 64), (100, 6, 64), (129, 3, 64), (501, 6, 64), (300, 2, 128), (70, 2, 72)])
def test_attention_with_scaled_operands(dev, T, H, D):
    g = np.random.Generator(np.random.PCG64(T + D))
    d = H * D
    x = g.standard_normal((1, T, d)).astype(F16)
    ws = [(g.standard_normal((d, d)) * 1.5 / np.sqrt(d)).astype(F16) for _ in range(3)] + [np.eye(d, dtype=F16)]

    def build():
        mha = callers.WhisperMHA(*[nn.Linear(tensor(dev, w)) for w in ws], H, tensor(dev, np.array([float(D) ** -0.25], F16)))
        return mha.schedule(tensor(dev, x)), ()

    (got, _, names), (want, _, _) = both(dev, build)
    assert any(n.startswith("attention") for n in names) and not any(n.startswith("softmax") for n in names), names
    close(got, want, (T, H, D))
    x64 = x[0].astype(np.float64)
    q, k, v = ((x64 @ w.astype(np.float64).T).astype(F16).astype(np.float64).reshape(T, H, D).transpose(1, 0, 2) for w in ws[:3])
    z = q @ k.transpose(0, 2, 1) * D ** -0.5
    p = np.exp(z - z.max(-1, keepdims=True))
    ref = ((p / p.sum(-1, keepdims=True)) @ v).transpose(1, 0, 2).reshape(1, T, d)
    assert np.linalg.norm(got - ref) <= 1.05 * np.linalg.norm(want - ref) + 1e-4 * np.linalg.norm(ref)


def test_scores_beyond_f16_behave_as_in_the_graph(dev):
    """A score that f16 cannot hold, and NaN in a value, reach the rows they reach with one kernel per op."""
    T, H, D = 130, 1, 64
    g = np.random.Generator(np.random.PCG64(1))
    q, k, v = (g.standard_normal((1, H, T, D)).astype(F16) for _ in range(3))
    q[0, 0, 3], k[0, 0, 2] = 60.0, 60.0
    v[0, 0, 120, 5] = np.nan

    def build():
        z = tensor(dev, q).full().matmul(tensor(dev, k).full(), False, True).mul(tensor(dev, np.array([1.0], np.float32))).cast(capi.F16)
        w = z.add(tensor(dev, causal(T, T))).full().softmax(3).cast(capi.F16)
        return w.matmul(tensor(dev, v), False, False).permute([0, 2, 1, 3]), ()

    (got, _, names), (want, _, _) = both(dev, build)
    assert any(n.startswith("attention") for n in names)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    close(np.nan_to_num(got), np.nan_to_num(want), "large")


# what a source has where the cache has one batch entry, two heads of 64
@pytest.mark.parametrize("B,H,D", [(1, 1, 64), (1, 4, 64), (1, 2, 32), (1, 2, 128), (2, 2, 64)])
@pytest.mark.parametrize("rotated", [False, True])
def test_a_source_that_differs_from_its_cache_is_refused(dev, B, H, D, rotated):
    T, h, d = 40, 2, 64
    g = np.random.Generator(np.random.PCG64(H * D))
    held = [tensor(dev, g.standard_normal((1, h, 48, d)).astype(F16)) for _ in range(2)]
    before = [c.to_numpy() for c in held]
    q = tensor(dev, g.standard_normal((1, h, T, d)).astype(F16))
    scale, rows = tensor(dev, np.array([0.125], np.float32)), g.standard_normal((B, T, H * D)).astype(F16)

    def source():
        s = tensor(dev, rows).view([B, T, H, D]).permute([0, 2, 1, 3])
        return s.full().rope(32, 10000.0, 0).half() if rotated else s

    k = held[0].cache(source(), 2, 0)
    v = held[1].cache(source(), 2, 0)
    z = q.full().matmul(k.full(), False, True).mul(scale).half()
    del k
    out = z.full().softmax(3).half().matmul(v, False, False).permute([0, 2, 1, 3])
    del z, v
    with pytest.raises(RatchetCudaError, match="source differs from cache"):
        out.resolve()
    for c, b in zip(held, before):
        assert np.array_equal(c.to_numpy(), b)


@pytest.mark.parametrize("dim", [0, 15, 80])
@pytest.mark.parametrize("cached", [False, True])
def test_a_rotation_of_no_features_or_too_many_is_refused(dev, dim, cached):
    T, H, D = 24, 2, 64
    g = np.random.Generator(np.random.PCG64(dim))
    q, v, rows = (tensor(dev, g.standard_normal(s).astype(F16)) for s in ((1, H, T, D), (1, H, T, D), (1, T, H * D)))
    k = rows.view([1, T, H, D]).permute([0, 2, 1, 3]).full().rope(dim, 10000.0, 0).half()
    if cached:
        held = tensor(dev, np.zeros((1, H, 32, D), F16))
        z = q.full().matmul(held.cache(k, 2, 0).full(), False, True).mul(tensor(dev, np.array([0.125], np.float32))).half()
        del k
        out = z.full().softmax(3).half().matmul(v, False, False).permute([0, 2, 1, 3])
        del z
    else:
        out = k
    with pytest.raises(RatchetCudaError, match="rope: dim must be even"):
        out.resolve()


# who appends: two caches; both to one; both to one, the second through a view; one whose rows are the queries
@pytest.mark.parametrize("caches", ["apart", "one", "view", "late view", "queries"])
def test_attention_over_caches_that_share_memory(dev, caches):
    T, H, D, cap = 70, 2, 64, 70 if caches == "queries" else 80
    g = np.random.Generator(np.random.PCG64(9))
    arrays = [g.standard_normal((1, H, n, D)).astype(F16) for n in (T, T, T, cap, cap)]
    scale = tensor(dev, np.array([0.125], np.float32))

    def build():
        q, ks, vs, kc, vc = (tensor(dev, a) for a in arrays)
        held = [kc, vc]
        if caches in ("one", "view"):
            vc = kc if caches == "one" else kc.view([1, H, cap, D])
            held = [kc]
        if caches == "late view":                     # a view made before its tensor was there
            kc = kc.mul(tensor(dev, np.array([1.0], F16)))
            vc = kc.view([1, H, cap, D])
            kc.resolve()
            held = [kc]
        if caches == "queries":
            q = kc
        z = q.full().matmul(kc.cache(ks, 2, 0).full(), False, True).mul(scale).half()
        return z.full().softmax(3).half().matmul(vc.cache(vs, 2, 0), False, False).permute([0, 2, 1, 3]), held

    (got, held, names), (want, held0, _) = both(dev, build)
    assert any(n.startswith("attention") for n in names) == (caches != "queries"), names
    close(got, want, caches)
    for a, b in zip(held, held0):
        assert np.array_equal(a, b)


def test_an_operand_that_is_written_before_the_op_runs(dev):
    """x W^T + r, where computing r appends to x: the product sees x as it was, as it does with one kernel per op."""
    T, d = 64, 128
    g = np.random.Generator(np.random.PCG64(10))
    x, w, new = g.standard_normal((1, T, d)).astype(F16), (g.standard_normal((d, d)) / 11).astype(F16), g.standard_normal((1, T, d)).astype(F16)

    def build():
        held, wt = tensor(dev, x), tensor(dev, w)
        h = wt.gemm(held, None, False, True, True)
        r = held.cache(tensor(dev, new), 1, 0)
        return h.add(r), [held]

    (got, held, _), (want, held0, _) = both(dev, build)
    assert np.array_equal(got, want) and np.array_equal(held[0], held0[0]) and np.array_equal(held[0], new)
    close(got, x[0].astype(np.float64) @ w.astype(np.float64).T + new, "product", 1e-2)


def test_held_tensors_are_computed(dev):
    """A score matrix or a cache's result that the caller keeps is there afterwards: no fusion passes over it."""
    T, H, D = 40, 2, 64
    g = np.random.Generator(np.random.PCG64(2))
    q, k, v = (tensor(dev, g.standard_normal((1, H, T, D)).astype(F16)) for _ in range(3))
    cache = tensor(dev, np.zeros((1, H, 64, D), F16))
    kk = cache.cache(k, 2, 0)
    z = q.full().matmul(kk.full(), False, True).mul(tensor(dev, np.array([0.125], np.float32))).cast(capi.F16)
    out = z.full().softmax(3).cast(capi.F16).matmul(v, False, False).permute([0, 2, 1, 3]).resolve()
    assert z.resolved() and kk.resolved() and out.shape() == (1, T, H, D)
    assert np.array_equal(kk.to_numpy(), k.to_numpy())
    # a later graph over the results does not run the first one again
    before = dev.launches
    out.full().resolve()
    assert dev.launches - before == 1


@pytest.mark.parametrize("rows,N", [(2, 8), (3, 384), (7, 2048), (5, 2056), (9, 3072), (2, 8192), (4, 8200), (3, 100)])
@pytest.mark.parametrize("kind", ["layer", "rms"])
def test_norm_between_casts(dev, rows, N, kind):
    g = np.random.Generator(np.random.PCG64(rows + N))
    x, s, b = (g.standard_normal((1, rows, N)) * 3 + 1).astype(F16), g.standard_normal(N).astype(np.float32), g.standard_normal(N).astype(np.float32)

    def build():
        m = nn.LayerNorm(tensor(dev, s), tensor(dev, b), 1e-5) if kind == "layer" else nn.RMSNorm(tensor(dev, s), 1e-5)
        return m.schedule(tensor(dev, x)), ()

    (got, _, names), (want, _, _) = both(dev, build)
    assert any(n.startswith("norm chain") for n in names) == (N % 8 == 0 and N <= 8192), names
    off = np.abs(got - want) > 0
    assert off.mean() < 0.01 and np.abs(got - want).max() <= 2.0 ** -10 * np.abs(want).max()


@pytest.mark.parametrize("shape", [(1, 2, 8), (1, 5, 24), (2, 33, 1536)])
def test_activation_and_gate_between_casts(dev, shape):
    g = np.random.Generator(np.random.PCG64(shape[-1]))
    x = (g.standard_normal(shape) * 3).astype(F16)
    x[0, 0, :4] = [np.inf, -np.inf, np.nan, -65504.0]
    F = shape[-1] // 2
    for fn in (lambda t: t.full().gelu().cast(capi.F16), lambda t: t.full().silu().cast(capi.F16)):
        (got, _, names), (want, _, _) = both(dev, lambda: (fn(tensor(dev, x)), ()))
        assert any(n.startswith("act chain") for n in names) and np.array_equal(got, want, equal_nan=True)

    def gate():
        t = tensor(dev, x)
        whole = [(0, n) for n in shape[:-1]]
        return t.slice(whole + [(F, 2 * F)]).mul(t.slice(whole + [(0, F)]).full().silu().cast(capi.F16)), ()

    (got, _, names), (want, _, _) = both(dev, gate)
    assert any(n.startswith("glu chain") for n in names) == (F % 8 == 0) and np.array_equal(got, want, equal_nan=True)


def test_a_prompt_on_a_device_that_is_not_the_current_one():
    import torch
    from ratchet_b200 import Device
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    torch.cuda.set_device(0)
    other, x = Device(1), np.random.Generator(np.random.PCG64(4)).standard_normal((1, 40, 128)).astype(F16)
    try:
        mha = callers.WhisperMHA(*[nn.Linear(tensor(other, np.eye(128, dtype=F16))) for _ in range(4)], 2, tensor(other, np.array([0.35], F16)))
        assert np.isfinite(mha.schedule(nn.RMSNorm(tensor(other, np.ones(128, np.float32)), 1e-5).schedule(tensor(other, x))).resolve().to_numpy()).all()
        assert torch.cuda.current_device() == 0
    finally:
        other.close()
