"""Attention of an f16 prompt gives the same bits every time: its pieces of the mask are replaced while the kernel runs, and a piece that is replaced
before every warp has read it shows in a few passes of a hundred."""
import numpy as np
import pytest

from ratchet_b200 import callers, nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [199, 200, 330])
def test_repeated_passes_agree(T):
    from ratchet_b200 import Device, Tensor
    H, D = 2, 64
    d, g = H * D, np.random.Generator(np.random.PCG64(T))
    x, w = g.standard_normal((1, T, d)).astype(np.float16), (g.standard_normal((3 * d, d)) * 2 / np.sqrt(d)).astype(np.float16)
    mask = np.triu(np.full((T, T), -65504.0, np.float16), 1)
    dev = Device(0)
    try:
        t = lambda a: Tensor.from_data(a, device=dev)
        w, eye, scale = t(w), t(np.eye(d, dtype=np.float16)), t(np.array([D ** -0.5], np.float32))
        first = None
        for _ in range(300):
            cache = nn.KVEntry(t(np.zeros((1, H, T, D), np.float16)), t(np.zeros((1, H, T, D), np.float16)))
            attn = callers.Phi3SelfAttention(nn.Linear(w), nn.Linear(eye), nn.RotaryEmbedding(D, False, 10000.0, 1.0), H, H, scale)
            got = attn.schedule(t(x), t(mask), cache).resolve().to_numpy()
            first = got if first is None else first
            assert np.array_equal(got, first)
    finally:
        dev.close()
