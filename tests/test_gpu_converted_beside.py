"""Large Q8_0 weights of a resolve: converted beside the product before their own.  Bit for bit what the products give one resolve at a time, where
each converts its own matrix first."""
import numpy as np
import pytest

from ratchet_b200 import Tensor, capi, nn

from .test_gpu_gemm_pair_quant import codes

pytestmark = pytest.mark.gpu

F16 = np.float16


# matrices (out, in) of a chain over the rows; the first and third are the same one, so both blocks hold it in turn; a small one in between, and
# one whose product takes the one-CTA kernel (few tiles: its successor is then converted by itself)
@pytest.mark.parametrize("M,dims,shared", [(1000, [512, 2560, 512 * 5, 2560, 2560], True), (600, [2048, 4864, 256, 4864, 3328], False), (700, [1024, 2600, 1024, 5000], False)])
def test_equals_one_resolve_per_product(M, dims, shared):
    from ratchet_b200 import Device
    dev = Device(0)
    try:
        g = np.random.Generator(np.random.PCG64(M))
        held = [codes(g, "q8_0h", n, k) for k, n in zip(dims, dims[1:])]
        if shared:
            held[2] = held[1]
        weights = [Tensor.from_quantized(raw, dt, (n, k), dev) for (raw, dt), k, n in zip(held, dims, dims[1:])]
        if shared:
            weights[2] = weights[1]
        x = Tensor.from_data((g.standard_normal((1, M, dims[0])) * 0.1).astype(F16), device=dev)
        for _ in range(3):                       # the pool's blocks of the passes before
            h, want = x, x
            for w in weights:
                h = nn.Linear(w).schedule(h)
                want = nn.Linear(w).schedule(want).resolve()
            got, want = h.resolve().to_numpy(), want.to_numpy()
            assert np.isfinite(want).all() and np.array_equal(got.view(np.uint16), want.view(np.uint16))
    finally:
        dev.close()
