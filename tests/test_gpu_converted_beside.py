"""Large Q8_0 weights of a resolve: converted beside the product before their own.  Bit for bit what the products give one resolve at a time, where
each converts its own matrix first; and where the pool has no room for the two blocks, each converts its own as well."""
import re

import numpy as np
import pytest

from ratchet_b200 import Tensor, capi, nn
from ratchet_b200.tensor import last_resolve_stats

from .test_gpu_gemm_pair_quant import codes

pytestmark = pytest.mark.gpu

F16 = np.float16
MIB = 1 << 20


def beside(capfd):
    """Conversions beside a product that the last logged resolve has started."""
    return int(re.findall(r"(\d+) weights converted beside", capfd.readouterr().err)[-1])


# matrices (out, in) of a chain over the rows; the second and third are the same one, so both blocks hold it in turn; a small one in between
# (its product takes the one-CTA kernel); rows that do not start on a block of 32; too few tiles for the pair kernel in all products but one
@pytest.mark.parametrize("M,dims,shared,conversions", [(1000, [512, 2560, 512 * 5, 2560, 2560], True, 3), (600, [2048, 4864, 256, 4864, 3328], False, 2), (700, [1024, 3400, 3400, 5000], False, 2),
                                                       (700, [1024, 2600, 1024, 5000], False, 0)])
def test_equals_one_resolve_per_product(M, dims, shared, conversions, capfd):
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
            dev.set_debug(log=True)
            capfd.readouterr()
            h = h.resolve()
            assert beside(capfd) == conversions
            dev.set_debug()
            got, want = h.to_numpy(), want.to_numpy()
            assert np.isfinite(want).all() and np.array_equal(got.view(np.uint16), want.view(np.uint16))
    finally:
        dev.close()


# Three gated products of 5120 x 2560: 25 MiB each once converted, and a gate wants that (the one-CTA kernel has none).  Room for one converted matrix and a half: the
# second block is not had.  Room for two and a half and the last matrix a Q4_KH one, which needs scratch of its own: the two blocks are given back for it (in the
# middle: with the third matrix converted in one of them).  3.5: room for all.
@pytest.mark.parametrize("kinds,room,conversions", [("888", 1.5, 0), ("888", 2.5, 2), ("884", 2.5, 1), ("884", 3.5, 1), ("848", 2.5, 1), ("848", 3.5, 1)])
def test_a_prompt_that_has_room_for_one_converted_matrix(kinds, room, conversions, monkeypatch, capfd):
    from ratchet_b200 import Device
    M, F, K = 1000, 2560, 2560
    block = -(-2 * F * K * 2 // MIB) * MIB
    g = np.random.Generator(np.random.PCG64(7))
    held = [codes(g, "q8_0h" if kind == "8" else "q4_kh", 2 * F, K) for kind in kinds]
    x = (g.standard_normal((1, M, K)) * 0.1).astype(F16)
    results, limit = [], None
    for _ in range(2):                           # without a limit, and with one
        if limit:
            monkeypatch.setenv("RCU_POOL_LIMIT", str(limit))
        dev = Device(0)
        try:
            h = Tensor.from_data(x, device=dev)
            weights = [Tensor.from_quantized(raw, dt, (2 * F, K), dev) for raw, dt in held]
            before = dev.pool_stats()[1]
            for w in weights:
                rows = nn.Linear(w).schedule(h)
                up, gate = rows.slice([(0, 1), (0, M), (F, 2 * F)]), rows.slice([(0, 1), (0, M), (0, F)])
                h = up.mul(gate.full().silu().cast(capi.F16))
            del rows, up, gate                   # nothing holds the ops between
            dev.set_debug(log=True)
            capfd.readouterr()
            h = h.resolve()
            n = beside(capfd)
            results.append(h.to_numpy())
            assert dev.pool_stats()[1] <= (limit or 1 << 40)
            stats = last_resolve_stats(dev)
            limit = before + stats["planned_bytes"] + stats["buffers"] * MIB + int(room * block)
        finally:
            dev.close()
    assert n == conversions
    assert np.isfinite(results[0]).all() and np.array_equal(results[0].view(np.uint16), results[1].view(np.uint16))
