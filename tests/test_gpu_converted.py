"""Small quantised weights of a prompt are converted in one launch: the same bits as with a conversion beside every product."""
import numpy as np
import pytest

from ratchet_b200 import capi, nn

pytestmark = pytest.mark.gpu


# more matrices than one launch holds, one that two products share, a large one that stays beside its product, rows below and above the rule
@pytest.mark.parametrize("dt", [capi.Q8_0H, capi.Q8_0F])
@pytest.mark.parametrize("M", [40, 257, 400])
def test_same_bits(dt, M):
    from oracle import oracle as orc
    from ratchet_b200 import Device, Tensor
    dev, act = Device(0), np.float16 if dt == capi.Q8_0H else np.float32
    try:
        g = np.random.Generator(np.random.PCG64(M))
        shapes = [(96, 96)] * 33 + [(160, 96), (96, 160), (11200, 96), (96, 11200)]
        quant = orc.quantize_q8 if dt == capi.Q8_0H else lambda w: orc.quantize_q8(w.astype(np.float32))
        ws = [Tensor.from_quantized(quant((g.standard_normal(s) / np.sqrt(s[1])).astype(act)), dt, s, dev) for s in shapes]
        b = Tensor.from_data(g.standard_normal(96).astype(np.float32), device=dev)
        x = g.standard_normal((1, M, 96)).astype(act)

        def build():
            h = Tensor.from_data(x, device=dev)
            for w in ws[:33] + ws[:1]:
                h = nn.Linear(w, b).schedule(h)
            for w in ws[33:]:
                h = nn.Linear(w).schedule(h)
            return h

        out = build().resolve()
        launches, got = dev.launches, out.to_numpy()
        dev.set_debug(no_reuse=True)
        want = build().resolve().to_numpy()
        dev.set_debug()
        before = dev.launches
        again = build().resolve().to_numpy()
        fused = dev.launches - before
        dev.set_debug(no_reuse=True)
        before = dev.launches
        build().resolve()
        assert np.array_equal(got, want) and np.array_equal(again, want) and np.isfinite(want).all()
        assert fused < dev.launches - before - (30 if M > 256 or dt == capi.Q8_0F else 0)
    finally:
        dev.close()


@pytest.mark.parametrize("dt", [capi.Q8_0H, capi.Q8_0F])
@pytest.mark.parametrize("few", [1, 2, 16])
def test_a_product_of_few_rows_over_a_converted_matrix(dt, few):
    """It reads the codes, as it does where no other product has the matrix converted."""
    from oracle import oracle as orc
    from ratchet_b200 import Device, Tensor
    dev, act = Device(0), np.float16 if dt == capi.Q8_0H else np.float32
    try:
        g = np.random.Generator(np.random.PCG64(few))
        raw = [orc.quantize_q8((g.standard_normal((96, 96)) / 10).astype(act)) for _ in range(2)]
        ws = [Tensor.from_quantized(r, dt, (96, 96), dev) for r in raw]
        many, one = (Tensor.from_data(g.standard_normal((1, m, 96)).astype(act), device=dev) for m in (300, few))

        def build():
            h = nn.Linear(ws[1]).schedule(nn.Linear(ws[0]).schedule(many))
            return h.slice([(0, 1), (0, few), (0, 96)]).add(nn.Linear(ws[0]).schedule(one))

        for _ in range(20):
            got = build().resolve().to_numpy()
            dev.set_debug(no_reuse=True)
            want = build().resolve().to_numpy()
            dev.set_debug()
            assert np.array_equal(got, want)
    finally:
        dev.close()
