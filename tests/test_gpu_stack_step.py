"""The fused decode step where the staging of a product's inputs changes its form: vectors that do not start on sixteen bytes, second inputs
of more than one batch of loads, the token's latent written beside the query expansion, and latent attention merged in clusters."""
import numpy as np
import pytest

from oracle import dadezen_plain as dz

from . import dadezen_builders as B

pytestmark = pytest.mark.gpu

# the bound of the bf16 model tests (root mean square over the logits'): bf16 cached rows and 16-bit activations through two layers
LIMIT = 4e-2
MODELS = {
    # a gate that starts at 2 * 63 + 64 floats: rows of whole blocks behind unaligned vectors
    "unaligned": B.config(128, 64, [B.lightning(1, 63, 64, (0.9,), ff=192), B.latent(2, 30, 6, 32, 64, 64, 5, 0.2, ff=64)]),
    # runs of positions in clusters of eight: 17 splits (the last cluster's others without a position), ranks that are no multiple of 16, a window of which
    # only the first runs have positions
    "clusters": B.config(64, 64, [B.latent(3, 16, 8, 16, 64, 1000, 272, 0.2, scaling=B.YARN), B.latent(17, 8, 4, 8, 64, 512, 1024, 0.25, scaling=B.YARN)]),
    # 8256 = 8192 + 64 activations of a feed-forward: more than a batch takes
    "long": B.config(64, 64, [B.lightning(2, 32, 32, (0.8, 0.99), ff=8256), B.latent(4, 16, 8, 16, 128, 192, 21, 0.25, scaling=B.YARN, ff=8192)]),
}


@pytest.mark.parametrize("name", sorted(MODELS))
def test_tokens_agree_with_the_restatement(name, tmp_path):
    from ratchet_b200 import Device
    from ratchet_b200.models import load_model
    cfg = MODELS[name]
    W = B.weights(cfg, seed=5)
    tokens = np.random.Generator(np.random.PCG64(3)).integers(0, cfg["vocab"], 300 if name == "clusters" else 40).tolist()
    want = dz.forward(cfg, W, tokens)
    dev = Device(0)
    try:
        m = load_model(B.write_model(str(tmp_path / name), cfg, W), dev, "bfloat16")
        st = m.new_state(len(tokens))
        got = np.concatenate([m.decode(st, t)[0].to_numpy() for t in tokens])
    finally:
        dev.close()
    assert np.sqrt(((got - want) ** 2).mean(-1) / (want ** 2).mean()).max() < LIMIT


def test_runs_that_share_a_state(tmp_path):
    """Two layers over one state: the second's step must see what the first's has written (states are otherwise read ahead of the kernel before)."""
    from ratchet_b200 import Device
    from ratchet_b200.models import load_model
    cfg = B.config(64, 64, [B.lightning(2, 32, 32, (0.8, 0.99), ff=64), B.lightning(2, 32, 32, (0.8, 0.99), ff=64)])
    W = B.weights(cfg, seed=6)
    dev = Device(0)
    try:
        m = load_model(B.write_model(str(tmp_path / "shared"), cfg, W), dev, "bfloat16")
        tokens = [5, 9, 60, 2, 33, 7, 7, 1]
        got = []
        for step in (lambda st, t: m.prefill([t], st, [0]), lambda st, t: m.decode(st, t)[0].to_numpy()):      # op by op, and the fused step
            st = m.new_state(len(tokens))
            st.runs[1] = st.runs[0]
            got.append(np.concatenate([step(st, t) for t in tokens]))
    finally:
        dev.close()
    assert np.sqrt(((got[1] - got[0]) ** 2).mean(-1) / (got[0] ** 2).mean()).max() < LIMIT
    assert np.sqrt(((got[0][1:] - got[0][:-1]) ** 2).mean()) > LIMIT


@pytest.mark.parametrize("vocab", [3, 4097, 33000])
def test_the_picked_token_is_the_first_maximum(tmp_path, vocab):
    """Vocabularies of less and more than a round of the cluster's threads; equal logits: the lowest id."""
    from ratchet_b200 import Device
    from ratchet_b200.models import load_model
    cfg = B.config(64, vocab, [B.lightning(2, 32, 32, (0.8, 0.99), ff=64)])
    W = B.weights(cfg, seed=vocab)
    W["head"][vocab // 2:] = W["head"][:vocab - vocab // 2]              # every logit of the first half comes again
    dev = Device(0)
    try:
        m = load_model(B.write_model(str(tmp_path / "v"), cfg, W), dev, "bfloat16")
        st = m.new_state(8)
        for t in (0, 1, 2, 1):
            logits, picked = m.decode(st, t)
            assert int(picked.to_numpy()[0]) == int(np.argmax(logits.to_numpy().reshape(-1)))
    finally:
        dev.close()
