"""The work whose speed counts: single matrix products as a host program asks for them through the C ABI, the forwards of the
models that ratchet runs (Phi-2's MLP block, Whisper's encoder, Phi-3), and the two served decoders, each over the sizes that it meets.

A case is a dict of plain values.  `prepare` makes what a program holds before the call (weights loaded, caches and handles made),
`run` is one pass, `exact` the same result in 64 bits by plain torch.  Weights and inputs are random: N(0, 0.02) matrices and N(0, 1)
activations, or codes and block scales that give such matrices."""
import ctypes
import math

import numpy as np
import torch

from ratchet_b200 import Device, Tensor, callers, capi, nn
from ratchet_b200.decoder import Decoder, DecoderConfig, DecoderLayer
from ratchet_b200.models import REGISTRY

DT = {"f32": capi.F32, "f16": capi.F16, "q8_0f": capi.Q8_0F, "q8_0h": capi.Q8_0H, "q4_kh": capi.Q4_KH}
_EPS = 1e-5

# Phi-3-mini, Phi-2's MLP and Whisper-tiny as their checkpoints have them
_PHI3 = dict(d=3072, heads=32, ffn=8192, vocab=32064, max_cache=4096)
_PHI2 = dict(d=2560, ffn=10240)
_WHISPER = dict(d=384, heads=6, mlp=1536, layers=4, mels=80)

# widths of served decoders, with the head counts, ranks and windows that go with them
_SERVED = {
    1024: dict(ff=2816, heads=8, l_heads=8, l_dim=64, l_rot=32, l_vdim=64, q_rank=384, kv_rank=256, window=512),
    2048: dict(ff=5632, heads=16, l_heads=16, l_dim=128, l_rot=64, l_vdim=128, q_rank=768, kv_rank=512, window=1024),
    4096: dict(ff=11008, heads=32, l_heads=32, l_dim=128, l_rot=64, l_vdim=128, q_rank=1536, kv_rank=512, window=2048),
}
_VOCAB = 32000


def listed():
    return [
        # one projection of a decode step: the smallest call that a host makes, all latency
        {"name": "gemv_q8_0h_3072x3072", "kind": "linear", "dt": "q8_0h", "m": 1, "n": 3072, "k": 3072},
        # a product that is all bandwidth, with 32-bit block scales under 16-bit activations
        {"name": "gemv_q8_0f_65536x16384", "kind": "linear", "dt": "q8_0f", "m": 1, "n": 65536, "k": 16384},
        # the up-projection of a 4-bit model over a prompt of ordinary length
        {"name": "gemm_q4_kh_512", "kind": "linear", "dt": "q4_kh", "m": 512, "n": 8192, "k": 3072},
        # 32-bit weights and activations: a model run without quantisation, 64 tokens at once
        {"name": "phi2_mlp_f32_64", "kind": "phi2", "tokens": 64},
        # transcription: thirty seconds of audio through the encoder in 32 bits, and a shorter clip through the 8-bit model
        {"name": "whisper_f32_3000", "kind": "whisper", "dt": "f32", "frames": 3000},
        {"name": "whisper_q8_0h_1001", "kind": "whisper", "dt": "q8_0h", "frames": 1001},
        # a prompt into an empty cache, with the causal mask that the model is given
        {"name": "phi3_prompt_q8_0h_1000", "kind": "phi3_prompt", "dt": "q8_0h", "layers": 8, "tokens": 1000},
        # one token of the whole model over a thousand cached ones
        {"name": "phi3_decode_q8_0h", "kind": "phi3_decode", "layers": 32, "prior": 1024},
        # served decoders: long prompts of which the last place's logits are wanted, and generation token by token
        {"name": "dadezen_prompt_2048", "kind": "served", "model": "Dadezen", "width": 2048, "layers": 8, "loops": 0, "prompt": 4096, "new": 0},
        {"name": "dadezen_generate_2048", "kind": "served", "model": "Dadezen", "width": 2048, "layers": 8, "loops": 0, "prompt": 600, "new": 24},
        {"name": "mefesun_prompt_4096", "kind": "served", "model": "Mefesun", "width": 4096, "layers": 4, "loops": 0, "prompt": 3001, "new": 0},
        {"name": "mefesun_generate_1024", "kind": "served", "model": "Mefesun", "width": 1024, "layers": 8, "loops": 0, "prompt": 333, "new": 32},
    ]


def _spread(rng, lo, hi):
    """A whole number between the two, even over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear"] * 6 + ["phi2", "whisper", "whisper", "phi3_prompt", "phi3_prompt", "phi3_decode"] + ["served"] * 4)
    if kind == "linear":
        dt = rng.choice(["q8_0h", "q8_0h", "q8_0f", "q4_kh", "q4_kh", "f16", "f32"])
        m = 1 if rng.random() < 0.5 else _spread(rng, 2, 2048)
        step = 256 if dt == "q4_kh" else 32
        k = step * _spread(rng, max(1, 256 // step), 16384 // step)
        n = _spread(rng, 64, max(64, min(65536, (1 << 29) // k, 10 ** 11 // (m * k))))
        return {"kind": kind, "dt": dt, "m": m, "n": n if rng.random() < 0.3 else -(-n // 64) * 64, "k": k}
    if kind == "phi2":
        return {"kind": kind, "tokens": _spread(rng, 2, 512)}
    if kind == "whisper":
        return {"kind": kind, "dt": rng.choice(["f32", "f16", "q8_0f", "q8_0h"]), "frames": rng.randint(200, 3000)}
    if kind == "phi3_prompt":
        return {"kind": kind, "dt": rng.choice(["f16", "q8_0h"]), "layers": rng.randint(2, 8), "tokens": _spread(rng, 9, 1500)}
    if kind == "phi3_decode":
        return {"kind": kind, "layers": rng.randint(2, 32), "prior": _spread(rng, 1, 4000)}
    model, generate = rng.choice(["Dadezen", "Mefesun"]), rng.random() < 0.5
    width = rng.choice([1024, 2048])
    return {"kind": kind, "model": model, "width": width, "layers": rng.randint(2, 8), "loops": rng.choice([0, 0, 2]) if model == "Dadezen" else 0,
            "prompt": _spread(rng, 2, 700) if generate else _spread(rng, 64, 4096), "new": rng.randint(4, 24) if generate else 0}


# ---------------------------------------------------------------------------------------- memory shared with torch
_device = None


def _dev():
    """The process's device handle; its weights stay as they are while products run."""
    global _device
    if _device is None:
        _device = Device(0)
        _device.set_constant_weights(True)
    return _device


_CODES = {capi.F32: ("<f4", None), capi.F16: ("<f2", None), capi.BF16: ("<i2", torch.bfloat16), capi.I32: ("<i4", None)}


class _Held:
    """Device memory of the framework as torch sees it; keeps its owner alive."""

    def __init__(self, owner, dt, shape, ptr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": _CODES[dt][0], "data": (ptr, False), "version": 2}


def _torch(owner, dt, shape, ptr):
    t = torch.as_tensor(_Held(owner, dt, shape, ptr), device="cuda")
    return t if _CODES[dt][1] is None else t.view(_CODES[dt][1])


def _out(t):
    """A resolved graph tensor."""
    return _torch(t, t.dt(), t.shape(), t.data_ptr())


def _lazy(t, dt=None, shape=None):
    """A graph tensor over torch's memory (which the caller keeps)."""
    dt = {torch.float32: capi.F32, torch.float16: capi.F16, torch.int32: capi.I32}[t.dtype] if dt is None else dt
    h, d = ctypes.c_void_p(), capi.describe(dt, t.shape if shape is None else shape, t.data_ptr())
    _dev().check(_dev()._lib.rcu_lazy_wrap(_dev().handle, ctypes.byref(d), ctypes.byref(h)))
    return Tensor(_dev(), h)


# ---------------------------------------------------------------------------------------- random weights
def _gen(seed):
    return torch.Generator("cuda").manual_seed(seed)


def _normal(g, *shape, dtype=torch.float32, std=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _matrix(g, dt, n, k):
    """W [n, k] in a storage type: a torch tensor, raw bytes in ratchet's layout for the quantised types."""
    if dt in ("f32", "f16"):
        return _normal(g, n, k, dtype=torch.float32 if dt == "f32" else torch.float16, std=0.02)
    code = DT[dt]
    at, raw = capi.dtype_segments(code, n * k), torch.zeros(capi.dtype_nbytes(code, n * k), dtype=torch.uint8, device="cuda")
    part = lambda i, dtype, count: raw[at[i]:at[i] + count * dtype.itemsize].view(dtype)
    if dt in ("q8_0f", "q8_0h"):
        rows = max(1, (1 << 27) // k)                          # a piece at a time: no large temporaries
        q = part(0, torch.int8, n * k).view(n, k)
        for a in range(0, n, rows):
            q[a:a + rows] = (torch.randn(min(rows, n - a), k, generator=g, device="cuda") * 50).round_().clamp_(-127, 127)
        scales = part(1, torch.float32 if dt == "q8_0f" else torch.float16, n * k // 32)
        scales.copy_((torch.rand(n * k // 32, generator=g, device="cuda") * 0.4 + 0.8) * 4e-4)
        return raw
    blocks = n * k // 256                                      # Q4_K: eight 6-bit scales and minima per block, packed into twelve bytes
    part(0, torch.uint8, n * k // 2).random_(0, 256, generator=g)
    s = torch.randint(24, 64, (blocks, 8), generator=g, device="cuda", dtype=torch.int32)
    m = (s + torch.randint(-3, 4, (blocks, 8), generator=g, device="cuda", dtype=torch.int32)).clamp_(0, 63)
    lo, hi = slice(0, 4), slice(4, 8)
    packed = torch.cat([s[:, lo] | (s[:, hi] >> 4) << 6, m[:, lo] | (m[:, hi] >> 4) << 6, (s[:, hi] & 15) | (m[:, hi] & 15) << 4], 1)
    part(1, torch.uint8, blocks * 12).copy_(packed.reshape(-1))
    d = (torch.rand(blocks, generator=g, device="cuda") * 0.4 + 0.8) * 1e-4
    part(2, torch.float16, blocks).copy_(d * 7.5)
    part(3, torch.float16, blocks).copy_(d)
    return raw


def _f64(w, dt, n, k, a=0, b=None):
    """Rows a to b of a stored matrix in 64 bits."""
    b = n if b is None else min(b, n)
    if dt in ("f32", "f16"):
        return w[a:b].double()
    code = DT[dt]
    at = capi.dtype_segments(code, n * k)
    part = lambda i, dtype, x, y: w[at[i] + x * dtype.itemsize:at[i] + y * dtype.itemsize].view(dtype)
    if dt in ("q8_0f", "q8_0h"):
        d = part(1, torch.float32 if dt == "q8_0f" else torch.float16, a * k // 32, b * k // 32).double()
        return (part(0, torch.int8, a * k, b * k).double().view(-1, 32) * d[:, None]).view(b - a, k)
    x, y = a * k // 256, b * k // 256
    c = part(1, torch.uint8, x * 12, y * 12).view(-1, 12).int()
    s = torch.cat([c[:, :4] & 63, (c[:, 8:] & 15) | (c[:, :4] >> 6) << 4], 1).double()
    m = torch.cat([c[:, 4:8] & 63, c[:, 8:] >> 4 | (c[:, 4:8] >> 6) << 4], 1).double()
    q = part(0, torch.uint8, x * 128, y * 128).view(-1, 4, 1, 32)
    q = torch.cat([q & 15, q >> 4], 2).double().view(-1, 8, 32)
    dmin, d = part(2, torch.float16, x, y).double(), part(3, torch.float16, x, y).double()
    return (q * (d[:, None] * s)[..., None] - (dmin[:, None] * m)[..., None]).view(b - a, k)


class _Weights:
    """Stored matrices [n, k] and float vectors by name, as graph tensors or in 64 bits."""

    def __init__(self, g, dt):
        self.g, self.dt, self.held = g, dt, {}

    def matrix(self, name, n, k):
        self.held[name] = (_matrix(self.g, self.dt, n, k), self.dt, n, k)

    def vector(self, name, t):
        self.held[name] = (t.contiguous(), None, None, None)

    def __contains__(self, name):
        return name in self.held

    def lazy(self, name):
        w, dt, n, k = self.held[name]
        return _lazy(w) if dt is None else _lazy(w, DT[dt], (n, k))

    def buffer(self, name):
        w, dt, n, k = self.held[name]
        return _dev().wrap(capi.F32, w.shape, w.data_ptr()) if dt is None else _dev().wrap(DT[dt], (n, k), w.data_ptr())

    def f64(self, name):
        w, dt, n, k = self.held[name]
        return w.double() if dt is None else _f64(w, dt, n, k)


def _norm(x, w, b=None, mean=True):
    d = x - x.mean(-1, keepdim=True) if mean else x
    y = d / torch.sqrt((d * d).mean(-1, keepdim=True) + _EPS) * w
    return y if b is None else y + b


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


# ---------------------------------------------------------------------------------------- one matrix product
def _linear_inputs(case, seed):
    g = _gen(seed)
    w = _matrix(g, case["dt"], case["n"], case["k"])
    return w, _normal(g, case["m"], case["k"], dtype=torch.float32 if case["dt"] == "f32" else torch.float16)


def _linear_prepare(case, seed):
    w, x = _linear_inputs(case, seed)
    y = torch.empty(case["m"], case["n"], dtype=x.dtype, device="cuda")
    act = DT["f32" if x.dtype == torch.float32 else "f16"]
    descs = [capi.describe(DT[case["dt"]], (case["n"], case["k"]), w.data_ptr()), capi.describe(act, x.shape, x.data_ptr()), capi.describe(act, y.shape, y.data_ptr())]
    return {"keep": (w, x, descs), "y": y, "call": _dev()._lib.rcu_matmul, "handle": _dev().handle, "refs": [ctypes.byref(d) for d in descs]}


def _linear_run(s):
    w, x, y = s["refs"]
    _dev().check(s["call"](s["handle"], w, x, None, 0, 1, 1, y))
    return s["y"]


def _linear_exact(case, seed):
    w, x = _linear_inputs(case, seed)
    rows, x = max(1, (1 << 28) // case["k"]), x.double()
    return torch.cat([x @ _f64(w, case["dt"], case["n"], case["k"], a, a + rows).T for a in range(0, case["n"], rows)], 1)


# ---------------------------------------------------------------------------------------- Phi-2's MLP block
def _phi2_weights(seed, tokens):
    g, d, ffn = _gen(seed), _PHI2["d"], _PHI2["ffn"]
    W = _Weights(g, "f32")
    W.vector("x", _normal(g, 1, tokens, d))
    W.vector("ln", 1 + _normal(g, d, std=0.1))
    W.vector("ln.b", _normal(g, d, std=0.1))
    W.matrix("fc1", ffn, d)
    W.matrix("fc2", d, ffn)
    W.vector("fc1.b", _normal(g, ffn, std=0.02))
    W.vector("fc2.b", _normal(g, d, std=0.02))
    return W


def _phi2_prepare(case, seed):
    W = _phi2_weights(seed, case["tokens"])
    t = W.lazy
    block = callers.Phi2MLPBlock(nn.LayerNorm(t("ln"), t("ln.b"), _EPS), nn.Linear(t("fc1"), t("fc1.b")), nn.Linear(t("fc2"), t("fc2.b")))
    return {"keep": W, "model": block, "x": t("x")}


def _graph_run(s):
    return _out(s["model"].schedule(s["x"]).resolve())


def _phi2_exact(case, seed):
    W = _phi2_weights(seed, case["tokens"]).f64
    x = W("x")
    return _gelu(_norm(x, W("ln"), W("ln.b")) @ W("fc1").T + W("fc1.b")) @ W("fc2").T + W("fc2.b") + x


# ---------------------------------------------------------------------------------------- Whisper's encoder
def _whisper_weights(case, seed):
    c, g = _WHISPER, _gen(seed)
    d, ctx = c["d"], (case["frames"] - 1) // 2 + 1
    W = _Weights(g, case["dt"])
    W.vector("mel", torch.rand(1, c["mels"], case["frames"], generator=g, device="cuda") * 2 - 1)
    for n, cin in (("conv1", c["mels"]), ("conv2", d)):
        W.vector(n, _normal(g, d, cin, 3, std=0.02))
        W.vector(n + ".b", _normal(g, d, std=0.02))
    at = torch.arange(ctx, device="cuda").double()[:, None] * torch.exp(-math.log(10000.0) / (d // 2 - 1) * torch.arange(d // 2, device="cuda").double())
    W.vector("pos", torch.cat([at.sin(), at.cos()], 1).float())
    for p in [f"{i}." for i in range(c["layers"])]:
        for n in ("ln1", "ln2"):
            W.vector(p + n, 1 + _normal(g, d, std=0.1))
            W.vector(p + n + ".b", _normal(g, d, std=0.1))
        for n, rows, cols in (("q", d, d), ("k", d, d), ("v", d, d), ("o", d, d), ("fc1", c["mlp"], d), ("fc2", d, c["mlp"])):
            W.matrix(p + n, rows, cols)
            if n != "k":
                W.vector(p + n + ".b", _normal(g, rows, std=0.02))
    W.vector("ln", 1 + _normal(g, d, std=0.1))
    W.vector("ln.b", _normal(g, d, std=0.1))
    W.vector("dk", torch.full((1,), (d // c["heads"]) ** -0.25, device="cuda", dtype=torch.float16 if case["dt"] in ("f16", "q8_0h") else torch.float32))
    return W


def _whisper_prepare(case, seed):
    W = _whisper_weights(case, seed)
    t = W.lazy
    norm = lambda n: nn.LayerNorm(t(n), t(n + ".b"), _EPS)
    linear = lambda n: nn.Linear(t(n), t(n + ".b") if n + ".b" in W else None)
    blocks = [callers.WhisperBlock(norm(p + "ln1"), callers.WhisperMHA(*[linear(p + n) for n in "qkvo"], _WHISPER["heads"], t("dk")), norm(p + "ln2"),
                                   callers.WhisperMLP(linear(p + "fc1"), linear(p + "fc2"))) for p in [f"{i}." for i in range(_WHISPER["layers"])]]
    act = capi.F16 if case["dt"] in ("f16", "q8_0h") else capi.F32
    return {"keep": W, "model": callers.WhisperEncoder(t("conv1"), t("conv1.b"), t("conv2"), t("conv2.b"), t("pos"), blocks, norm("ln"), act), "x": t("mel")}


def _whisper_exact(case, seed):
    W, H = _whisper_weights(case, seed).f64, _WHISPER["heads"]
    x = _gelu(torch.nn.functional.conv1d(W("mel"), W("conv1"), W("conv1.b"), 1, 1))
    x = _gelu(torch.nn.functional.conv1d(x, W("conv2"), W("conv2.b"), 2, 1))[0].T + W("pos")
    for p in [f"{i}." for i in range(_WHISPER["layers"])]:
        h = _norm(x, W(p + "ln1"), W(p + "ln1.b"))
        q, k, v = ((h @ W(p + n).T + (W(p + n + ".b") if n != "k" else 0)).view(len(x), H, -1).transpose(0, 1) for n in "qkv")
        o = torch.softmax((q * W("dk")) @ (k * W("dk")).transpose(1, 2), -1) @ v
        x = x + o.transpose(0, 1).reshape(len(x), -1) @ W(p + "o").T + W(p + "o.b")
        h = _gelu(_norm(x, W(p + "ln2"), W(p + "ln2.b")) @ W(p + "fc1").T + W(p + "fc1.b"))
        x = x + h @ W(p + "fc2").T + W(p + "fc2.b")
    return _norm(x, W("ln"), W("ln.b"))[None]


# ---------------------------------------------------------------------------------------- Phi-3
def _phi3_weights(g, dt, layers):
    c, W = _PHI3, _Weights(g, dt)
    d, ffn = c["d"], c["ffn"]
    for p in [f"{i}." for i in range(layers)]:
        for n in ("n1", "n2"):
            W.vector(p + n, 1 + _normal(g, d, std=0.1))
        for n, rows, cols in (("qkv", 3 * d, d), ("o", d, d), ("up", 2 * ffn, d), ("down", d, ffn)):
            W.matrix(p + n, rows, cols)
    W.matrix("embed", c["vocab"], d)
    W.matrix("head", c["vocab"], d)
    W.vector("norm", 1 + _normal(g, d, std=0.1))
    return W


def _phi3_prompt_inputs(case, seed):
    g = _gen(seed)
    return _phi3_weights(g, case["dt"], case["layers"]), torch.randint(_PHI3["vocab"], (1, case["tokens"]), generator=g, device="cuda", dtype=torch.int32)


def _phi3_prompt_prepare(case, seed):
    c = _PHI3
    W, ids = _phi3_prompt_inputs(case, seed)
    t, hd = W.lazy, c["d"] // c["heads"]
    cache = torch.zeros(case["layers"], 2, 1, c["heads"], c["max_cache"], hd, dtype=torch.float16, device="cuda")
    mask = torch.full((case["tokens"], case["tokens"]), -65504.0, dtype=torch.float16, device="cuda").triu_(1)
    scale = torch.full((1,), hd ** -0.5, device="cuda")
    rope = nn.RotaryEmbedding(hd, False, 10000.0, 1.0)
    layers = [callers.Phi3DecoderLayer(nn.RMSNorm(t(p + "n1"), _EPS), callers.Phi3SelfAttention(nn.Linear(t(p + "qkv")), nn.Linear(t(p + "o")), rope, c["heads"],
                                                                                             c["heads"], _lazy(scale)),
                                       nn.RMSNorm(t(p + "n2"), _EPS), callers.Phi3MLP(nn.Linear(t(p + "up")), nn.Linear(t(p + "down"))))
              for p in [f"{i}." for i in range(case["layers"])]]
    kv = nn.KVCache([nn.KVEntry(_lazy(cache[i, 0]), _lazy(cache[i, 1])) for i in range(case["layers"])])
    model = callers.Phi3(nn.Embedding(t("embed")), layers, nn.RMSNorm(t("norm"), _EPS), nn.Linear(t("head")), kv)
    return {"keep": (W, ids, mask, scale), "model": model, "ids": _lazy(ids), "mask": _lazy(mask), "kv": kv, "tokens": case["tokens"], "cache": cache}


def _phi3_prompt_run(s):
    s["kv"].reset()
    logits = s["model"].schedule(s["ids"], s["mask"]).resolve().to_numpy()
    s["kv"].update(s["tokens"])
    return {"logits": logits, "cache": s["cache"]}


def _rope_half(x, at):
    """x [heads, tokens, dim], pairs half a head apart."""
    half = x.shape[-1] // 2
    a = at.double()[:, None] * torch.exp(-math.log(10000.0) / half * torch.arange(half, device="cuda").double())
    return torch.cat([x[..., :half] * a.cos() - x[..., half:] * a.sin(), x[..., :half] * a.sin() + x[..., half:] * a.cos()], -1)


def _phi3_exact(W, layers, ids, prior, cache):
    """Logits of the last token; `cache` [layers, 2, heads, rows, dim] in 64 bits receives the new rows behind `prior`."""
    c, T = _PHI3, len(ids)
    at, x = torch.arange(prior, prior + T, device="cuda"), W("embed")[ids.long()]
    for i, p in enumerate([f"{i}." for i in range(layers)]):
        q, k, v = ((_norm(x, W(p + "n1"), mean=False) @ W(p + "qkv").T).view(T, 3, c["heads"], -1).permute(1, 2, 0, 3))
        cache[i, 0, :, prior:prior + T], cache[i, 1, :, prior:prior + T] = _rope_half(k, at), v
        q, o = _rope_half(q, at), torch.empty_like(q)
        for h in range(c["heads"]):
            z = q[h] @ cache[i, 0, h, :prior + T].T * q.shape[-1] ** -0.5
            o[h] = torch.softmax(z.masked_fill(torch.arange(prior + T, device="cuda") > at[:, None], -math.inf), -1) @ cache[i, 1, h, :prior + T]
        x = x + o.transpose(0, 1).reshape(T, -1) @ W(p + "o").T
        gate, up = (_norm(x, W(p + "n2"), mean=False) @ W(p + "up").T).chunk(2, -1)
        x = x + (torch.nn.functional.silu(gate) * up) @ W(p + "down").T
    return (_norm(x[-1:], W("norm"), mean=False) @ W("head").T)[None]


def _phi3_prompt_exact(case, seed):
    W, ids = _phi3_prompt_inputs(case, seed)
    c = _PHI3
    cache = torch.zeros(case["layers"], 2, c["heads"], c["max_cache"], c["d"] // c["heads"], dtype=torch.float64, device="cuda")
    return {"logits": _phi3_exact(W.f64, case["layers"], ids[0], 0, cache), "cache": cache[:, :, None]}


def _phi3_decode_inputs(case, seed):
    c, g = _PHI3, _gen(seed)
    W = _phi3_weights(g, "q8_0h", case["layers"])
    cache = torch.zeros(case["layers"], 2, c["heads"], c["max_cache"], c["d"] // c["heads"], dtype=torch.float16, device="cuda")
    cache[..., :case["prior"], :] = torch.randn(*cache.shape[:3], case["prior"], cache.shape[-1], generator=g, device="cuda", dtype=torch.float16)
    return W, cache, int(torch.randint(c["vocab"], (1,), generator=g, device="cuda"))


def _phi3_decode_prepare(case, seed):
    c, d = _PHI3, _PHI3["d"]
    W, cache, token = _phi3_decode_inputs(case, seed)
    b, hd = W.buffer, d // c["heads"]
    kv = lambda i, j: _dev().wrap(capi.F16, cache.shape[2:], cache[i, j].data_ptr())
    layers = [DecoderLayer(b(p + "n1"), b(p + "qkv"), b(p + "o"), b(p + "n2"), b(p + "up"), b(p + "down"), kv(i, 0), kv(i, 1))
              for i, p in enumerate([f"{i}." for i in range(case["layers"])])]
    cfg = DecoderConfig(case["layers"], d, c["heads"], c["heads"], hd, c["ffn"], c["vocab"], c["max_cache"], hd, 10000.0, _EPS, capi.Q8_0H)
    return {"keep": W, "decoder": Decoder(_dev(), cfg, layers, b("embed"), b("norm"), b("head")), "prior": case["prior"], "token": token, "cache": cache}


def _phi3_decode_run(s):
    s["decoder"].position = s["prior"]
    return {"logits": s["decoder"].step(s["token"]), "cache": s["cache"]}


def _phi3_decode_exact(case, seed):
    W, cache, token = _phi3_decode_inputs(case, seed)
    cache = cache.double()
    return {"logits": _phi3_exact(W.f64, case["layers"], torch.tensor([token], device="cuda"), case["prior"], cache), "cache": cache}


# ---------------------------------------------------------------------------------------- served decoders
def _served_config(case):
    c, d, n = _SERVED[case["width"]], case["width"], case["layers"]
    yarn = {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}
    mlp = {"kind": "dense", "ff": c["ff"]}
    if case["model"] == "Mefesun":
        layer = {"type": "attention", "mixer": {"heads": d // 128, "kv_heads": max(d // 512, 1), "dim": 128, "vdim": 128, "mask": {"size": c["window"]},
                                                "scale": 128 ** -0.5, "rot": {"base": 10000.0, "dims": 128, "scaling": yarn}}, "mlp": mlp}
        return {"architecture": "Mefesun", "width": d, "vocab": _VOCAB, "norm": {"eps": _EPS}, "logit_softcap": 50.0, "layers": [layer] * n}
    decay = [1.0 - 2.0 ** -(2 + 6 * i / c["heads"]) for i in range(c["heads"])]
    pair = [{"type": "lightning", "mixer": {"heads": c["heads"], "dim": 128, "vdim": 128, "decay": decay}, "mlp": mlp},
            {"type": "latent_attention", "mixer": {"heads": c["l_heads"], "dim": c["l_dim"], "rot_dim": c["l_rot"], "vdim": c["l_vdim"], "q_rank": c["q_rank"],
                                                   "kv_rank": c["kv_rank"], "mask": {"size": c["window"]}, "scale": (c["l_dim"] + c["l_rot"]) ** -0.5,
                                                   "rot": {"base": 10000.0, "dims": c["l_rot"], "scaling": yarn}}, "mlp": mlp}]
    cfg = {"architecture": "Dadezen", "width": d, "vocab": _VOCAB, "norm": {"eps": _EPS}, "residual_mult": 0.5, "layers": (pair * n)[:n]}
    if case["loops"]:
        cfg["loop"] = {"start": 0, "stop": 2, "times": case["loops"]}
    return cfg


def _served_shapes(cfg):
    d = cfg["width"]
    S = {"embed": (_VOCAB, d), "final.norm": (d,)}
    S.update({"final.norm.b": (d,)} if cfg["architecture"] == "Mefesun" else {"head": (_VOCAB, d)})
    if cfg.get("loop"):
        S.update({"loop.in": (d, 2 * d), "loop.step": (cfg["loop"]["times"], d)})
    for i, e in enumerate(cfg["layers"]):
        m, ff, p, x = e["mixer"], e["mlp"]["ff"], f"l{i}.", f"l{i}.mix."
        H, D, E = m["heads"], m["dim"], m["vdim"]
        S.update({x + "o": (d, H * E), p + "mlp.up": (ff, d), p + "mlp.down": (d, ff)})
        if e["type"] == "attention":
            for n, rows in (("q", H * D), ("k", m["kv_heads"] * D), ("v", m["kv_heads"] * E)):
                S.update({x + n: (rows, d), x + n + ".b": (rows,)})
            S.update({x + "o.b": (d,), x + "q.norm": (D,), x + "k.norm": (D,), x + "sink": (H,)})
            S.update({f"{p}{n}": (d,) for n in ("norm1", "norm1.b", "ls1", "norm2", "norm2.b", "ls2")})
            continue
        S.update({p + "norm1": (d,), p + "norm2": (d,), p + "mlp.gate": (ff, d)})
        if e["type"] == "lightning":
            S.update({x + "q": (H * D, d), x + "k": (H * D, d), x + "v": (H * E, d), x + "g": (H * E, d), x + "norm": (H * E,)})
        else:
            Q, C, R = m["q_rank"], m["kv_rank"], m["rot_dim"]
            S.update({x + "dq": (Q, d), x + "dq.norm": (Q,), x + "uq": (H * (D + R), Q), x + "dkv": (C + R, d), x + "dkv.norm": (C,), x + "uk": (H * D, C),
                      x + "uv": (H * E, C)})
    return S


class _ServedFile:
    """The weights of a served decoder as the loader reads a file: bf16 matrices, vectors in 32 bits."""

    def __init__(self, cfg, seed):
        g = _gen(seed)
        self.held = {}
        for name, s in _served_shapes(cfg).items():
            if name == "embed":
                self.held[name] = _normal(g, *s, dtype=torch.bfloat16)
            elif len(s) == 2:
                self.held[name] = _normal(g, *s, dtype=torch.bfloat16, std=s[1] ** -0.5)
            elif name.endswith((".b", ".sink")):
                self.held[name] = _normal(g, *s, std=0.1)
            else:
                self.held[name] = 1 + _normal(g, *s, std=0.1)
        if cfg["architecture"] == "Mefesun":                   # the embedding is the head too: logits of ordinary size
            self.held["embed"] *= cfg["width"] ** -0.5 * 4

    def __contains__(self, name):
        return name in self.held

    def shape(self, name):
        return tuple(self.held[name].shape)

    def raw(self, name):
        t = self.held[name].cpu()
        return ("BF16", t.view(torch.int16).numpy().view(np.uint16)) if t.dtype == torch.bfloat16 else ("F32", t.numpy())

    def f32(self, name):
        return self.held[name].float().cpu().numpy()

    def f64(self, name):
        return self.held[name].double()


def _served_tokens(case, seed):
    return [int(t) for t in np.random.Generator(np.random.PCG64(seed)).integers(0, _VOCAB, case["prompt"] + case["new"])]


def _served_prepare(case, seed):
    cfg, tokens = _served_config(case), _served_tokens(case, seed)
    model = REGISTRY[case["model"]](cfg, _ServedFile(cfg, seed), _dev())
    state = model.new_state(8192)
    return {"model": model, "state": state, "prompt": tokens[:case["prompt"]], "new": tokens[case["prompt"]:], "runs": [_out(t) for t in state.runs]}


def _served_run(s):
    """A sequence from its beginning: the prompt, then single tokens (given ones, in the place of those that are picked)."""
    model, state = s["model"], s["state"]
    state.reset()
    got = {"prompt": model.prefill(s["prompt"], state, [len(s["prompt"]) - 1])}
    for t in s["new"]:
        logits, picked = model.decode(state, t)
        picked.to_numpy()                                      # the id that a greedy caller waits for
    if s["new"]:
        got["last"] = logits.to_numpy()
    got["state"] = s["runs"]
    return got


def _rotate(x, rot):
    """x [tokens, heads, dim] at positions 0, 1, ..: interleaved pairs of the leading features, YaRN frequencies."""
    n, sc = rot["dims"], rot["scaling"]
    f = rot["base"] ** (-2.0 * torch.arange(n // 2, device="cuda").double() / n)
    turn = lambda t: n * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(rot["base"]))
    lo, hi = max(math.floor(turn(sc["fast"])), 0), min(math.ceil(turn(sc["slow"])), n - 1)
    r = ((torch.arange(n // 2, device="cuda").double() - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    a = (torch.arange(len(x), device="cuda").double()[:, None] * (f / sc["factor"] * r + f * (1 - r)))[:, None]
    mag = 0.1 * math.log(sc["factor"]) + 1
    e, o = x[..., 0:n:2], x[..., 1:n:2]
    out = x.clone()
    out[..., 0:n:2], out[..., 1:n:2] = (e * a.cos() - o * a.sin()) * mag, (o * a.cos() + e * a.sin()) * mag
    return out


def _attend(q, k, v, scale, sees, sink=None):
    """q [T, H, D], k and v of grouped heads; sees(i, j): the mask."""
    T, H, per = len(q), q.shape[1], q.shape[1] // k.shape[1]
    at, o = torch.arange(T, device="cuda"), torch.empty(T, H, v.shape[2], dtype=torch.float64, device="cuda")
    hidden = ~sees(at[:, None], at[None, :])
    for h in range(H):
        z = (q[:, h] @ k[:, h // per].T * scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink[h].expand(T, 1)], 1)
        o[:, h] = torch.softmax(z, -1)[:, :T] @ v[:, h // per]
    return o.reshape(T, -1)


def _lightning_exact(q, k, v, decay):
    T, at = len(q), torch.arange(len(q), device="cuda").double()
    gap, o, S = at[:, None] - at[None, :], torch.empty_like(v), []
    for h, d in enumerate(decay):
        o[:, h] = ((q[:, h] @ k[:, h].T) * torch.where(gap >= 0, d ** gap.clamp(min=0), 0.0)) @ v[:, h]
        S.append(k[:, h].T @ (v[:, h] * (d ** (T - 1 - at))[:, None]))
    return o.reshape(T, -1), torch.stack(S)


def _served_exact(case, seed):
    cfg, tokens = _served_config(case), torch.tensor(_served_tokens(case, seed), device="cuda")
    f, T, T0 = _ServedFile(cfg, seed), len(tokens), case["prompt"]
    W, state = f.f64, []
    x = x0 = W("embed")[tokens]

    def ring(rows, size, kept):
        """Position p in row p mod size; of the prompt only its last `kept` rows are written."""
        r = torch.zeros(size, rows.shape[1], dtype=torch.float64, device="cuda")
        for p in list(range(T0 - kept, T0)) + list(range(T0, T)):
            r[p % size] = rows[p]
        return r

    n, loop = len(cfg["layers"]), cfg.get("loop")
    runs = [(i, None) for i in range(n)] if not loop else [(i, t) for t in range(loop["times"]) for i in range(loop["stop"])] + [(i, None) for i in range(loop["stop"], n)]
    for i, t in runs:
        e, p, xm = cfg["layers"][i], f"l{i}.", f"l{i}.mix."
        m = e["mixer"]
        H, D, E = m["heads"], m["dim"], m["vdim"]
        if loop and t is not None and i == 0:
            x = torch.cat([x, x0], 1) @ W("loop.in").T + W("loop.step")[t]
        size = m["mask"]["size"] if "mask" in m else 0
        if e["type"] == "attention":
            G = m["kv_heads"]
            q, k, v = (x @ W(xm + c).T + W(xm + c + ".b") for c in "qkv")
            q = _rotate(_norm(q.view(T, H, D), W(xm + "q.norm"), mean=False), m["rot"])
            k = _rotate(_norm(k.view(T, G, D), W(xm + "k.norm"), mean=False), m["rot"])
            o = _attend(q, k, v.view(T, G, E), m["scale"], lambda a, b: (b <= a) & (a // size == b // size), W(xm + "sink"))
            state.append(ring(torch.cat([k.reshape(T, -1), v], 1), size, min(T0, T0 % size)))
            x = x + W(p + "ls1") * _norm(o @ W(xm + "o").T + W(xm + "o.b"), W(p + "norm1"), W(p + "norm1.b"))
            x = x + W(p + "ls2") * _norm((x @ W(p + "mlp.up").T).clamp(min=0) ** 2 @ W(p + "mlp.down").T, W(p + "norm2"), W(p + "norm2.b"))
            continue
        h = _norm(x, W(p + "norm1"))
        if e["type"] == "lightning":
            q, k, v = (torch.nn.functional.silu(h @ W(xm + c).T).view(T, H, -1) for c in "qkv")
            o, S = _lightning_exact(q, k, v, m["decay"])
            state.append(S)
            y = (_norm(o, W(xm + "norm"), mean=False) * torch.sigmoid(h @ W(xm + "g").T)) @ W(xm + "o").T
        else:
            R, C = m["rot_dim"], m["kv_rank"]
            q = (_norm(h @ W(xm + "dq").T, W(xm + "dq.norm"), mean=False) @ W(xm + "uq").T).view(T, H, D + R)
            q = torch.cat([q[..., :D], _rotate(q[..., D:], m["rot"])], -1)
            low = h @ W(xm + "dkv").T
            c, kr = _norm(low[:, :C], W(xm + "dkv.norm"), mean=False), _rotate(low[:, None, C:], m["rot"])
            k = torch.cat([(c @ W(xm + "uk").T).view(T, H, D), kr.expand(T, H, R)], -1)
            o = _attend(q, k, (c @ W(xm + "uv").T).view(T, H, E), m["scale"], lambda a, b: (b <= a) & (b > a - size))
            state.append(ring(torch.cat([c, kr[:, 0]], 1), size, min(T0, size)))
            y = o @ W(xm + "o").T
        h = _norm(x, W(p + "norm2"))
        y = y + (_gelu(h @ W(p + "mlp.gate").T) * (h @ W(p + "mlp.up").T)) @ W(p + "mlp.down").T
        x = x + cfg["residual_mult"] * y
    places = [T0 - 1] + ([T - 1] if case["new"] else [])
    if cfg["architecture"] == "Mefesun":
        z = _norm(x[places], W("final.norm"), W("final.norm.b")) @ W("embed").T
        z = cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])
    else:
        z = _norm(x[places], W("final.norm")) @ W("head").T
    got = {"prompt": z[:1], "state": state}
    return dict(got, last=z[1:]) if case["new"] else got


def _served_work(case):
    """Every weight once for the prompt and once for each further token, states written; products of the prompt and of the tokens."""
    cfg, T0, new = _served_config(case), case["prompt"], case["new"]
    loop, mats, attn, kept = cfg.get("loop"), 0, 0.0, 0
    shapes = _served_shapes(cfg)
    for i, e in enumerate(cfg["layers"]):
        times = loop["times"] if loop and i < loop["stop"] else 1
        m = e["mixer"]
        mats += times * sum(s[0] * s[1] for n, s in shapes.items() if n.startswith(f"l{i}.") and len(s) == 2)
        if e["type"] == "lightning":
            attn += times * (T0 + new) * 4.0 * m["heads"] * m["dim"] * m["vdim"]
            kept += times * 4 * m["heads"] * m["dim"] * m["vdim"]
            continue
        size = m["mask"]["size"]
        sees = (lambda p: p % size + 1) if e["type"] == "attention" else (lambda p: min(p + 1, size))
        attn += times * sum(sees(p) for p in range(T0 + new)) * 2.0 * m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"])
        kept += times * 2 * min(size, T0 + new) * (m["kv_heads"] * (m["dim"] + m["vdim"]) if e["type"] == "attention" else m["kv_rank"] + m["rot_dim"])
    if loop:
        mats += loop["times"] * 2 * cfg["width"] ** 2
    head = _VOCAB * cfg["width"]
    return {"bytes": 2.0 * (mats + head) * (1 + new) + kept * (1 + new), "flops": 2.0 * mats * (T0 + new) + 2.0 * head * (1 + new) + attn}


# ---------------------------------------------------------------------------------------- the five functions
_PARTS = {"linear": (_linear_prepare, _linear_run, _linear_exact), "phi2": (_phi2_prepare, _graph_run, _phi2_exact),
          "whisper": (_whisper_prepare, _graph_run, _whisper_exact), "phi3_prompt": (_phi3_prompt_prepare, _phi3_prompt_run, _phi3_prompt_exact),
          "phi3_decode": (_phi3_decode_prepare, _phi3_decode_run, _phi3_decode_exact), "served": (_served_prepare, _served_run, _served_exact)}


def prepare(case, seed):
    s = _PARTS[case["kind"]][0](case, seed)
    s["run"] = _PARTS[case["kind"]][1]
    return s


def run(state):
    return state["run"](state)


def exact(case, seed):
    return _PARTS[case["kind"]][2](case, seed)


_BYTES = {"f32": 4.0, "f16": 2.0, "q8_0f": 1.125, "q8_0h": 1.0625, "q4_kh": 0.5625}


def work(case):
    kind = case["kind"]
    if kind == "linear":
        act, (m, n, k) = 4 if case["dt"] == "f32" else 2, (case[x] for x in "mnk")
        return {"bytes": _BYTES[case["dt"]] * n * k + act * m * (n + k), "flops": 2.0 * m * n * k}
    if kind == "phi2":
        d, ffn, t = _PHI2["d"], _PHI2["ffn"], case["tokens"]
        return {"bytes": 8.0 * d * ffn + 8.0 * t * d, "flops": 4.0 * t * d * ffn}
    if kind == "whisper":
        c, frames = _WHISPER, case["frames"]
        d, ctx = c["d"], (frames - 1) // 2 + 1
        mats = c["layers"] * (4 * d * d + 2 * d * c["mlp"])
        return {"bytes": _BYTES[case["dt"]] * mats + 12.0 * d * (d + c["mels"]) + 4.0 * c["mels"] * frames + 8.0 * ctx * d,
                "flops": 6.0 * d * (frames * c["mels"] + ctx * d) + 2.0 * ctx * mats + c["layers"] * 4.0 * ctx * ctx * d}
    if kind == "served":
        return _served_work(case)
    c, d, layers = _PHI3, _PHI3["d"], case["layers"]
    mats, head = layers * (4 * d * d + 3 * d * c["ffn"]), c["vocab"] * d
    if kind == "phi3_prompt":
        t = case["tokens"]
        return {"bytes": _BYTES[case["dt"]] * (mats + head) + layers * 4.0 * t * d, "flops": 2.0 * t * mats + 2.0 * head + layers * 2.0 * t * (t + 1) * d}
    return {"bytes": _BYTES["q8_0h"] * (mats + head) + layers * 4.0 * (case["prior"] + 1) * d, "flops": 2.0 * (mats + head) + layers * 4.0 * case["prior"] * d}


def tolerance(case):
    """About four times what the present code is off `exact` by, as another order of sums or other roundings between ops would be."""
    if case["kind"] == "phi2" or case.get("dt") == "f32" or (case["kind"], case.get("dt")) == ("whisper", "q8_0f"):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 2.5e-3, "max": 0.1} if case["kind"] in ("linear", "whisper") else {"rel": 1.5e-2, "max": 0.5}
