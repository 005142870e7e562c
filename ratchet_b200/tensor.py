"""Lazy ``Tensor`` over the CUDA device: same method names, argument meaning and error behaviour as
ratchet-core's ``Tensor`` (crates/ratchet-core/src/tensor.rs:294-510).

A ``Tensor`` owns one reference to a node of the C++ lazy graph (``rcu_lazy``).  As in the
reference, builder methods only record operations; ``resolve()`` runs them.  The reference's
methods take ``self`` by value: calling ``x.add(y)`` consumes ``x`` unless the caller wrote
``x.clone()``.  Python has no moves, so builders here borrow their operands; to let an op run in
place (the reference allows it only when the op is the operand's sole owner) drop your handle with
``Tensor.consume()`` or simply let it go out of scope before ``resolve()``.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional, Sequence

import numpy as np

from . import capi
from .capi import RatchetCudaError
from .device import Device

Node = capi.graph_module().Node


def _u64(seq):
    return (C.c_uint64 * len(seq))(*[int(s) for s in seq])


class Tensor(Node):
    """The builder methods that are not here are ``Node``'s (csrc/pygraph.c): same names, arguments and errors."""
    __slots__ = ()

    # ------------------------------------------------------------------ constructors
    @staticmethod
    def from_data(data, shape=None, device: Device = None, dt: Optional[int] = None) -> "Tensor":
        """Tensor::from_data (tensor.rs:578-616)."""
        a = np.ascontiguousarray(data)
        if shape is not None:
            a = a.reshape(shape)
        if dt is None:
            dt = capi.dt_of_numpy(a)
        shp = a.shape if a.ndim else (1,)
        h = C.c_void_p()
        device.check(device._lib.rcu_lazy_from_host(device.handle, dt, len(shp), _u64(shp), a.ctypes.data_as(C.c_void_p),
                                                    a.nbytes, C.byref(h)))
        return Tensor(device, h)

    @staticmethod
    def from_quantized(raw, dt: int, shape, device: Device) -> "Tensor":
        """Tensor::from_quantized (tensor.rs:618-628): raw bytes of a ratchet segment buffer."""
        raw = np.ascontiguousarray(raw).view(np.uint8).reshape(-1)
        n = int(np.prod(shape))
        if raw.nbytes < capi.dtype_nbytes(dt, n):
            raise RatchetCudaError(capi.ERR_INVALID_ARG, "quantised buffer is smaller than its layout")
        h = C.c_void_p()
        device.check(device._lib.rcu_lazy_from_host(device.handle, dt, len(shape), _u64(shape), raw.ctypes.data_as(C.c_void_p),
                                                    raw.nbytes, C.byref(h)))
        return Tensor(device, h)

    @staticmethod
    def zeros(shape, dt: int, device: Device) -> "Tensor":
        h = C.c_void_p()
        device.check(device._lib.rcu_lazy_zeros(device.handle, dt, len(shape), _u64(shape), C.byref(h)))
        return Tensor(device, h)

    @staticmethod
    def randn(shape, device: Device, dt: int = capi.F32, seed: int = 0) -> "Tensor":
        g = np.random.Generator(np.random.PCG64(seed))
        return Tensor.from_data(g.standard_normal(shape).astype(capi.np_dtype(dt)), device=device)

    def _info(self):
        t = capi.rcu_tensor()
        resolved = self.dev._lib.rcu_lazy_info(self._h, C.byref(t))
        return t, bool(resolved)

    # ------------------------------------------------------------------ builders
    def _new(self, fn, *args) -> "Tensor":
        h = C.c_void_p()
        self.dev.check(fn(*args, C.byref(h)))
        return Tensor(self.dev, h)

    def _slice(self, ranges: Sequence) -> "Tensor":
        """``slice``: one (start, stop) pair or Python ``slice`` per dimension (tensor.rs:421-448)."""
        shp = self.shape()
        start, stop = [], []
        for i, r in enumerate(ranges):
            if isinstance(r, slice):
                a, b = (0 if r.start is None else r.start), (shp[i] if r.stop is None else r.stop)
            else:
                a, b = r
            start.append(a)
            stop.append(b)
        if len(start) != len(shp):
            raise RatchetCudaError(capi.ERR_INVALID_ARG, "slice: one range per dimension is required")
        return self._new(self.dev._lib.rcu_lazy_slice, self._h, _u64(start), _u64(stop))

    def _permute_rank(self):
        raise RatchetCudaError(capi.ERR_INVALID_ARG, "permute: one entry per dimension is required")

    @staticmethod
    def cat(tensors: Sequence["Tensor"], dim: int) -> "Tensor":
        dev = tensors[0].dev
        arr = (C.c_void_p * len(tensors))(*[t._h for t in tensors])
        h = C.c_void_p()
        dev.check(dev._lib.rcu_lazy_concat(arr, len(tensors), dim, C.byref(h)))
        return Tensor(dev, h)

    def index_write(self, src: "Tensor", write_start: Sequence[int]) -> "Tensor":
        return self._new(self.dev._lib.rcu_lazy_index_write, self._h, src._h, _u64(write_start))

    # ------------------------------------------------------------------ ops of models with a 32-bit residual stream
    def linear(self, x: "Tensor", bias: Optional["Tensor"] = None, resid: Optional["Tensor"] = None, alpha: float = 1.0,
               x_col: int = 0, act: Optional[str] = None, act_cols: Optional[int] = None, act_param: float = 0.0, dt: Optional[int] = None) -> "Tensor":
        """resid + alpha * f(x[..., x_col:] . self^T + bias), self the [N, K] weight, f `act` (silu, relu_squared, softcap) on the first
        `act_cols` columns (None: all); dt: the activations' dtype or F32."""
        return self._linear(x, x_col, bias, capi.LINEAR_ACTS[act], self.shape()[0] if act_cols is None else act_cols, act_param, resid, alpha,
                            x.dt() if dt is None else dt)

    def norm_rows(self, kind: int, scale: "Tensor", eps: float, dt: int, col: int = 0, gate: Optional["Tensor"] = None, gate_col: int = 0,
                  shift: Optional["Tensor"] = None):
        """LayerNorm / RMSNorm of columns [col, col + len(scale)), plus `shift`, optionally times sigmoid(gate[:, gate_col:])."""
        return self._norm_rows(kind, col, scale, shift, gate, gate_col, eps, dt)

    # Node.stream_rows(copy_dt): rows of a residual stream, f32 values followed by their bf16 roundings when `copy_dt` is BF16
    # Node.post_norm(y, scale, shift, eps): these stream rows + LayerNorm(y) * scale + shift
    # Node.bitcast(dt): the same bytes as elements of `dt` (a view)

    def glu(self, act: str) -> "Tensor":
        """act(gate) * up of rows that hold gate, then up."""
        return self._glu(capi.UNARY_OPS[act])

    def rotary(self, freqs: "Tensor", magnitude: float, position: int, first: int = 0) -> "Tensor":
        """Interleaved-pair rotation of features [first, first + 2 pairs) of [tokens, heads, dim]."""
        return self._rotary(first, freqs, magnitude, position)

    # Node.lightning(decay_pow, state): linear attention over q, k, v columns of these rows; `state` is updated in place

    def latent_append(self, scale: "Tensor", eps: float, freqs: "Tensor", magnitude: float, position: int, ring: "Tensor", rows: int, col: int = 0):
        """Latents and rotated key parts of a block into `ring`; the result is the `rows` rows the block sees."""
        return self._latent_append(col, scale, eps, freqs, magnitude, position, ring, rows)

    # Node.window_attention(kv, shared, shared_col, vdim, window, scale)
    # Node.rotary_angles(magnitude, position, tokens): [tokens, 2 pairs], cos and sin, times `magnitude`, of this frequency table's angles
    # from `position` on

    def norm_rotary(self, heads: int, scale: "Tensor", eps: float, angles: "Tensor", col: int = 0) -> "Tensor":
        """RMSNorm of each head of columns [col, col + heads * len(scale)), then the rotation by `angles`: [tokens, heads, dim]."""
        return self._norm_rotary(col, heads, scale, eps, angles)

    def kv_append(self, kv_heads: int, scale: "Tensor", eps: float, angles: "Tensor", position: int, keep: int, ring: "Tensor", rows: int, col: int = 0):
        """Keys (normed, rotated) and values of a block, its last `keep` rows into `ring`; the result is the `rows` rows the block sees."""
        return self._kv_append(col, kv_heads, scale, eps, angles, position, keep, ring, rows)

    def grouped_attention(self, kv: "Tensor", kv_heads: int, vdim: int, scale: float, sink: Optional["Tensor"] = None, window: int = 0, chunk: int = 0,
                          position: int = 0) -> "Tensor":
        """Softmax attention of these queries [tokens, heads, dim] over kv rows, the first of which is `position`: a sliding window, runs
        of `chunk` positions, or everything before."""
        return self._grouped_attention(kv, sink, kv_heads, vdim, window, chunk, position, scale)

    # ------------------------------------------------------------------ execution
    def resolve(self) -> "Tensor":
        """Tensor::resolve (tensor.rs:861-863). Asynchronous; ``to_numpy`` / ``Device.sync`` wait."""
        self.dev.check(self.dev._lib.rcu_lazy_resolve(self._h))
        return self

    def to_numpy(self) -> np.ndarray:
        """``.to(&Device::CPU)`` + ``to_vec`` (tensor.rs:949-975)."""
        t, _ = self._info()
        shape = tuple(t.shape[i] for i in range(t.rank))
        if t.dt in (capi.Q8_0F, capi.Q8_0H, capi.Q4_KF, capi.Q4_KH):
            out = np.empty(capi.dtype_nbytes(t.dt, int(np.prod(shape))), np.uint8)
        else:
            out = np.empty(shape, capi.np_dtype(t.dt))
        self.dev.check(self.dev._lib.rcu_lazy_to_host(self._h, out.ctypes.data_as(C.c_void_p), out.nbytes))
        return out


def last_resolve_stats(dev: Device) -> dict:
    s = capi.rcu_resolve_stats()
    dev._lib.rcu_last_resolve_stats(dev.handle, C.byref(s))
    return {f: getattr(s, f) for f, _ in capi.rcu_resolve_stats._fields_}
