"""PackedWeight / PackedMLP: thin owners of the C-ABI handles (tllm_weight, tllm_mlp)."""
from __future__ import annotations

import ctypes as C

import numpy as np

from . import _lib
from ._lib import PackOpts, WeightInfo, check, lib, np_ptr


def _opts(tile_rows=0, num_ctas=0, max_rows=0, k_splits=0, no_bit_tiles=0, no_nibbles=0):
    return PackOpts(int(tile_rows), int(num_ctas), 0, int(max_rows), int(k_splits), int(no_bit_tiles), int(no_nibbles))


def _dense_i8(w):
    if hasattr(w, "detach"):
        w = w.detach().cpu().numpy()
    w = np.ascontiguousarray(w)
    if w.dtype != np.int8:
        if np.any((w < -1) | (w > 1)):
            raise ValueError("weight is not ternary")
        w = w.astype(np.int8)
    return w


_HOST_CODES = {np.dtype(np.float32): _lib.F32, np.dtype(np.float16): _lib.F16, np.dtype(np.int8): _lib.I8}


class PackedWeight:
    """A ternary matrix W [inners, columns] packed into the bank-stream format on the current CUDA device."""

    def __init__(self, handle, device_index):
        self._h = handle
        self._call = None                    # (entry point, handle as an integer, device, inners, columns): made on first use
        self.device_index = device_index

    # ---- constructors -------------------------------------------------------------------------------
    @classmethod
    def from_dense(cls, w, scale=1.0, device=None, **opts):
        w = _dense_i8(w)
        K, N = w.shape
        return cls._create(lambda o, h: lib().tllm_weight_create_dense(np_ptr(w), K, N, float(scale), C.byref(o), C.byref(h)),
                           device, opts)

    @classmethod
    def from_ssr(cls, image, inners, columns, scale=1.0, device=None, **opts):
        """From the library's sparse-segment image (`ternaryllm_b200.ssr.encode`): validated and decoded on the host."""
        img = np.ascontiguousarray(np.asarray(image), dtype=np.uint8)
        return cls._create(lambda o, h: lib().tllm_weight_create_ssr(np_ptr(img), img.size, int(inners), int(columns), float(scale),
                                                                     C.byref(o), C.byref(h)),
                           device, opts)

    @classmethod
    def from_mcsc(cls, row_idx, col_off, columns, inners, tile_k, scale=1.0, device=None, **opts):
        ri = np.ascontiguousarray(np.asarray(row_idx), dtype=np.int32)
        co = np.ascontiguousarray(np.asarray(col_off), dtype=np.int32)
        return cls._create(lambda o, h: lib().tllm_weight_create_mcsc(np_ptr(ri), np_ptr(co), int(columns), int(inners),
                                                                      int(tile_k), float(scale), C.byref(o), C.byref(h)),
                           device, opts)

    @classmethod
    def from_cpu_format(cls, kind, group, chunk, metadata, row_index, columns, inners, aux=0, scale=1.0, device=None, **opts):
        meta = np.ascontiguousarray(np.asarray(metadata), dtype=np.int32)
        ri = np.ascontiguousarray(np.asarray(row_index))
        if ri.dtype not in (np.int16, np.int32):
            raise ValueError("row_index must be int16 or int32")
        return cls._create(lambda o, h: lib().tllm_weight_create_cpu_format(int(kind), int(group), int(chunk), np_ptr(meta), np_ptr(ri),
                                                                            int(ri.dtype == np.int32), int(aux), int(columns),
                                                                            int(inners), float(scale), C.byref(o), C.byref(h)),
                           device, opts)

    @classmethod
    def _create(cls, fn, device, opts):
        import torch

        dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
        if dev.type != "cuda":
            raise RuntimeError("PackedWeight lives on a CUDA device; there is no CPU implementation")
        h = C.c_void_p()
        o = _opts(**opts)
        with torch.cuda.device(dev):
            check(fn(o, h), "PackedWeight")
        return cls(h, dev.index if dev.index is not None else torch.cuda.current_device())

    @classmethod
    def load(cls, path, device=None):
        """A handle from a file written by `save` (no repacking)."""
        import torch

        dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
        h = C.c_void_p()
        with torch.cuda.device(dev):
            check(lib().tllm_weight_load(str(path).encode(), C.byref(h)), "PackedWeight.load")
        return cls(h, dev.index if dev.index is not None else torch.cuda.current_device())

    def save(self, path):
        check(lib().tllm_weight_save(self._h, str(path).encode()), "PackedWeight.save")

    # ---- use ---------------------------------------------------------------------------------------
    @property
    def info(self):
        i = WeightInfo()
        check(lib().tllm_weight_get_info(self._h, C.byref(i)))
        return i.as_dict()

    def set_scale(self, s):
        check(lib().tllm_weight_set_scale(self._h, float(s)))

    def check(self):
        check(lib().tllm_weight_check(self._h), "PackedWeight")

    def matmul(self, x, out=None, col_major=False):
        """y = x @ W * s for a 2-D CUDA tensor x [rows, inners] (or [inners, rows] with col_major)."""
        c = self._call or self._bind()
        return c[0](c[1], x, out, col_major, c[2], c[3], c[4])

    def _bind(self):
        info = self.info
        self._call = (_lib.binding().matmul, self._h.value, self.device_index, info["inners"], info["columns"])
        return self._call

    def matmul_host(self, x, col_major=False, y_col_major=False):
        """Same on numpy host arrays (copies in, runs, copies out, synchronises): the CPU entry points' form."""
        x = np.ascontiguousarray(x)
        code = _HOST_CODES[x.dtype]
        c = self._call or self._bind()
        rows = x.shape[1] if col_major else x.shape[0]
        if x.ndim != 2 or x.shape[0 if col_major else 1] != c[3]:
            raise RuntimeError(f"activation has {x.shape} but the weight has {c[3]} inners")
        y = np.empty((c[4], rows) if y_col_major else (rows, c[4]), np.int32 if code == _lib.I8 else x.dtype)
        _lib.binding().matmul_host(c[1], x, code, bool(col_major), rows, y, _lib.I32 if code == _lib.I8 else code, bool(y_col_major), c[2])
        return y

    def close(self):
        if self._h:
            lib().tllm_weight_destroy(self._h)
            self._h = self._call = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def ternarize(w, sparsity=None, threshold_factor=0.7):
    """Float weights [inners, columns] -> (int8 ternary weights, per-tensor scale); see tllm_ternarize."""
    if hasattr(w, "detach"):
        w = w.detach().float().cpu().numpy()
    w = np.ascontiguousarray(w, dtype=np.float32)
    if w.ndim != 2:
        raise ValueError("ternarize expects a 2-D weight")
    out = np.empty(w.shape, np.int8)
    scale = C.c_float()
    check(lib().tllm_ternarize(np_ptr(w), w.shape[0], w.shape[1], float(threshold_factor), float(sparsity or 0.0), np_ptr(out), C.byref(scale)),
          "tllm_ternarize")
    return out, float(scale.value)


class PackedMLP:
    """gate / up / down of one ternary MLP block, fused (see tllm_mlp_* in include/tllm.h)."""

    def __init__(self, w_gate, w_up, w_down, s_gate=1.0, s_up=1.0, s_down=1.0, device=None, **opts):
        import torch

        g, u, d = _dense_i8(w_gate), _dense_i8(w_up), _dense_i8(w_down)
        hidden, inter = g.shape
        if u.shape != (hidden, inter) or d.shape != (inter, hidden):
            raise ValueError("gate/up must be [hidden, intermediate] and down [intermediate, hidden]")
        dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
        self.device_index = dev.index if dev.index is not None else torch.cuda.current_device()
        self.hidden, self.inter = hidden, inter
        h = C.c_void_p()
        o = _opts(**opts)
        with torch.cuda.device(dev):
            check(lib().tllm_mlp_create(np_ptr(g), np_ptr(u), np_ptr(d), hidden, inter, float(s_gate), float(s_up), float(s_down),
                                        C.byref(o), C.byref(h)), "PackedMLP")
        self._h = h
        self._handle, self._forward = h.value, _lib.binding().mlp_forward

    @property
    def info(self):
        a, b = WeightInfo(), WeightInfo()
        check(lib().tllm_mlp_get_info(self._h, C.byref(a), C.byref(b)))
        return a.as_dict(), b.as_dict()

    def forward(self, x, out=None, h=None):
        return self._forward(self._handle, x, out, h, self.hidden)

    def close(self):
        if self._h:
            lib().tllm_mlp_destroy(self._h)
            self._h = None
            self._handle = 0                 # the library refuses a null handle

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass
