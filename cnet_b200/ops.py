"""Direct calls of the C-ABI operators (include/cnet_b200.h) on torch CUDA tensors.

torch only owns the memory and the stream; every operator below is one call into
libcnet_b200.so, of Linear, FourierTrans, SoftMax and CrossEntropy by way of ops_native.so (host/ops_native.cpp), which
makes the results too.  Complex tensors are (re, im) pairs of contiguous float32 tensors.
"""
import ctypes as C
import importlib.machinery
import importlib.util
import os

from . import build as _build
from . import lib as _lib


def _p(t):
    return None if t is None else t.data_ptr()


_native = None


def _load_native():
    """The module ops_native.so beside the library (once)."""
    global _native
    if _native is None:
        path = os.path.join(_lib.HERE, "ops_native.so")
        if not os.path.exists(path):
            raise _lib.CnetError("ops_native.so is not built (run `python -m cnet_b200.build`)")
        import torch  # noqa: F401                       # the module finds torch's libraries loaded,
        _lib.load()                                      # and this one
        loader = importlib.machinery.ExtensionFileLoader("ops_native", path)
        try:
            mod = importlib.util.module_from_spec(importlib.util.spec_from_file_location("ops_native", path, loader=loader))
            loader.exec_module(mod)
            made_for = mod.built_for
        except ImportError as e:                         # symbols that this torch or interpreter does not have
            made_for = str(e)
        if made_for != _build.ops_key():                 # layouts of tensors and Python objects are compiled into it
            raise _lib.CnetError("ops_native.so is built for another torch or Python (%s; this is %s): run `python -m cnet_b200.build`"
                                 % (made_for, _build.ops_key()))
        mod.set_error_class(_lib.CnetError)
        _native = mod
    return _native


class Context:
    """cnb_create: a device arena for scratch, twiddles and GEMM staging."""

    def __init__(self, device=0, arena_bytes=256 << 20):
        import torch
        if not torch.cuda.is_available():
            raise _lib.CnetError("no CUDA device: the path has no CPU fallback")
        self.lib = _lib.load()
        self.torch = torch
        self.native = _load_native()
        self.h = C.c_void_p()
        _lib.check(self.lib.cnb_create(device, arena_bytes, C.byref(self.h)), "cnb_create")
        # The raw handle of the current stream costs 0.15 us where torch exposes it and 3.2 us as a Stream object: a
        # quarter of an operator's time on the host.
        raw, dev = getattr(torch._C, "_cuda_getCurrentRawStream", None), getattr(torch._C, "_cuda_getDevice", None)
        if raw and dev:
            self._stream = lambda: raw(dev())

    def close(self):
        if self.h:
            self.lib.cnb_destroy(self.h)
            self.h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    def _stream(self):
        return self.torch.cuda.current_stream().cuda_stream

    def _like(self, x):
        """A fresh pair of planes of the shape of x's, contiguous float32 as the kernels write them, whatever the strides
        and type of x (cheaper than naming the shape)."""
        like, t = self.torch.empty_like, self.torch
        return (like(x[0], dtype=t.float32, memory_format=t.contiguous_format),
                like(x[0], dtype=t.float32, memory_format=t.contiguous_format))

    def _new(self, *shape):
        return (self.torch.empty(*shape, dtype=self.torch.float32, device="cuda"),
                self.torch.empty(*shape, dtype=self.torch.float32, device="cuda"))

    # ------------------------------------------------------------------ Linear
    def linear_fwd(self, x, w, res=None):
        return self.native.linear_fwd(self.h.value if self.h else None, x, w, res)

    def linear_bwd_x(self, g, w, out=None):
        return self.native.linear_bwd_x(self.h.value if self.h else None, g, w, out)

    def linear_bwd_w(self, g, x, out=None):
        return self.native.linear_bwd_w(self.h.value if self.h else None, g, x, out)

    # operands split once (fp32 hi, bf16 hi and lo) and reused by several products
    def split(self, x):
        n = x[0].numel()
        out = self.torch.empty(self.lib.cnb_split_floats(n), dtype=self.torch.float32, device="cuda")
        _lib.check(self.lib.cnb_split_planes(self.h, _p(x[0]), _p(x[1]), n, _p(out), self._stream()), "split_planes")
        return out

    def linear_fwd_split(self, x_split, w_split, B, n_in, n_out, res=None, out=None):
        y = out if out is not None else self._new(B, n_out)
        _lib.check(self.lib.cnb_linear_fwd_split(self.h, _p(x_split), _p(w_split), _p(res[0]) if res else None,
                                                 _p(res[1]) if res else None, _p(y[0]), _p(y[1]), B, n_in, n_out,
                                                 self._stream()), "linear_fwd_split")
        return y

    def linear_bwd_x_split(self, g_split, w_split, B, n_in, n_out, out=None, accumulate=False):
        dx = out if out is not None else self._new(B, n_in)
        _lib.check(self.lib.cnb_linear_bwd_x_split(self.h, _p(g_split), _p(w_split), _p(dx[0]), _p(dx[1]), B, n_in,
                                                   n_out, int(accumulate), self._stream()), "linear_bwd_x_split")
        return dx

    def linear_bwd_w_split(self, g_split, x_split, B, n_in, n_out, out=None, accumulate=False):
        dw = out if out is not None else self._new(n_out, n_in)
        _lib.check(self.lib.cnb_linear_bwd_w_split(self.h, _p(g_split), _p(x_split), _p(dw[0]), _p(dw[1]), B, n_in,
                                                   n_out, int(accumulate), self._stream()), "linear_bwd_w_split")
        return dw

    def last_gemm_engine(self):
        return self.lib.cnb_last_gemm_engine()

    # ------------------------------------------------------------ FourierTrans
    def dft_fwd(self, x):
        return self.native.dft_fwd(self.h.value if self.h else None, x)

    def dft_bwd(self, g, out=None):
        return self.native.dft_bwd(self.h.value if self.h else None, g, out)

    def dft_hadamard_gelu_fwd(self, x, h, u=None, split=None):
        """FourierTrans forward with the Hadamard(h) -> CGelu tail in the same kernel: u = FFT(x) and the operand
        split of y = gelu(u o h) (y itself is not stored).  Returns (u, split)."""
        B, N = x[0].shape
        u = u if u is not None else self._like(x)
        if split is None:
            split = self.torch.empty(self.lib.cnb_split_floats(B * N), dtype=self.torch.float32, device="cuda")
        _lib.check(self.lib.cnb_dft_hadamard_gelu_fwd(self.h, _p(x[0]), _p(x[1]), _p(h[0]), _p(h[1]), _p(u[0]), _p(u[1]),
                                                      None, None, _p(split), B, N, self._stream()), "dft_hadamard_gelu_fwd")
        return u, split

    # ------------------------------------------------------------ element-wise
    def hadamard_fwd(self, u, v):
        B, N = u[0].shape
        y = self._like(u)
        _lib.check(self.lib.cnb_hadamard_fwd(self.h, _p(u[0]), _p(u[1]), _p(v[0]), _p(v[1]), int(v[0].dim() == 2),
                                             _p(y[0]), _p(y[1]), B, N, self._stream()), "hadamard_fwd")
        return y

    def hadamard_bwd(self, g, u, v):
        B, N = u[0].shape
        du = self._like(u)
        dv = self._like(v)
        _lib.check(self.lib.cnb_hadamard_bwd(self.h, _p(g[0]), _p(g[1]), _p(u[0]), _p(u[1]), _p(v[0]), _p(v[1]),
                                             int(v[0].dim() == 2), _p(du[0]), _p(du[1]), 0, _p(dv[0]), _p(dv[1]), 0,
                                             B, N, self._stream()), "hadamard_bwd")
        return du, dv

    def gelu_fwd(self, z):
        y = self._like(z)
        _lib.check(self.lib.cnb_gelu_fwd(self.h, _p(z[0]), _p(z[1]), _p(y[0]), _p(y[1]), z[0].numel(), self._stream()),
                   "gelu_fwd")
        return y

    def gelu_bwd(self, g, z):
        d = self._like(z)
        _lib.check(self.lib.cnb_gelu_bwd(self.h, _p(g[0]), _p(g[1]), _p(z[0]), _p(z[1]), _p(d[0]), _p(d[1]),
                                         z[0].numel(), 0, self._stream()), "gelu_bwd")
        return d

    def hadamard_gelu_fwd(self, u, h):
        B, N = u[0].shape
        a, y = self._like(u), self._like(u)
        _lib.check(self.lib.cnb_hadamard_gelu_fwd(self.h, _p(u[0]), _p(u[1]), _p(h[0]), _p(h[1]), _p(a[0]), _p(a[1]),
                                                  _p(y[0]), _p(y[1]), B, N, self._stream()), "hadamard_gelu_fwd")
        return a, y

    def hadamard_gelu_bwd(self, g, a, u, h):
        B, N = u[0].shape
        du, dh = self._like(u), self._like(h)
        _lib.check(self.lib.cnb_hadamard_gelu_bwd(self.h, _p(g[0]), _p(g[1]), _p(a[0]), _p(a[1]), _p(u[0]), _p(u[1]),
                                                  _p(h[0]), _p(h[1]), _p(du[0]), _p(du[1]), 0, _p(dh[0]), _p(dh[1]), 0,
                                                  B, N, self._stream()), "hadamard_gelu_bwd")
        return du, dh

    def residual_fwd(self, u, v):
        y = self._like(u)
        _lib.check(self.lib.cnb_residual_fwd(self.h, _p(u[0]), _p(u[1]), _p(v[0]), _p(v[1]), _p(y[0]), _p(y[1]),
                                             u[0].numel(), self._stream()), "residual_fwd")
        return y

    def axpy(self, src, dst, accumulate=True):
        _lib.check(self.lib.cnb_axpy(self.h, _p(src[0]), _p(src[1]), _p(dst[0]), _p(dst[1]), src[0].numel(),
                                     int(accumulate), self._stream()), "axpy")
        return dst

    # ---------------------------------------------------------- row reductions
    def softmax_fwd(self, z):
        return self.native.softmax_fwd(self.h.value if self.h else None, z)

    def softmax_bwd(self, g, z, inv):
        return self.native.softmax_bwd(self.h.value if self.h else None, g, z, inv)

    def crossent(self, z, labels, backward=True):
        return self.native.crossent(self.h.value if self.h else None, z, labels, backward)

    # --------------------------------------------------------------- embedding
    def embed_fwd(self, table, tokens):
        V, D = table[0].shape
        B, T = tokens.shape
        out = self._new(B, T * D)
        _lib.check(self.lib.cnb_embed_fwd(self.h, _p(table[0]), _p(table[1]), _p(tokens), _p(out[0]), _p(out[1]),
                                          B, T, D, V, self._stream()), "embed_fwd")
        return out

    def embed_bwd(self, g, tokens, dtable):
        V, D = dtable[0].shape
        B, T = tokens.shape
        _lib.check(self.lib.cnb_embed_bwd(self.h, _p(g[0]), _p(g[1]), _p(tokens), _p(dtable[0]), _p(dtable[1]),
                                          B, T, D, V, self._stream()), "embed_bwd")
        return dtable

    def sgd_update_split(self, w, g, lr, spans, zero_grad=True):
        """spans: [(begin, count, hi (float32), h16 (bfloat16), l16 (bfloat16))]; the updated floats of each span
        also leave their operand split: hi = w cut to TF32, h16 = bf16(hi), l16 = bf16(w - hi)."""
        arr = (_lib.SplitSpan * len(spans))()
        for k, (begin, count, hi, h16, l16) in enumerate(spans):
            arr[k].begin, arr[k].count = begin, count
            arr[k].hi, arr[k].h16, arr[k].l16 = hi.data_ptr(), h16.data_ptr(), l16.data_ptr()
        _lib.check(self.lib.cnb_sgd_update_split(self.h, _p(w), _p(g), w.numel(), lr, int(zero_grad), arr, len(spans),
                                                 self._stream()), "sgd_update_split")

    def sgd_update(self, w, g, lr, zero_grad=True):
        _lib.check(self.lib.cnb_sgd_update(self.h, _p(w), _p(g), w.numel(), lr, int(zero_grad), self._stream()),
                   "sgd_update")
