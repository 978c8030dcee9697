"""Small helpers over the C ABI for tests and benchmarks (torch is used for
device memory only; every computation goes through ``launch_*``)."""
from __future__ import annotations

import ctypes as C
import functools

from . import abi


@functools.lru_cache(maxsize=None)
def lib() -> C.CDLL:
    """The loaded shared library (raises ImportError when it is not built)."""
    return abi.load()


@functools.lru_cache(maxsize=None)
def _suffixes():
    import torch
    return {torch.float16: "r16", torch.float32: "r32", torch.float64: "r64"}


def suffix_of(dtype) -> str:
    """Dtype-key suffix in the order of the reference's scalar.zig Tag enum."""
    return _suffixes()[dtype]


def _arg(a):
    # torch tensors are passed as raw device pointers
    if hasattr(a, "data_ptr"):
        return C.c_void_p(a.data_ptr())
    if a is None:
        return C.c_void_p(0)
    return a


class Stream:
    """A StreamContext obtained from mpInitStream (own stream) or mpWrapStream
    (``wrap`` = an existing ``cudaStream_t`` value, e.g. torch's current stream)."""

    def __init__(self, wrap: int | None = None):
        self._lib = lib()
        if wrap is None:
            self.ctx = self._lib.mpInitStream()
        else:
            self.ctx = self._lib.mpWrapStream(C.c_void_p(wrap))
        self._open = True

    @property
    def handle(self) -> int:
        return self.ctx.cuda_stream.ptr or 0

    def torch_stream(self):
        import torch
        return torch.cuda.ExternalStream(self.handle)

    def sync(self):
        self._lib.mpStreamSynchronize(self.ctx)

    def status(self) -> int:
        return int(self._lib.mpGetStatus(self.ctx))

    def close(self):
        if self._open:
            self._lib.mpDeinitStream(self.ctx)
            self._open = False

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.close()


def _launch_ctypes(name: str, dtype, *args):
    """``launch`` for arguments that the native path does not convert itself."""
    fn = getattr(lib(), f"launch_{name}_{suffix_of(dtype)}")
    conv = [_arg(a) for a in args[:-1]]
    ctx = args[-1].ctx if isinstance(args[-1], Stream) else args[-1]
    fn(*conv, ctx)


@functools.lru_cache(maxsize=None)
def _native():
    """The native call path (host/py_launch.cpp); raises ImportError while it, or the library behind it, is not built."""
    import importlib.machinery
    import importlib.util
    lib()
    path = abi.LIB_PATH.parent / "mp_launch.so"
    if not path.exists():
        raise ImportError(f"{path} is missing: run `python -m metaphor_b200.build` (needs nvcc)")
    import torch
    loader = importlib.machinery.ExtensionFileLoader("mp_launch", str(path))
    mod = importlib.util.module_from_spec(importlib.util.spec_from_loader("mp_launch", loader))
    loader.exec_module(mod)
    mod.setup((torch.float16, torch.float32, torch.float64), torch.Tensor, C.Array, C.c_void_p, abi.StreamContext, Stream, _launch_ctypes)
    return mod


try:
    launch = _native().launch
except ImportError:      # not built yet, or built from other sources: this package also holds the build
    def launch(name: str, dtype, *args):
        """``launch_<name>_<suffix>(*args)`` as soon as the library is built."""
        return _native().launch(name, dtype, *args)


class FusedChain:
    """A JIT-compiled element-wise expression (include/mp_jit.h)."""

    def __init__(self, expr: str, dtype):
        self._lib = lib()
        _native()
        self.dtype = dtype
        key = {"r16": 0, "r32": 1, "r64": 2}[suffix_of(dtype)]
        self.handle = self._lib.mpJitCompile(expr.encode(), key)
        if not self.handle:
            raise ValueError(f"cannot compile expression {expr!r}")
        n = self._lib.mpJitNumLeaves(self.handle)
        self.leaves = [self._lib.mpJitLeafName(self.handle, i).decode() for i in range(n)]

    def forward(self, leaves, out, n, stream):
        assert len(leaves) == len(self.leaves)
        _native().chain_forward(self.handle, leaves, out, n, stream.ctx)

    def reverse(self, leaves, g_out, g_leaves, alpha, n, stream):
        assert len(leaves) == len(self.leaves) == len(g_leaves)
        _native().chain_reverse(self.handle, leaves, g_out, g_leaves, float(alpha), n, stream.ctx)

    def close(self):
        if self.handle:
            self._lib.mpJitRelease(self.handle)
            self.handle = None
