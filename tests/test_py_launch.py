"""The native call path of `launch` (host/py_launch.cpp): every form of an argument is taken, or refused, as ctypes takes or refuses it,
and arrives at the launcher with the same value."""
import ctypes as C

import numpy as np
import pytest


def both(mp):
    from metaphor_b200 import runtime
    return runtime._native().launch, runtime._launch_ctypes


def outcome(call, *args, **kw):
    try:
        call(*args, **kw)
        return "taken"
    except Exception as e:
        return type(e).__name__


def test_taken_and_refused_alike(mp):
    """No elements: the launchers return before they touch CUDA."""
    import torch
    r32, ctx = torch.float32, mp.StreamContext()
    stream = mp.Stream.__new__(mp.Stream)
    stream.ctx, stream._open = ctx, False

    class Buffer:
        def data_ptr(self):
            return 16

    class Sub(torch.Tensor):
        pass

    t = torch.zeros(4)
    pointers = [t, t.as_subclass(Sub), torch.nn.Parameter(t), Buffer(), None, 16, True, 1 << 64, -1, 1.0, "16", b"16", C.c_void_p(16), C.c_void_p(), (C.c_ulong * 2)(1, 2),
                C.pointer(C.c_int(1)), C.byref(C.c_int(1)), [16], np.zeros(2)]
    doubles = [1.0, 1, True, 1 << 2000, np.float64(1), np.float32(1), np.int64(1), "1", None, C.c_double(1), t]
    counts = [0, False, 1 << 64, -(1 << 64), 0.0, np.int64(0), None, "0", C.c_ulong(0), C.c_ulong(0).value]
    ends = [ctx, stream, None, 0, ctx.cuda_stream]
    calls = [("fill", r32, p, 1.0, 0, ctx) for p in pointers] + [("fill", r32, t, d, 0, ctx) for d in doubles]
    calls += [("fill", r32, t, 1.0, n, ctx) for n in counts] + [("fill", r32, t, 1.0, 0, e) for e in ends]
    calls += [("fill", d, t, 1.0, 0, ctx) for d in (torch.float16, torch.float64, torch.bfloat16, "r32", None)]
    calls += [("no_such_launcher", r32, t, 0, ctx), ("fill", r32, t, 1.0, ctx), ("fill", r32, t, 1.0, 0, 0, ctx), ("fill", r32), (7, r32, t, ctx),
              ("permutate", r32, t, t, 0.0, (C.c_ulong * 2)(0, 1), (C.c_ulong * 2)(1, 0), 2, ctx)]
    native, plain = both(mp)
    for args in calls:
        assert outcome(native, *args) == outcome(plain, *args), args
    assert outcome(native, name="fill", dtype=r32) == outcome(plain, name="fill", dtype=r32)


@pytest.mark.gpu
def test_values_arrive_alike(mp, stream):
    import torch
    n = 1000
    src = torch.randn(n, device="cuda")
    for scale in (0.75, 3, True, np.float64(0.3), np.float32(0.3), C.c_double(0.7), -0.0, float("inf")):
        for count in (n, 0, 1, n + (1 << 64)):
            outs = []
            for call in both(mp):
                out = torch.full((n,), 7.0, device="cuda")
                torch.cuda.current_stream().synchronize()
                call("dilate", torch.float32, src, scale, out, count, stream)
                call("dilate", torch.float32, C.c_void_p(src.data_ptr()), scale, out.data_ptr(), count, stream.ctx)
                stream.sync()
                outs.append(out)
            assert torch.equal(outs[0].nan_to_num(), outs[1].nan_to_num()), (scale, count)
            want = src[:count % (1 << 64)] * float(getattr(scale, "value", scale))
            assert torch.equal(outs[0][:want.numel()].nan_to_num(), want.nan_to_num()) and torch.all(outs[0][want.numel():] == 7), (scale, count)
    sizes, perm = (C.c_ulong * 3)(10, 20, 5), (C.c_ulong * 3)(2, 0, 1)
    outs = []
    for call in both(mp):
        out = torch.zeros(n, device="cuda")
        torch.cuda.current_stream().synchronize()
        call("permutate", torch.float32, src, out, 0.0, sizes, perm, 3, stream)
        stream.sync()
        outs.append(out)
    assert torch.equal(*outs) and torch.equal(outs[0].sort().values, src.sort().values)
