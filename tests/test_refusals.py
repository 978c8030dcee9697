"""Calls that the host refuses before anything is launched (no GPU needed: each runs in a process of its own, with addresses
that are only looked at)."""
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def refused(call: str) -> str:
    code = ("import torch, metaphor_b200 as mp\nr16, r32 = torch.float16, torch.float32\nctx = mp.StreamContext()\n" + call + "\nprint('went through')\n")
    res = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert res.returncode != 0 and "went through" not in res.stdout, (res.stdout, res.stderr)
    return res.stdout + res.stderr


# Whole chunks move r16 tensors in 16-byte pieces: one pointer two bytes behind a boundary.
@pytest.mark.parametrize("which,headdim", [(0, 64), (5, 64), (5, 128)])
def test_scan_pointers(which, headdim):
    ptrs = [1 << 20] * 7                      # x, dt, A, B, C, y, scratch
    ptrs[which] += 2
    out = refused(f"mp.launch('ssd_scan', r16, *{ptrs}, 1, 256, 2, {headdim}, 128, 1, 128, ctx)")
    assert "16-byte aligned" in out, out


@pytest.mark.parametrize("which", [3, 5, 6, 10])
def test_scan_reverse_pointers(which):
    ptrs = [1 << 20] * 12                     # x, dt, A, B, C, gy, gx, gdt, gA, gB, gC, scratch
    ptrs[which] += 2
    out = refused(f"mp.launch('ssd_scan_reverse', r16, *{ptrs}, 1, 256, 2, 64, 128, 1, 128, ctx)")
    assert "16-byte aligned" in out, out


# Operands of a fused chain.  The handle is a buffer that the library recognises as no chain and exits on, so a call whose operands are
# accepted ends the process there.
CHAIN = """
import ctypes
buf = ctypes.create_string_buffer(64)
c = mp.FusedChain.__new__(mp.FusedChain)
c.handle, c.leaves, t = ctypes.addressof(buf), ['a'], torch.zeros(4)
s = mp.Stream.__new__(mp.Stream)
s.ctx, s._open = ctx, False
class Buffer:
    def data_ptr(self):
        return 1 << 20
def closed():
    c.handle = None
    c.forward([t], t, 4, s)
"""


def test_chain_operands():
    cases = [("c.forward([t], None, 4, s)", "AttributeError"), ("c.forward([t], 1 << 20, 4, s)", "AttributeError"),
             ("c.forward([None], t, 4, s)", "AttributeError"), ("c.forward([1 << 20], t, 4, s)", "AttributeError"),
             ("c.forward([t], t, 4, ctx)", "AttributeError"), ("c.forward([t], t, 4.0, s)", "TypeError"),
             ("c.forward([t, t], t, 4, s)", "AssertionError"), ("c.reverse([t], 1 << 20, [None], 0.0, 4, s)", "AttributeError"),
             ("c.reverse([t], t, [1 << 20], 0.0, 4, s)", "AttributeError"), ("closed()", "ValueError")]
    code = CHAIN + f"got = []\nfor call, _ in {cases}:\n    try:\n        eval(call)\n    except Exception as e:\n        got.append(type(e).__name__)\n"
    assert str([want for _, want in cases]) in refused(code + "raise SystemExit(str(got))")


@pytest.mark.parametrize("call", ["c.forward([Buffer()], Buffer(), 4, s)", "c.reverse([None], None, [None], 0, 4, s)",
                                  "c.reverse([Buffer()], Buffer(), [t], 1.0, 4, s)"])
def test_chain_operands_that_are_taken(call):
    assert "not a handle from mpJitCompile" in refused(CHAIN + call)
