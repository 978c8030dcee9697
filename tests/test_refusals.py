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
