"""GPU parity of the Mamba-2 SSD chunked scan (forward and reverse, r16 storage,
fp32 accumulation) against the sequential-recurrence CPU oracle in float64.
Inputs follow the benchmark configuration's distributions: x, B, C ~ N(0,1) in
r16, dt = softplus(N(-4,1)), A = -exp(U(log 1, log 16))."""
import numpy as np
import pytest

from util import assert_close, dev, host

pytestmark = pytest.mark.gpu

TOL = 1e-2   # r16 storage


def make_inputs(seed, nb, L, H, P, N, G):
    r = np.random.default_rng(seed)
    x = r.standard_normal((nb, L, H, P)).astype(np.float16)
    Bm = r.standard_normal((nb, L, G, N)).astype(np.float16)
    Cm = r.standard_normal((nb, L, G, N)).astype(np.float16)
    dt = np.log1p(np.exp(r.standard_normal((nb, L, H)) - 4.0)).astype(np.float32)
    A = (-np.exp(r.uniform(0.0, np.log(16.0), H))).astype(np.float32)
    gy = r.standard_normal((nb, L, H, P)).astype(np.float16)
    return x, dt, A, Bm, Cm, gy


def scratch_for(mp, dims, reverse):
    import torch
    n = mp.lib().mpSsdScanScratchBytes(*dims, 1 if reverse else 0)
    return torch.empty(n, dtype=torch.uint8, device="cuda")


CASES = [  # (batch, seqlen, heads, headdim, dstate, groups, chunk)
    (2, 512, 4, 64, 128, 1, 256),
    (1, 768, 4, 64, 128, 2, 256),
    (2, 256, 2, 64, 128, 1, 128),
    (1, 512, 2, 128, 128, 1, 256),
    # more sequences than SMs (and than half of them, the reverse's share per walk): the chunk walk gives every CTA the
    # same number of chunks, so sequences are cut between CTAs and their state crosses through global memory
    (10, 384, 16, 64, 128, 1, 128),
    (5, 640, 20, 64, 128, 2, 128),
]


@pytest.mark.parametrize("dims", CASES)
def test_ssd_forward(mp, stream, orc, dims):
    import torch
    nb, L, H, P, N, G, Q = dims
    x, dt, A, Bm, Cm, _ = make_inputs(0, nb, L, H, P, N, G)
    y = dev(np.full(x.shape, np.nan, np.float16))
    scratch = scratch_for(mp, dims, False)
    args = [dev(a) for a in (x, dt, A, Bm, Cm)]
    torch.cuda.current_stream().synchronize()
    mp.launch("ssd_scan", torch.float16, *args, y, scratch, nb, L, H, P, N, G, Q, stream)
    stream.sync()
    assert stream.status() == 0
    f64 = lambda a: np.ascontiguousarray(a.astype(np.float64))
    ref = orc.ssd_forward(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm))
    assert_close(host(y), ref.astype(np.float16), TOL, f"ssd forward {dims}")


@pytest.mark.parametrize("dims", CASES)
def test_ssd_reverse(mp, stream, orc, dims):
    import torch
    nb, L, H, P, N, G, Q = dims
    x, dt, A, Bm, Cm, gy = make_inputs(1, nb, L, H, P, N, G)
    gx = dev(np.full(x.shape, np.nan, np.float16)); gdt = dev(np.full(dt.shape, np.nan, np.float32))
    gA = dev(np.full(A.shape, np.nan, np.float32)); gB = dev(np.full(Bm.shape, np.nan, np.float16))
    gC = dev(np.full(Cm.shape, np.nan, np.float16))
    scratch = scratch_for(mp, dims, True)
    args = [dev(a) for a in (x, dt, A, Bm, Cm, gy)]
    torch.cuda.current_stream().synchronize()
    mp.launch("ssd_scan_reverse", torch.float16, *args, gx, gdt, gA, gB, gC, scratch, nb, L, H, P, N, G, Q, stream)
    stream.sync()
    assert stream.status() == 0
    f64 = lambda a: np.ascontiguousarray(a.astype(np.float64))
    rgx, rgdt, rgA, rgB, rgC = orc.ssd_reverse(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm), f64(gy))
    assert_close(host(gx), rgx.astype(np.float16), TOL, f"gx {dims}")
    assert_close(host(gC), rgC.astype(np.float16), TOL, f"gC {dims}")
    assert_close(host(gB), rgB.astype(np.float16), TOL, f"gB {dims}")
    assert_close(host(gdt), rgdt, TOL, f"gdt {dims}")
    assert_close(host(gA), rgA, TOL, f"gA {dims}")


def test_full_length_against_the_sequential_path(mp, stream):
    """Benchmark-length sequences (seqlen 8192 = 32 chunks, 32 heads, one batch): the chunked tensor-core path
    against the sequential-recurrence kernels of the same library, forward and every gradient."""
    import os
    import torch
    dims = (1, 8192, 32, 64, 128, 1, 256)
    nb, L, H, P, N, G, Q = dims
    x, dt, A, Bm, Cm, gy = make_inputs(11, nb, L, H, P, N, G)
    args = [dev(a) for a in (x, dt, A, Bm, Cm)]
    dgy = dev(gy)
    lib = mp.lib()
    out = {}
    for path in ("tensor", "sequential"):
        if path == "sequential":
            os.environ["MP_SSD_FORCE_GENERIC"] = "1"
        try:
            n = max(lib.mpSsdScanScratchBytes(*dims, 0), lib.mpSsdScanScratchBytes(*dims, 1))
            scr = torch.empty(n, dtype=torch.uint8, device="cuda")
            y = dev(np.full(x.shape, np.nan, np.float16))
            gx = dev(np.full(x.shape, np.nan, np.float16)); gdt = dev(np.full(dt.shape, np.nan, np.float32))
            gA = dev(np.full(A.shape, np.nan, np.float32)); gB = dev(np.full(Bm.shape, np.nan, np.float16)); gC = dev(np.full(Cm.shape, np.nan, np.float16))
            torch.cuda.current_stream().synchronize()
            mp.launch("ssd_scan", torch.float16, *args, y, scr, *dims, stream)
            mp.launch("ssd_scan_reverse", torch.float16, *args, dgy, gx, gdt, gA, gB, gC, scr, *dims, stream)
            stream.sync()
            assert stream.status() == 0
            out[path] = [host(t).astype(np.float64) for t in (y, gx, gdt, gA, gB, gC)]
        finally:
            os.environ.pop("MP_SSD_FORCE_GENERIC", None)
    for got, want, name in zip(out["tensor"], out["sequential"], ("y", "gx", "gdt", "gA", "gB", "gC")):
        assert_close(got, want, 1e-2, f"full-length {name}")


@pytest.mark.parametrize("dims", [(2, 512, 4, 64, 128, 1, 256), (10, 384, 16, 64, 128, 1, 128), (1, 512, 2, 128, 128, 1, 256)])
def test_scan_from_raw_step_sizes_is_the_three_launches_in_one(mp, stream, dims):
    """launch_ssd_scan_raw (softplus of the raw step sizes and -exp(A_log) inside the scan) against launch_softplus_bias +
    launch_neg_exp + launch_ssd_scan on the same inputs: dt, A and y bit for bit (the last shape takes the composed path)."""
    import torch
    nb, L, H, P, N, G, Q = dims
    x, _, _, Bm, Cm, _ = make_inputs(5, nb, L, H, P, N, G)
    r = np.random.default_rng(6)
    pitch = H + 8
    raw = (r.standard_normal((nb * L, pitch)) - 4.0).astype(np.float16)
    bias = (0.5 * r.standard_normal(H)).astype(np.float32)
    A_log = np.log(r.uniform(1.0, 16.0, H)).astype(np.float32)
    dx, dB, dC, draw, dbias, dAlog = (dev(a) for a in (x, Bm, Cm, raw, bias, A_log))
    scratch = scratch_for(mp, dims, False)
    dt1 = dev(np.full((nb, L, H), np.nan, np.float32)); A1 = dev(np.full(H, np.nan, np.float32)); y1 = dev(np.full(x.shape, np.nan, np.float16))
    dt2 = dev(np.full((nb, L, H), np.nan, np.float32)); A2 = dev(np.full(H, np.nan, np.float32)); y2 = dev(np.full(x.shape, np.nan, np.float16))
    torch.cuda.current_stream().synchronize()
    mp.launch("softplus_bias", torch.float16, draw, pitch, dbias, dt1, nb * L, H, stream)
    mp.launch("neg_exp", torch.float32, dAlog, A1, H, stream)
    mp.launch("ssd_scan", torch.float16, dx, dt1, A1, dB, dC, y1, scratch, *dims, stream)
    mp.launch("ssd_scan_raw", torch.float16, dx, draw, pitch, dbias, dAlog, dB, dC, y2, dt2, A2, scratch, *dims, stream)
    stream.sync()
    assert stream.status() == 0
    assert np.array_equal(host(dt1), host(dt2))
    assert np.array_equal(host(A1), host(A2))
    assert np.array_equal(host(y1), host(y2))
    assert np.isfinite(host(y2).astype(np.float32)).all()


@pytest.mark.parametrize("dims", [(2, 512, 4, 64, 128, 1, 256), (10, 384, 16, 64, 128, 1, 128), (1, 512, 2, 128, 128, 1, 256)])
def test_reverse_with_the_raw_side_gradients_is_the_three_launches_in_one(mp, stream, dims):
    """launch_ssd_scan_reverse_raw against launch_ssd_scan_reverse + launch_softplus_bias_reverse + launch_hadamard_reverse:
    gx, gdt, gA, gB, gC and the raw step sizes' gradient bit for bit, the accumulated dt_bias / A_log gradients to 1e-5."""
    import torch
    nb, L, H, P, N, G, Q = dims
    x, _, _, Bm, Cm, gy = make_inputs(7, nb, L, H, P, N, G)
    r = np.random.default_rng(8)
    pitch = H + 8
    raw = (r.standard_normal((nb * L, pitch)) - 4.0).astype(np.float16)
    bias = (0.5 * r.standard_normal(H)).astype(np.float32)
    A_log = np.log(r.uniform(1.0, 16.0, H)).astype(np.float32)
    dx, dB, dC, dgy, draw, dbias, dAlog = (dev(a) for a in (x, Bm, Cm, gy, raw, bias, A_log))
    dt = dev(np.zeros((nb, L, H), np.float32)); A = dev(np.zeros(H, np.float32))
    torch.cuda.current_stream().synchronize()
    mp.launch("softplus_bias", torch.float16, draw, pitch, dbias, dt, nb * L, H, stream)
    mp.launch("neg_exp", torch.float32, dAlog, A, H, stream)
    scratch = scratch_for(mp, dims, True)
    gb0 = r.standard_normal(H).astype(np.float32); gl0 = r.standard_normal(H).astype(np.float32)
    outs = []
    for fused in (False, True):
        gx = dev(np.full(x.shape, np.nan, np.float16)); gdt = dev(np.full((nb, L, H), np.nan, np.float32)); gA = dev(np.full(H, np.nan, np.float32))
        gB = dev(np.full(Bm.shape, np.nan, np.float16)); gC = dev(np.full(Cm.shape, np.nan, np.float16))
        graw = dev(np.full((nb * L, pitch), 2, np.float16)); gbias = dev(gb0.copy()); glog = dev(gl0.copy())
        torch.cuda.current_stream().synchronize()
        if fused:
            mp.launch("ssd_scan_reverse_raw", torch.float16, dx, dt, A, dB, dC, dgy, draw, pitch, dbias, gx, gdt, gA, graw, pitch, gbias, glog,
                      gB, gC, scratch, *dims, stream)
        else:
            mp.launch("ssd_scan_reverse", torch.float16, dx, dt, A, dB, dC, dgy, gx, gdt, gA, gB, gC, scratch, *dims, stream)
            mp.launch("softplus_bias_reverse", torch.float16, draw, pitch, dbias, gdt, graw, pitch, gbias, nb * L, H, stream)
            mp.launch("hadamard_reverse", torch.float32, gA, A, glog, H, stream)
        stream.sync()
        assert stream.status() == 0
        outs.append([host(t) for t in (gx, gdt, gA, gB, gC, graw, gbias, glog)])
    for a, b, name in zip(outs[0][:6], outs[1][:6], ("gx", "gdt", "gA", "gB", "gC", "graw")):
        assert np.array_equal(a, b), name
    assert np.all(outs[1][5][:, H:] == 2)
    for a, b, name in zip(outs[0][6:], outs[1][6:], ("gdt_bias", "gA_log")):
        assert_close(b, a.astype(np.float64), 1e-5, name)


def test_scans_on_several_streams_share_a_bias_gradient(mp):
    """Every scan adds its step sizes' bias gradient: 4 streams x 16 scans of the same inputs into one vector."""
    import torch
    dims = nb, L, H, P, N, G, Q = 1, 128, 8, 64, 128, 1, 128
    x, _, _, Bm, Cm, gy = make_inputs(30, *dims[:-1])
    ins = [dev(a) for a in (x, np.full((nb, L, H), 0.5, np.float32), -np.ones(H, np.float32), Bm, Cm)]
    zero, draw, dbias, dgy = dev(np.zeros(H, np.float32)), dev(np.zeros((nb * L, H), np.float16)), dev(np.zeros(H, np.float32)), dev(gy)
    shared = torch.zeros_like(zero)

    class Lane:
        def __init__(self):
            self.stream = mp.Stream()
            self.out = [torch.empty_like(t) for t in (ins[0], ins[1], ins[2], draw, ins[3], ins[4])]
            self.scratch = scratch_for(mp, dims, True)

        def scan(self, gbias):
            gx, gdt, gA, graw, gB, gC = self.out
            mp.launch("ssd_scan_reverse_raw", torch.float16, *ins, dgy, draw, H, dbias, gx, gdt, gA, graw, H, gbias, None, gB, gC, self.scratch, *dims,
                      self.stream)

    lanes = [Lane() for _ in range(4)]
    one = torch.zeros_like(zero)
    torch.cuda.synchronize()
    lanes[0].scan(one)
    lanes[0].stream.sync()
    for _ in range(16):
        for lane in lanes:
            lane.scan(shared)
    for lane in lanes:
        lane.stream.sync()
        assert lane.stream.status() == 0
        lane.stream.close()
    # 64 additions of one value: each rounds the sum, by 2^-24 of it at most
    np.testing.assert_allclose(host(shared), 64 * host(one).astype(np.float64), rtol=64 * 2.0 ** -24)


@pytest.mark.parametrize("dims", [
    # (batch, seqlen, heads, headdim, dstate, groups, chunk): the chunk walk on lengths that are no multiple of its 128-step
    # chunk - the shortest, less than one chunk, one step past a chunk, one step short of one, and sequences cut between CTAs
    (2, 32, 2, 64, 128, 1, 128), (1, 50, 4, 64, 128, 2, 64), (2, 129, 2, 64, 128, 1, 128), (1, 383, 4, 64, 128, 1, 256),
    (10, 333, 16, 64, 128, 1, 128)])
def test_ssd_on_ragged_lengths(mp, stream, orc, dims):
    import torch
    nb, L, H, P, N, G, Q = dims
    x, dt, A, Bm, Cm, gy = make_inputs(9, nb, L, H, P, N, G)
    f64 = lambda a: np.ascontiguousarray(a.astype(np.float64))
    args = [dev(a) for a in (x, dt, A, Bm, Cm)]
    # outputs carry guard rows: nothing may be written behind the last step of the last batch entry
    guarded = lambda a: dev(np.full((a.size + 4096,), np.nan, a.dtype))
    y, gx, gdt, gB, gC = (guarded(a) for a in (x, x, dt, Bm, Cm))
    gA = dev(np.full(A.shape, np.nan, np.float32))
    n = max(mp.lib().mpSsdScanScratchBytes(*dims, 0), mp.lib().mpSsdScanScratchBytes(*dims, 1))
    scratch = torch.full((n,), 255, dtype=torch.uint8, device="cuda")
    torch.cuda.current_stream().synchronize()
    mp.launch("ssd_scan", torch.float16, *args, y, scratch, *dims, stream)
    mp.launch("ssd_scan_reverse", torch.float16, *args, dev(gy), gx, gdt, gA, gB, gC, scratch, *dims, stream)
    stream.sync()
    assert stream.status() == 0
    ref = (orc.ssd_forward(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm)),) + tuple(orc.ssd_reverse(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm), f64(gy)))
    for got, want, name in zip((y, gx, gdt, gA, gB, gC), ref, ("y", "gx", "gdt", "gA", "gB", "gC")):
        got = host(got)
        assert np.isnan(got[want.size:]).all(), f"{name} written past its end {dims}"
        assert_close(got[:want.size].reshape(want.shape), want.astype(got.dtype), TOL, f"{name} {dims}")


@pytest.mark.parametrize("dims,shift", [
    # (batch, seqlen, heads, headdim, dstate, groups, chunk), shift of the raw step sizes.  The walk takes two heads of a group at a time
    # where there are enough sequences: uncut in the forward and cut in the reverse, cut in both (two groups), an odd number of
    # heads per group beside it (one head at a time), and steps that decay by more than e^-80 in eight, whose mask is made step by step.
    # The lengths that are no multiple of the chunk take the fp32 segments.
    ((14, 300, 16, 64, 128, 1, 128), 0.0), ((20, 256, 32, 64, 128, 2, 128), 0.0), ((20, 200, 15, 64, 128, 1, 128), 0.0),
    ((14, 200, 16, 64, 128, 1, 128), 7.0), ((20, 160, 15, 64, 128, 1, 128), 7.0), ((14, 384, 16, 64, 128, 1, 128), 0.0),
    ((20, 256, 15, 64, 128, 1, 128), 0.0), ((14, 256, 16, 64, 128, 1, 128), 7.0), ((20, 128, 15, 64, 128, 1, 128), 7.0)])
def test_ssd_heads_in_pairs(mp, stream, orc, dims, shift):
    import torch
    nb, L, H, P, N, G, Q = dims
    x, dt, A, Bm, Cm, gy = make_inputs(12, nb, L, H, P, N, G)
    if shift:
        dt = (dt + shift * np.random.default_rng(13).uniform(size=dt.shape)).astype(np.float32)
    f64 = lambda a: np.ascontiguousarray(a.astype(np.float64))
    args = [dev(a) for a in (x, dt, A, Bm, Cm)]
    y, gx, gdt, gA, gB, gC = (dev(np.full(a.shape, np.nan, a.dtype)) for a in (x, x, dt, A, Bm, Cm))
    n = max(mp.lib().mpSsdScanScratchBytes(*dims, 0), mp.lib().mpSsdScanScratchBytes(*dims, 1))
    scratch = torch.full((n,), 255, dtype=torch.uint8, device="cuda")
    torch.cuda.current_stream().synchronize()
    mp.launch("ssd_scan", torch.float16, *args, y, scratch, *dims, stream)
    mp.launch("ssd_scan_reverse", torch.float16, *args, dev(gy), gx, gdt, gA, gB, gC, scratch, *dims, stream)
    stream.sync()
    assert stream.status() == 0
    ref = (orc.ssd_forward(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm)),) + tuple(orc.ssd_reverse(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm), f64(gy)))
    for got, want, name in zip((y, gx, gdt, gA, gB, gC), ref, ("y", "gx", "gdt", "gA", "gB", "gC")):
        got = host(got)
        if shift and name == "gA" and L % Q == 0:
            # The walk's g_a is a sum of differences of row dots whose r16 score tiles round differently: over a chunk's steps up to
            # 2^-11 sqrt(128) of a row dot v = <gx, x>, which under strong decay is all of gA.
            v = np.abs((ref[1] * f64(x)).sum(-1))
            bound = 2.0 ** -11 * np.sqrt(128) * (f64(dt) * v).sum((0, 1))
            assert np.all(np.abs(got - want) <= bound), (np.abs(got - want) / bound).max()
        else:
            assert_close(got, want.astype(got.dtype), TOL, f"{name} {dims} {shift}")


@pytest.mark.parametrize("dims,shift", [((14, 384, 16, 64, 128, 1, 128), 0.0), ((20, 256, 32, 64, 128, 2, 256), 0.0), ((8, 512, 24, 64, 128, 1, 256), 0.0),
                                        ((14, 256, 16, 64, 128, 1, 128), 7.0)])
def test_ssd_heads_in_pairs_have_the_bits_of_single_heads(mp, stream, monkeypatch, dims, shift):
    """Whether the walk takes two heads of a group at a time depends on the batch size; its results must not."""
    import torch
    x, dt, A, Bm, Cm, gy = make_inputs(23, *dims[:-1])
    if shift:
        dt = (dt + shift * np.random.default_rng(24).uniform(size=dt.shape)).astype(np.float32)
    args = [dev(a) for a in (x, dt, A, Bm, Cm)]
    dgy = dev(gy)
    outs = []
    for single in (False, True):
        if single:
            monkeypatch.setenv("MP_SSD_WALK_NO_PAIRS", "1")      # read at every launch
        y, gx, gdt, gA, gB, gC = (dev(np.full(a.shape, np.nan, a.dtype)) for a in (x, x, dt, A, Bm, Cm))
        scratch = scratch_for(mp, dims, True)
        torch.cuda.current_stream().synchronize()
        mp.launch("ssd_scan", torch.float16, *args, y, scratch, *dims, stream)
        mp.launch("ssd_scan_reverse", torch.float16, *args, dgy, gx, gdt, gA, gB, gC, scratch, *dims, stream)
        stream.sync()
        assert stream.status() == 0
        outs.append((y, gx, gdt, gA, gB, gC))
    for a, b, name in zip(*outs, ("y", "gx", "gdt", "gA", "gB", "gC")):
        assert torch.equal(a, b), name


@pytest.mark.parametrize("dims,shift,off", [
    # (batch, seqlen, heads, headdim, dstate, groups, chunk), shift of the raw step sizes, elements between a 16-byte boundary and the
    # r16 bases.  fp32 segments of 64 steps: one segment and its edges, several, one step past a segment and one short of it, whole
    # lengths with a chunk that the chunk walk does not take, groups of one head and of an odd number, group gradients in one share
    # of the heads and in several
    ((2, 32, 2, 64, 128, 1, 128), 0.0, 0), ((1, 63, 4, 64, 128, 2, 64), 0.0, 1), ((2, 64, 3, 64, 128, 3, 64), 0.0, 0), ((2, 65, 5, 64, 128, 1, 128), 7.0, 1),
    ((1, 383, 4, 64, 128, 1, 256), 0.0, 0), ((2, 256, 6, 64, 128, 2, 64), 0.0, 3), ((2, 200, 16, 64, 128, 1, 128), 7.0, 0), ((1, 1000, 24, 64, 128, 1, 128), 0.0, 0),
    ((10, 4033, 2, 64, 128, 1, 128), 0.0, 0)])
def test_ssd_segments_keep_fp32(mp, stream, orc, dims, shift, off):
    import torch
    nb, L, H, P, N, G, Q = dims
    x, dt, A, Bm, Cm, gy = make_inputs(21, nb, L, H, P, N, G)
    if shift:
        dt = (dt + shift * np.random.default_rng(22).uniform(size=dt.shape)).astype(np.float32)

    def placed(a):     # r16: `off` elements behind a 16-byte boundary, guard values on both sides
        o = off if a.dtype == np.float16 else 0
        flat = dev(np.full((a.size + o + 64,), 7, a.dtype))
        flat[o:o + a.size] = torch.from_numpy(a.reshape(-1)).cuda()
        return flat, flat[o:o + a.size]

    ins = [placed(a)[1] for a in (x, dt, A, Bm, Cm)]
    outs = [placed(np.full(a.shape, np.nan, a.dtype)) for a in (x, x, dt, A, Bm, Cm)]
    y, gx, gdt, gA, gB, gC = (o[1] for o in outs)
    n = max(mp.lib().mpSsdScanScratchBytes(*dims, 0), mp.lib().mpSsdScanScratchBytes(*dims, 1))
    scratch = torch.full((n + 1,), 255, dtype=torch.uint8, device="cuda")[off % 2:]
    torch.cuda.current_stream().synchronize()
    mp.launch("ssd_scan", torch.float16, *ins, y, scratch, *dims, stream)
    mp.launch("ssd_scan_reverse", torch.float16, *ins, placed(gy)[1], gx, gdt, gA, gB, gC, scratch, *dims, stream)
    stream.sync()
    assert stream.status() == 0
    f64 = lambda a: np.ascontiguousarray(a.astype(np.float64))
    ref = (orc.ssd_forward(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm)),) + tuple(orc.ssd_reverse(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm), f64(gy)))
    # r16 results: the rounding of the result itself, at most 2^-11 / sqrt(3) of its norm.  r32 results: fp32 sums, 2^-24 times the square
    # root of a few hundred terms; gA sums both signs, which leaves it a tenth of its terms' norm.
    tol = dict(y=2.9e-4, gx=2.9e-4, gB=2.9e-4, gC=2.9e-4, gdt=2e-6, gA=2e-5)
    for (flat, got), want, name in zip(outs, ref, ("y", "gx", "gdt", "gA", "gB", "gC")):
        o = off if flat.dtype == torch.float16 else 0
        assert torch.all(flat[:o] == 7) and torch.all(flat[o + want.size:] == 7), f"{name} written outside {dims}"
        d = host(got).astype(np.float64).reshape(want.shape) - want
        assert np.linalg.norm(d) <= tol[name] * np.linalg.norm(want), (name, np.linalg.norm(d) / np.linalg.norm(want))


@pytest.mark.parametrize("which", ["x", "gy", "dt", "C"])
def test_ssd_segments_of_values_far_apart(mp, stream, orc, which):
    """Values of one 16 x 16 block up to 2^33 apart, the large ones against zeros of the other operand: the small ones alone make the results and
    keep their bits.  A channel of x (of gy) at the end of r16's range where gy (x) has none, next to channels of 1e-5; step sizes of 1e-10
    next to 1 where x is zero; rows of C at the end of the range where gy is zero, next to some of 1e-5."""
    import torch
    dims = (1, 200, 4, 64, 128, 2, 128)
    nb, L, H, P, N, G, Q = dims
    x, dt, A, Bm, Cm, gy = (a.astype(np.float64) for a in make_inputs(41, nb, L, H, P, N, G))
    late = np.arange(L) % 16 >= 8
    if which in ("x", "gy"):
        large, other = (x, gy) if which == "x" else (gy, x)
        Bm, Cm = 0.05 * Bm, 0.05 * Cm
        large *= 1e-5
        large[..., 3], other[..., 3] = 3e4, 0.0
        other *= 1e3
    elif which == "dt":
        A *= 0.02
        Bm, Cm = 30 * Bm, 30 * Cm
        dt[:] = np.where(late, 1.0, 1e-10)[None, :, None]
        x *= np.where(late, 0.0, 1000.0)[None, :, None, None]
        gy *= 1e-2
    else:
        Bm, gy = 0.05 * Bm, 1e3 * gy
        Cm *= np.where(late, 1e4, 1e-5)[None, :, None, None]
        gy[:, late] = 0
    x, Bm, Cm, gy = (a.astype(np.float16) for a in (x, Bm, Cm, gy))
    dt, A = dt.astype(np.float32), A.astype(np.float32)
    args = [dev(a) for a in (x, dt, A, Bm, Cm)]
    y, gx, gdt, gA, gB, gC = (dev(np.full(a.shape, np.nan, a.dtype)) for a in (x, x, dt, A, Bm, Cm))
    scratch = scratch_for(mp, dims, True)
    torch.cuda.current_stream().synchronize()
    mp.launch("ssd_scan", torch.float16, *args, y, scratch, *dims, stream)
    mp.launch("ssd_scan_reverse", torch.float16, *args, dev(gy), gx, gdt, gA, gB, gC, scratch, *dims, stream)
    stream.sync()
    assert stream.status() == 0
    f64 = lambda a: np.ascontiguousarray(a.astype(np.float64))
    ref = (orc.ssd_forward(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm)),) + tuple(orc.ssd_reverse(f64(x), f64(dt), f64(A), f64(Bm), f64(Cm), f64(gy)))
    for got, want, name in zip((y, gx, gB, gC), (ref[0], ref[1], ref[4], ref[5]), ("y", "gx", "gB", "gC")):
        # every row by itself, up to the rounding of its r16 values: 2^-11 / sqrt(3) of its norm, and half of 2^-24 each where that is more
        d = np.linalg.norm(host(got).astype(np.float64) - want, axis=-1)
        bound = 4e-4 * np.linalg.norm(want, axis=-1) + 2.0 ** -25 * np.sqrt(want.shape[-1])
        if name == {"x": "y", "gy": "gx"}.get(which):     # (the large channel alone would be seen)
            d = np.linalg.norm(np.delete(host(got).astype(np.float64) - want, 3, -1), axis=-1)
            bound = 4e-4 * np.linalg.norm(np.delete(want, 3, -1), axis=-1) + 2.0 ** -25 * np.sqrt(want.shape[-1])
        assert np.all(d <= bound), (name, (d / bound).max())
    d = host(gdt).astype(np.float64) - ref[2]
    assert np.linalg.norm(d) <= 2e-6 * np.linalg.norm(ref[2]), ("gdt", np.linalg.norm(d) / np.linalg.norm(ref[2]))


@pytest.mark.parametrize("which,value,dims", [
    # an infinity or a NaN at two steps, in the middle of a segment and in the last one, which is partly filled: no product may carry it to a step or
    # a column that the recurrence keeps finite, and what is finite keeps its accuracy
    (0, np.inf, (1, 200, 4, 64, 128, 2, 128)), (3, -np.inf, (1, 200, 4, 64, 128, 2, 128)), (4, np.inf, (1, 200, 4, 64, 128, 2, 128)),
    (5, np.inf, (1, 200, 4, 64, 128, 2, 128)), (0, np.nan, (1, 200, 4, 64, 128, 2, 128)), (3, np.inf, (2, 50, 2, 64, 128, 1, 128))])
def test_ssd_segments_with_infinities(mp, stream, orc, which, value, dims):
    import torch
    nb, L, H, P, N, G, Q = dims
    ins = list(make_inputs(31, nb, L, H, P, N, G))   # x, dt, A, B, C, gy
    ins[which][0, 27, 0, 3] = ins[which][nb - 1, L - 5, min(1, G - 1) if which in (3, 4) else 1, 5] = value
    x, dt, A, Bm, Cm, gy = ins
    outs = [dev(np.full(a.shape, 7, a.dtype)) for a in (x, x, dt, A, Bm, Cm)]
    y, gx, gdt, gA, gB, gC = outs
    scratch = scratch_for(mp, dims, True)
    args = [dev(a) for a in ins]
    torch.cuda.current_stream().synchronize()
    mp.launch("ssd_scan", torch.float16, *args[:5], y, scratch, *dims, stream)
    mp.launch("ssd_scan_reverse", torch.float16, *args, gx, gdt, gA, gB, gC, scratch, *dims, stream)
    stream.sync()
    assert stream.status() == 0
    f64 = [np.ascontiguousarray(a.astype(np.float64)) for a in ins]
    with np.errstate(all="ignore"):
        ref = (orc.ssd_forward(*f64[:5]),) + tuple(orc.ssd_reverse(*f64))
    # (tolerances of test_ssd_segments_keep_fp32)
    for got, want, name, tol in zip((y, gx, gdt, gA, gB, gC), ref, ("y", "gx", "gdt", "gA", "gB", "gC"), (2.9e-4, 2.9e-4, 2e-6, 2e-5, 2.9e-4, 2.9e-4)):
        got = host(got).astype(np.float64)
        finite = np.isfinite(want)
        assert np.array_equal(np.isfinite(got), finite), f"{name}: {np.sum(~np.isfinite(got))} not finite, {np.sum(~finite)} expected"
        d = got[finite] - want[finite]
        assert np.linalg.norm(d) <= tol * np.linalg.norm(want[finite]), name
