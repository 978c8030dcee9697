"""Performance cases of the framework: what a program built on it has it do, through the public entry points
(`metaphor_b200.launch`, `FusedChain`, `MambaLM`), over the range of sizes and storage types in use.

Seven kinds of work, each a pass that a training program repeats:

    block     one training step of the README's feed-forward block  y = selu(x A + b)
    rows      softmax and RMSNorm over the rows of a matrix, forward and reverse
    chain     the fused element-wise chain  e = selu((a + b) * (c + d))  and its reverse
    scan      the Mamba-2 SSD scan, forward and reverse
    contract  a projection y = x W and the two contractions of its reverse
    heads     attention over heads, composed of permutations, batched contractions and a row softmax
    lm        one training step of a Mamba-2 language model, batch upload included

`listed()` holds fixed cases (the benchmark configurations, the tests' small model, and odd or ragged sizes beside
them), `draw(rng)` one more case of the same ranges.  `prepare` makes what the program holds before the call, `run`
is one pass.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import torch

import metaphor_b200 as mp
from metaphor_b200.mamba_lm import LMConfig, MambaLM

DTYPES = {"r16": torch.float16, "r32": torch.float32}
SIZE = {"r16": 2, "r32": 4}
CHAIN = "selu((a+b)*(c+d))"
EPS = 1e-6


def listed():
    return [
        # The README's block at its own size: ten launches on half a megabyte, so launch latency and the host path count.
        dict(name="block_readme_r32", kind="block", dtype="r32", m=32, d_in=256, d_out=256),
        # The same step on an ordinary minibatch with widths that are not round (features of a tabular or spectral set).
        dict(name="block_odd_r16", kind="block", dtype="r16", m=1500, d_in=777, d_out=1030),
        # Row reductions at the benchmark size: memory-bound, half a gigabyte per tensor.
        dict(name="rows_65536x4096_r16", kind="rows", dtype="r16", m=65536, n=4096),
        # A minibatch of odd-length rows (class scores): the data stays in L2, rows are not 16-byte aligned.
        dict(name="rows_3000x1001_r32", kind="rows", dtype="r32", m=3000, n=1001),
        # The fused chain at the benchmark size: 1 GiB per tensor.
        dict(name="chain_2p28_r32", kind="chain", dtype="r32", n=1 << 28),
        # The scan at the benchmark size.
        dict(name="scan_8x8192x32", kind="scan", batch=8, seqlen=8192, heads=32, groups=1, chunk=256),
        # A document whose length is no multiple of the chunk.
        dict(name="scan_2x1000x24", kind="scan", batch=2, seqlen=1000, heads=24, groups=1, chunk=128),
        # The language model's input projection and its reverse.
        dict(name="contract_16384x768x3352_r16", kind="contract", dtype="r16", m=16384, n=768, k=3352),
        # A projection in r32 between odd widths.
        dict(name="contract_2000x999x1501_r32", kind="contract", dtype="r32", m=2000, n=999, k=1501),
        # Attention over heads [batch, length, heads, head size] on an ordinary sequence.
        dict(name="heads_4x512x12x64_r16", kind="heads", dtype="r16", batch=4, length=512, heads=12, dim=64),
        # The tests' small language model: some sixty launches of a few microseconds each.
        dict(name="lm_2x256_2layers", kind="lm", d_model=256, n_layer=2, vocab=1024, batch=2, seqlen=256, chunk=128),
        # The benchmark's training step (129 M parameters, 16384 tokens).
        dict(name="lm_8x2048_24layers", kind="lm", d_model=768, n_layer=24, vocab=50280, batch=8, seqlen=2048, chunk=256),
    ]


# --------------------------------------------------------------------------------------------------------------
# drawn cases
# --------------------------------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi, step):
    """A size spread over the logarithm of [lo, hi]: every other one a multiple of `step` (model widths), the rest as they fall."""
    v = _log(rng, lo, hi)
    return max(lo, min(hi, v // step * step)) if rng.random() < 0.5 else v


def draw(rng):
    kind = rng.choice(("block", "rows", "chain", "scan", "contract", "heads", "lm"))
    if kind == "block":
        return dict(kind=kind, dtype=rng.choice(("r16", "r32")), m=_size(rng, 4, 4096, 8), d_in=_size(rng, 32, 2048, 64), d_out=_size(rng, 32, 2048, 64))
    if kind == "rows":
        n = _size(rng, 64, 16384, 64)
        return dict(kind=kind, dtype=rng.choice(("r16", "r32")), m=_size(rng, 16, min(65536, (1 << 28) // n), 16), n=n)
    if kind == "chain":
        return dict(kind=kind, dtype=rng.choice(("r16", "r32")), n=_size(rng, 1 << 10, 1 << 28, 1024))
    if kind == "scan":
        batch, heads = _log(rng, 1, 8), 2 * _log(rng, 1, 16)
        return dict(kind=kind, batch=batch, seqlen=_size(rng, 64, 8192, 128), heads=heads, groups=rng.choice((1, 1, 2)), chunk=128)
    if kind == "contract":
        return dict(kind=kind, dtype=rng.choice(("r16", "r32")), m=_size(rng, 16, 16384, 128), n=_size(rng, 32, 4096, 64), k=_size(rng, 32, 4096, 64))
    if kind == "heads":
        return dict(kind=kind, dtype=rng.choice(("r16", "r32")), batch=_log(rng, 1, 8), length=_size(rng, 32, 1024, 64), heads=_log(rng, 1, 24),
                    dim=rng.choice((32, 64, 80, 128)))
    seqlen = 128 * _log(rng, 1, 16)
    return dict(kind=kind, d_model=128 * rng.randint(2, 6), n_layer=_log(rng, 1, 12), vocab=_size(rng, 512, 32000, 64), batch=_log(rng, 1, 8),
                seqlen=seqlen, chunk=256 if seqlen % 256 == 0 else 128)


# --------------------------------------------------------------------------------------------------------------
# what a program holds before the call
# --------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _stream():
    """The program's stream, opened once."""
    return mp.Stream()


class _Inputs:
    """Seeded random tensors on the device."""

    def __init__(self, seed, dtype):
        self.g, self.dtype = torch.Generator(device="cuda").manual_seed(seed), dtype

    def normal(self, *shape, scale=1.0, shift=0.0, dtype=None):
        return torch.randn(*shape, generator=self.g, device="cuda").mul_(scale).add_(shift).to(dtype or self.dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0, dtype=None):
        return torch.rand(*shape, generator=self.g, device="cuda").mul_(hi - lo).add_(lo).to(dtype or self.dtype)


def _prepare_block(c, r):
    m, di, do = c["m"], c["d_in"], c["d_out"]
    s = dict(x=r.normal(m, di), A=r.normal(di, do, scale=1 / math.sqrt(di)), b=torch.zeros(do, dtype=r.dtype, device="cuda"))
    s.update({k: torch.empty(m, do, dtype=r.dtype, device="cuda") for k in ("h", "y", "gh", "gy")})
    s.update(gx=torch.empty_like(s["x"]), gA=torch.empty_like(s["A"]), gb=torch.empty_like(s["b"]))
    return s


def _prepare_rows(c, r):
    m, n = c["m"], c["n"]
    s = dict(x=r.normal(m, n), gy=r.normal(m, n), gain=r.normal(n, scale=0.02, shift=1.0), rstd=torch.empty(m, dtype=torch.float32, device="cuda"))
    s.update({k: torch.empty_like(s["x"]) for k in ("soft", "gsoft", "norm", "gnorm")})
    s.update(ggain=torch.empty_like(s["gain"]),
             scratch=torch.empty(max(16, mp.lib().mpRmsnormReverseScratchBytes(m, n, _stream().ctx)), dtype=torch.uint8, device="cuda"))
    return s


@functools.lru_cache(maxsize=None)
def _chain(dtype):
    return mp.FusedChain(CHAIN, dtype)


def _prepare_chain(c, r):
    n = c["n"]
    leaves = [r.uniform(n, lo=-1.0, hi=1.0) for _ in range(4)]
    return dict(chain=_chain(r.dtype), leaves=leaves, out=torch.empty_like(leaves[0]), gout=r.normal(n), grads=[torch.empty_like(leaves[0]) for _ in range(4)])


def _scan_dims(c):
    return c["batch"], c["seqlen"], c["heads"], 64, 128, c["groups"], c["chunk"]


def _prepare_scan(c, r):
    nb, L, H, P, N, G, _ = dims = _scan_dims(c)
    f32 = torch.float32
    s = dict(dims=dims, x=r.normal(nb, L, H, P), B=r.normal(nb, L, G, N), C=r.normal(nb, L, G, N), gy=r.normal(nb, L, H, P),
             dt=torch.nn.functional.softplus(r.normal(nb, L, H, shift=-4.0, dtype=f32)), A=-torch.exp(r.uniform(H, hi=math.log(16.0), dtype=f32)))
    s.update(y=torch.empty_like(s["x"]), gx=torch.empty_like(s["x"]), gdt=torch.empty_like(s["dt"]), gA=torch.empty_like(s["A"]),
             gB=torch.empty_like(s["B"]), gC=torch.empty_like(s["C"]))
    nbytes = max(mp.lib().mpSsdScanScratchBytes(*dims, 0), mp.lib().mpSsdScanScratchBytes(*dims, 1))
    s["scratch"] = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    return s


def _prepare_contract(c, r):
    m, n, k = c["m"], c["n"], c["k"]
    s = dict(x=r.normal(m, n), W=r.normal(n, k, scale=1 / math.sqrt(n)), gy=r.normal(m, k))
    s.update(y=torch.empty_like(s["gy"]), gx=torch.empty_like(s["x"]), gW=torch.empty_like(s["W"]))
    return s


def _prepare_heads(c, r):
    b, l, h, d = c["batch"], c["length"], c["heads"], c["dim"]
    s = {k: r.normal(b, l, h, d) for k in ("q", "k", "v")}
    s.update({k + "h": torch.empty(b, h, l, d, dtype=r.dtype, device="cuda") for k in ("q", "k", "v", "o")})
    s.update(scores=torch.empty(b * h, l, l, dtype=r.dtype, device="cuda"), probs=torch.empty(b * h, l, l, dtype=r.dtype, device="cuda"),
             o=torch.empty_like(s["q"]))
    len4 = C.c_ulong * 4
    s.update(blhd=len4(b, l, h, d), bhld=len4(b, h, l, d), swap=len4(0, 2, 1, 3))
    return s


class _Model:
    """A model with its captured step; gives its streams and graphs back when the program drops it."""

    def __init__(self, model):
        self.model = model

    def __del__(self):
        self.model.release()


def _lm_config(c):
    return LMConfig(d_model=c["d_model"], n_layer=c["n_layer"], vocab=c["vocab"], chunk=c["chunk"])


def _lm_weights(cfg, r):
    """The initial weights of `mamba_lm.init_weights`, drawn on the device (a full-size model has 129 M of them)."""
    w = {}
    for name, shape in cfg.param_shapes():
        leaf = name.split(".")[-1]
        if leaf in ("norm_w", "gnorm_w", "normf_w", "D"):
            a = torch.ones(shape, device="cuda")
        elif leaf == "conv_b":
            a = torch.zeros(shape, device="cuda")
        elif leaf == "conv_w":
            a = r.uniform(*shape, lo=-1.0, hi=1.0) / math.sqrt(cfg.d_conv)
        elif leaf == "dt_bias":
            dt = torch.exp(r.uniform(*shape, lo=math.log(1e-3), hi=math.log(1e-1)))
            a = dt + torch.log(-torch.expm1(-dt))
        elif leaf == "A_log":
            a = torch.log(r.uniform(*shape, lo=1.0, hi=16.0))
        else:
            a = r.normal(*shape, scale=0.02)
        w[name] = a.cpu().numpy()
    return w


def _prepare_lm(c, seed):
    cfg, r = _lm_config(c), _Inputs(seed, torch.float32)
    tokens = c["batch"] * c["seqlen"]
    ids, targets = (torch.randint(0, cfg.vocab, (tokens,), generator=r.g, device="cuda", dtype=torch.int32).cpu().pin_memory() for _ in range(2))
    model = MambaLM(cfg, c["batch"], c["seqlen"], weights=_lm_weights(cfg, r))
    held = _Model(model)
    torch.cuda.synchronize()
    model.set_batch(ids, targets)
    model.capture()     # runs the first step and records the main-stream work of the following ones
    return dict(held=held, ids=ids, targets=targets)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "lm":
        s = _prepare_lm(case, seed)
    else:
        s = globals()["_prepare_" + kind](case, _Inputs(seed, DTYPES[case.get("dtype", "r16")]))
    s["case"] = case
    torch.cuda.synchronize()    # the inputs were made on torch's stream
    return s


# --------------------------------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------------------------------
def _run_block(s, c, st):
    """Forward, sum-loss reverse and an SGD step, in the launches that the host layer issues for the block."""
    m, di, do, dt = c["m"], c["d_in"], c["d_out"], DTYPES[c["dtype"]]
    x, A, b, h, y, gh, gy, gx, gA, gb = (s[k] for k in ("x", "A", "b", "h", "y", "gh", "gy", "gx", "gA", "gb"))
    mp.launch("linear_ij_jk_ik", dt, x, A, b, 1.0, h, 0.0, m, di, do, st)
    mp.launch("selu", dt, h, y, m * do, st)
    mp.launch("fill", dt, gy, 1.0, m * do, st)
    mp.launch("fill", dt, gh, 0.0, m * do, st)
    mp.launch("selu_reverse", dt, h, gh, gy, m * do, st)
    mp.launch("inner_product_ij_kj_ik", dt, gh, A, 1.0, gx, 0.0, m, do, di, st)
    mp.launch("inner_product_ji_jk_ik", dt, x, gh, 1.0, gA, 0.0, di, m, do, st)
    mp.launch("reduce_ij_j", dt, gh, gb, 0.0, m, do, st)
    rate = 0.32 / m
    mp.launch("sgd", dt, A, gA, rate, -math.inf, math.inf, di * do, st)
    mp.launch("sgd", dt, b, gb, rate, -math.inf, math.inf, do, st)
    return dict(y=y, gx=gx, gA=gA, gb=gb, A=A, b=b)


def _run_rows(s, c, st):
    m, n, dt = c["m"], c["n"], DTYPES[c["dtype"]]
    mp.launch("softmax_ij_j", dt, s["x"], s["soft"], m, n, st)
    mp.launch("softmax_ij_j_reverse", dt, s["soft"], s["gy"], s["gsoft"], 0.0, m, n, st)
    mp.launch("rmsnorm_ij_j", dt, s["x"], s["gain"], EPS, s["norm"], s["rstd"], m, n, st)
    mp.launch("rmsnorm_ij_j_reverse", dt, s["x"], s["gain"], s["rstd"], s["gy"], EPS, s["gnorm"], s["ggain"], 0.0, s["scratch"], m, n, st)
    return {k: s[k] for k in ("soft", "gsoft", "norm", "rstd", "gnorm", "ggain")}


def _run_chain(s, c, st):
    s["chain"].forward(s["leaves"], s["out"], c["n"], st)
    s["chain"].reverse(s["leaves"], s["gout"], s["grads"], 0.0, c["n"], st)
    return dict(out=s["out"], grads=s["grads"])


def _run_scan(s, c, st):
    ins = [s[k] for k in ("x", "dt", "A", "B", "C")]
    mp.launch("ssd_scan", torch.float16, *ins, s["y"], s["scratch"], *s["dims"], st)
    mp.launch("ssd_scan_reverse", torch.float16, *ins, s["gy"], s["gx"], s["gdt"], s["gA"], s["gB"], s["gC"], s["scratch"], *s["dims"], st)
    return {k: s[k] for k in ("y", "gx", "gdt", "gA", "gB", "gC")}


def _run_contract(s, c, st):
    m, n, k, dt = c["m"], c["n"], c["k"], DTYPES[c["dtype"]]
    mp.launch("inner_product_ij_jk_ik", dt, s["x"], s["W"], 1.0, s["y"], 0.0, m, n, k, st)
    mp.launch("inner_product_ij_kj_ik", dt, s["gy"], s["W"], 1.0, s["gx"], 0.0, m, k, n, st)
    mp.launch("inner_product_ji_jk_ik", dt, s["x"], s["gy"], 1.0, s["gW"], 0.0, n, m, k, st)
    return dict(y=s["y"], gx=s["gx"], gW=s["gW"])


def _run_heads(s, c, st):
    l, d, bh, dt = c["length"], c["dim"], c["batch"] * c["heads"], DTYPES[c["dtype"]]
    for k in ("q", "k", "v"):
        mp.launch("permutate", dt, s[k], s[k + "h"], 0.0, s["blhd"], s["swap"], 4, st)
    mp.launch("inner_product_bij_bkj_bik", dt, s["qh"], s["kh"], 1.0 / math.sqrt(d), s["scores"], 0.0, bh, l, d, l, st)
    mp.launch("softmax_ij_j", dt, s["scores"], s["probs"], bh * l, l, st)
    mp.launch("inner_product_bij_bjk_bik", dt, s["probs"], s["vh"], 1.0, s["oh"], 0.0, bh, l, l, d, st)
    mp.launch("permutate", dt, s["oh"], s["o"], 0.0, s["bhld"], s["swap"], 4, st)
    return dict(probs=s["probs"], o=s["o"])


def _run_lm(s, c, st):
    model = s["held"].model
    model.set_batch(s["ids"], s["targets"])
    model.train_step()
    return dict(loss=model.loss_sum, loss_rows=model.loss_rows, w32=model.w32, w16=model.w16, m=model.m, v=model.v)


def run(state):
    case = state["case"]
    return globals()["_run_" + case["kind"]](state, case, _stream())


# --------------------------------------------------------------------------------------------------------------
# the work that a pass cannot do without, and how exact its results are
# --------------------------------------------------------------------------------------------------------------
def _scan_work(nb, L, H, P, N, G, Q):
    """Bytes and flops of the chunked scan, forward and reverse (scores counted once per group)."""
    chunks = nb * L / Q
    fwd = 2 * Q * Q * N * chunks * G + (2 * Q * Q * P + 4 * Q * N * P) * chunks * H
    rev = (4 * Q * Q * P + 8 * Q * N * P) * chunks * H + 4 * Q * Q * N * chunks * G
    x, bc, dt = nb * L * H * P * 2, nb * L * G * N * 2, nb * L * H * 4
    return (2 * x + 2 * bc + dt) + (2 * x + 2 * bc + dt) + (x + 2 * bc + dt), fwd + rev


def work(case):
    c, kind = case, case["kind"]
    e = SIZE[c.get("dtype", "r16")]
    if kind == "block":
        m, di, do = c["m"], c["d_in"], c["d_out"]
        # x, A, b in; y, gx, gA, gb, A, b out (what lies between can stay on chip)
        return dict(bytes=e * (2 * m * di + 3 * di * do + m * do + 3 * do), flops=6 * m * di * do)
    if kind == "rows":
        m, n = c["m"], c["n"]
        return dict(bytes=e * (6 * m * n + 2 * n) + 4 * m, flops=20 * m * n)     # x, gy in; four results out
    if kind == "chain":
        return dict(bytes=10 * e * c["n"], flops=16 * c["n"])
    if kind == "scan":
        nbytes, flops = _scan_work(*_scan_dims(c))
        return dict(bytes=nbytes, flops=flops)
    if kind == "contract":
        m, n, k = c["m"], c["n"], c["k"]
        return dict(bytes=2 * e * (m * n + n * k + m * k), flops=6 * m * n * k)
    if kind == "heads":
        l, d, bh = c["length"], c["dim"], c["batch"] * c["heads"]
        return dict(bytes=e * bh * (4 * l * d + l * l), flops=4 * bh * l * l * d)
    cfg, T = _lm_config(c), c["batch"] * c["seqlen"]
    matmul = cfg.n_layer * (cfg.d_model * cfg.d_in_proj + cfg.d_inner * cfg.d_model) + cfg.vocab * cfg.d_model
    scan_bytes, scan_flops = _scan_work(c["batch"], c["seqlen"], cfg.heads, cfg.headdim, cfg.d_state, cfg.ngroups, cfg.chunk)
    # weights and both moments read and written, the r16 copy written; per layer and token the block's input, projection and
    # output once each way
    nbytes = cfg.n_params() * (6 * 4 + 2) + cfg.n_layer * (T * 2 * 3 * (2 * cfg.d_model + cfg.d_in_proj)) + 2 * T * cfg.vocab
    return dict(bytes=nbytes, flops=6 * matmul * T + cfg.n_layer * scan_flops)


def tolerance(case):
    kind = case["kind"]
    if kind in ("scan", "lm"):      # r16 activations through several rounded stages; the scan's dt and A gradients cancel
        return {"rel": 1e-2}
    if case["dtype"] == "r16":      # rounding of each stored value (2^-11), compounded over the stages of a pass
        return {"rel": 3e-3}
    return {"rel": 2e-5}            # r32 sums
