"""GPU parity of the einsum contractions (inner_product NN / NT / TN, linear)
against the fp64-accumulating CPU oracle, through the C ABI."""
import numpy as np
import pytest

from util import TOL_RED, assert_close, dev, host, narrow, rng_normal, run, wide

pytestmark = pytest.mark.gpu

# (m, n, k) in the reference's naming: C[m,k] = A[m,n] * B[n,k]
SHAPES = [(3, 2, 2), (32, 256, 256), (128, 64, 128), (129, 72, 200), (256, 384, 512), (100, 1000, 24), (1, 8, 8),
          (300, 40, 264), (64, 2048, 64), (5, 7, 3)]
DTYPES = ["r16", "r32", "r64"]
VARIANTS = [("inner_product_ij_jk_ik", False, False), ("inner_product_ij_kj_ik", False, True),
            ("inner_product_ji_jk_ik", True, False)]


def operands(sfx, m, n, k, ta, tb, seed=0):
    a = rng_normal(seed, (n, m) if ta else (m, n), sfx, scale=1.0)
    b = rng_normal(seed + 1, (k, n) if tb else (n, k), sfx, scale=1.0 / np.sqrt(n))
    return a, b


@pytest.mark.parametrize("sfx", DTYPES)
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("variant", VARIANTS, ids=[v[0][-8:] for v in VARIANTS])
def test_inner_product_variants(mp, stream, orc, sfx, shape, variant):
    name, ta, tb = variant
    m, n, k = shape
    a, b = operands(sfx, m, n, k, ta, tb)
    c = dev(np.full((m, k), np.nan, a.dtype))           # fresh output: beta = 0 must not read it
    run(mp, stream, name, sfx, dev(a), dev(b), 1.0, c, 0.0, m, n, k)
    ref = orc.inner_product(wide(a), wide(b), ta=ta, tb=tb)
    assert_close(host(c), narrow(ref, sfx), TOL_RED[sfx], f"{name} {sfx} {shape}")
    # accumulate form used by the reverse pass: alpha = scale, beta = 1 (inner_product.zig:275-301)
    c0 = rng_normal(7, (m, k), sfx)
    c = dev(c0)
    run(mp, stream, name, sfx, dev(a), dev(b), 0.5, c, 1.0, m, n, k)
    ref = orc.inner_product(wide(a), wide(b), 0.5, wide(c0).copy(), 1.0, ta=ta, tb=tb)
    assert_close(host(c), narrow(ref, sfx), TOL_RED[sfx], f"{name} accumulate {sfx} {shape}")
    assert stream.status() == 0


@pytest.mark.parametrize("sfx", DTYPES)
@pytest.mark.parametrize("shape", [(32, 256, 256), (129, 72, 200), (5, 7, 3)])
def test_linear_adds_bias_in_the_epilogue(mp, stream, orc, sfx, shape):
    m, n, k = shape
    a, b = operands(sfx, m, n, k, False, False, seed=3)
    bias = rng_normal(9, k, sfx)
    c = dev(np.full((m, k), np.nan, a.dtype))
    run(mp, stream, "linear_ij_jk_ik", sfx, dev(a), dev(b), dev(bias), 1.0, c, 0.0, m, n, k)
    ref = orc.inner_product(wide(a), wide(b), bias=wide(bias))
    assert_close(host(c), narrow(ref, sfx), TOL_RED[sfx], f"linear {sfx} {shape}")


# The residual form "ij,jk,ik->ik": a full [m, k] term added in the epilogue.  Shapes reach the FP-pipe kernel, the
# single-CTA tensor kernel, the CTA-pair kernel (>= 74 tiles of 256 x 256, ragged last column tile) and the split-K fold.
@pytest.mark.parametrize("sfx", DTYPES)
@pytest.mark.parametrize("shape", [(5, 7, 3), (129, 72, 200), (300, 40, 264), (2560, 64, 1992), (256, 4096, 512)])
def test_linear_with_a_full_matrix_term(mp, stream, orc, sfx, shape):
    m, n, k = shape
    a, b = operands(sfx, m, n, k, False, False, seed=5)
    r = rng_normal(11, (m, k), sfx)
    c = dev(np.full((m, k), np.nan, a.dtype))
    run(mp, stream, "linear_ij_jk_ik_ik", sfx, dev(a), dev(b), dev(r), 0.5, c, 0.0, m, n, k)
    ref = orc.inner_product(wide(a), wide(b), 0.5) + wide(r)
    assert_close(host(c), narrow(ref, sfx), TOL_RED[sfx], f"linear + matrix {sfx} {shape}")
    # in place on the residual stream: r is also the output
    rc = dev(r.copy())
    run(mp, stream, "linear_ij_jk_ik_ik", sfx, dev(a), dev(b), rc, 0.5, rc, 0.0, m, n, k)
    assert_close(host(rc), narrow(ref, sfx), TOL_RED[sfx], f"linear + matrix in place {sfx} {shape}")
    assert stream.status() == 0


BATCHED = [("inner_product_bij_bjk_bik", False, False), ("inner_product_bij_bkj_bik", False, True),
           ("inner_product_bji_bjk_bik", True, False)]
# (batch, m, n, k): tiles cut at the edges of every batch entry, one entry, odd pitches (FP-pipe kernel), deep n
BATCHED_SHAPES = [(3, 129, 72, 200), (1, 64, 64, 64), (5, 7, 3, 5), (16, 128, 64, 128), (4, 100, 1000, 24), (2, 300, 40, 264),
                  (6, 33, 8, 8)]


@pytest.mark.parametrize("sfx", DTYPES)
@pytest.mark.parametrize("shape", BATCHED_SHAPES)
@pytest.mark.parametrize("variant", BATCHED, ids=[v[0][-11:] for v in BATCHED])
def test_batched_inner_product_variants(mp, stream, orc, sfx, shape, variant):
    name, ta, tb = variant
    nb, m, n, k = shape
    a = rng_normal(20, (nb, n, m) if ta else (nb, m, n), sfx)
    b = rng_normal(21, (nb, k, n) if tb else (nb, n, k), sfx, scale=1.0 / np.sqrt(n))
    c = dev(np.full((nb, m, k), np.nan, a.dtype))        # beta = 0 must not read the fresh output
    run(mp, stream, name, sfx, dev(a), dev(b), 1.0, c, 0.0, nb, m, n, k)
    ref = orc.inner_product_batched(wide(a), wide(b), ta=ta, tb=tb)
    assert_close(host(c), narrow(ref, sfx), TOL_RED[sfx], f"{name} {sfx} {shape}")
    c0 = rng_normal(22, (nb, m, k), sfx)
    c = dev(c0)
    run(mp, stream, name, sfx, dev(a), dev(b), 0.5, c, 1.0, nb, m, n, k)
    ref = orc.inner_product_batched(wide(a), wide(b), 0.5, wide(c0).copy(), 1.0, ta=ta, tb=tb)
    assert_close(host(c), narrow(ref, sfx), TOL_RED[sfx], f"{name} accumulate {sfx} {shape}")
    assert stream.status() == 0


@pytest.mark.parametrize("sfx", ["r16", "r32"])
def test_batched_entries_equal_the_rank2_contraction(mp, stream, sfx):
    # every batch entry is bit-identical to the rank-2 launcher run on that entry alone (same kernel, same tile walk),
    # at a size the oracle does not reach
    import torch
    nb, m, n, k = 12, 512, 256, 384
    dt = {"r16": torch.float16, "r32": torch.float32}[sfx]
    a = torch.randn(nb, m, n, device="cuda").to(dt); b = (torch.randn(nb, n, k, device="cuda") / 16).to(dt)
    c = torch.empty(nb, m, k, device="cuda", dtype=dt); c1 = torch.empty(m, k, device="cuda", dtype=dt)
    run(mp, stream, "inner_product_bij_bjk_bik", sfx, a, b, 1.0, c, 0.0, nb, m, n, k)
    for q in (0, 5, 11):
        run(mp, stream, "inner_product_ij_jk_ik", sfx, a[q], b[q], 1.0, c1, 0.0, m, n, k)
        assert torch.equal(c[q], c1)


def test_experimental_example_through_the_abi(mp, stream):
    # src/examples/experimental.zig: x = sequence(1,1)[3,2], y = sequence(1,1)[2,2]; z = x.y; reverse with seed 1
    import torch
    x = torch.empty(3, 2, device="cuda"); y = torch.empty(2, 2, device="cuda")
    run(mp, stream, "sequence", "r32", x, 1.0, 1.0, 6)
    run(mp, stream, "sequence", "r32", y, 1.0, 1.0, 4)
    z = torch.empty(3, 2, device="cuda")
    run(mp, stream, "inner_product_ij_jk_ik", "r32", x, y, 1.0, z, 0.0, 3, 2, 2)
    assert z.cpu().tolist() == [[7, 10], [15, 22], [23, 34]]
    gz = torch.empty_like(z); gx = torch.zeros_like(x); gy = torch.zeros_like(y)
    run(mp, stream, "fill", "r32", gz, 1.0, 6)
    run(mp, stream, "inner_product_ij_kj_ik", "r32", gz, y, 1.0, gx, 1.0, 3, 2, 2)   # dx = G . y^T
    run(mp, stream, "inner_product_ji_jk_ik", "r32", x, gz, 1.0, gy, 1.0, 2, 3, 2)   # dy = x^T . G
    assert gx.cpu().tolist() == [[3, 7], [3, 7], [3, 7]]
    assert gy.cpu().tolist() == [[9, 9], [12, 12]]


@pytest.mark.parametrize("sfx", ["r16", "r32"])
def test_large_shape_against_float64_matmul(mp, stream, sfx):
    """A projection-sized contraction (4096 x 768 x 3352): checked against a
    float64 matmul on the GPU instead of the scalar oracle."""
    import torch
    from util import torch_dtype
    m, n, k = 4096, 768, 3352
    g = torch.Generator(device="cuda").manual_seed(0)
    dt = torch_dtype(sfx)
    a = torch.randn(m, n, generator=g, device="cuda").to(dt)
    b = (torch.randn(n, k, generator=g, device="cuda") / n ** 0.5).to(dt)
    c = torch.empty(m, k, device="cuda", dtype=dt)
    run(mp, stream, "inner_product_ij_jk_ik", sfx, a, b, 1.0, c, 0.0, m, n, k)
    ref = a.double() @ b.double()
    err = float((c.double() - ref).abs().max() / ref.abs().max())
    assert err <= TOL_RED[sfx], err
    assert stream.status() == 0


# Operands whose rows are not 16-byte aligned are copied into aligned rows and multiplied on the tensor cores.  (batch, m, n, k):
# one ragged tile, ragged tiles of the single-CTA kernel, enough 256 x 256 tiles for the CTA-pair kernel, a split of a long odd n
# (partial rows padded to four columns), odd batch entries, and copies beyond the workspace (worked off in slabs of rows, of
# columns, of batch entries).
ODD_SHAPES = [(1, 101, 103, 107), (1, 257, 65, 515), (1, 2571, 77, 1993), (1, 255, 4099, 130), (1, 130, 4098, 131), (7, 101, 99, 63),
              (1, 16411, 1101, 67), (1, 67, 1101, 16411), (90, 513, 301, 515),
              # a single result, rows and columns of one, both sides of the lines to the tensor cores (K of 16, 64 and 96, volume of 6e7)
              (1, 1, 97, 1), (1, 2, 131, 1), (5, 3, 99, 2), (1, 1, 4099, 1), (1, 33, 63, 35), (1, 33, 65, 35), (1, 2001, 15, 2003), (1, 2001, 17, 2003),
              (1, 1001, 95, 33),
              # more rows than the FP-pipe kernel's grid holds
              (1, 4194401, 9, 3)]


@pytest.mark.parametrize("sfx", ["r16", "r32"])
@pytest.mark.parametrize("shape", ODD_SHAPES)
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ij_kj_ik", "ji_jk_ik"])
def test_unaligned_operands(mp, stream, sfx, shape, variant):
    import torch
    from util import torch_dtype
    nb, m, n, k = shape
    dt = torch_dtype(sfx)
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    ta, tb = variant[0] == "j", variant[3:5] == "kj"
    # bases one element off a 16-byte boundary in two of three variants
    def operand(rows, cols, scale, off):
        flat = (torch.randn(nb * rows * cols + off, generator=g, device="cuda") * scale).to(dt)
        return flat[off:].view(nb, rows, cols)
    a = operand(*((n, m) if ta else (m, n)), 1.0, int(ta))
    b = operand(*((k, n) if tb else (n, k)), n ** -0.5, int(tb))
    c0 = operand(m, k, 1.0, 1)
    c = torch.full_like(c0, float("nan"))
    name = "inner_product_" + ("_".join("b" + p for p in variant.split("_")) if nb > 1 else variant)
    dims = (nb, m, n, k) if nb > 1 else (m, n, k)
    ref = (a.double().transpose(1, 2) if ta else a.double()) @ (b.double().transpose(1, 2) if tb else b.double())
    run(mp, stream, name, sfx, a, b, 1.0, c, 0.0, *dims)
    assert float((c.double() - ref).abs().max() / ref.abs().max()) <= TOL_RED[sfx]
    c1 = operand(m, k, 0.0, 1)
    c1.copy_(c0)
    run(mp, stream, name, sfx, a, b, 0.5, c1, 1.0, *dims)
    ref = 0.5 * ref + c0.double()
    assert float((c1.double() - ref).abs().max() / ref.abs().max()) <= TOL_RED[sfx]
    if nb == 1 and variant == "ij_jk_ik":      # the bias and the matrix term through the same stores
        bias = operand(1, k, 1.0, 1)
        run(mp, stream, "linear_ij_jk_ik", sfx, a, b, bias, 1.0, c, 0.0, *dims)
        ref = a.double()[0] @ b.double()[0]
        assert float((c.double()[0] - ref - bias.double()[0]).abs().max() / ref.abs().max()) <= TOL_RED[sfx]
        run(mp, stream, "linear_ij_jk_ik_ik", sfx, a, b, c0, 1.0, c, 0.0, *dims)
        assert float((c.double()[0] - ref - c0.double()[0]).abs().max() / ref.abs().max()) <= TOL_RED[sfx]
    assert stream.status() == 0


# Contractions of unaligned r32 operands are as exact as sums of K fused multiply-adds.  The bound is that of such a sum of random
# signs, 2^-24 sqrt(K / 2) of the result's norm at most (its roundings are half an ulp at most, and grow with the partial sums), but at
# least 2.2e-7: two roundings of the operands' splits and the four truncated additions of a k-block.  K: below and at the line to the
# tensor cores, one k-block and one value more, chunks of one block with a remainder, a split of K.
@pytest.mark.parametrize("shape", [(301, 33, 307), (301, 95, 307), (301, 97, 307), (301, 129, 307), (2001, 999, 1501), (131, 4097, 127), (129, 16385, 67)])
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ij_kj_ik", "ji_jk_ik"])
@pytest.mark.parametrize("positive", [False, True])
def test_unaligned_r32_keeps_fp32_sums(mp, stream, shape, variant, positive):
    import torch
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    a = torch.randn(*((n, m) if variant[0] == "j" else (m, n)), generator=g, device="cuda")
    b = torch.randn(*((k, n) if variant[3:5] == "kj" else (n, k)), generator=g, device="cuda")
    if positive:
        a, b = a.abs(), b.abs()
    c = torch.empty(m, k, device="cuda")
    run(mp, stream, "inner_product_" + variant, "r32", a, b, 1.0, c, 0.0, m, n, k)
    ref = (a.double().t() if variant[0] == "j" else a.double()) @ (b.double().t() if variant[3:5] == "kj" else b.double())
    err = float((c.double() - ref).norm() / ref.norm())
    assert err <= max(2.2e-7, 2.0 ** -24 * (n / 2) ** 0.5), err
    assert stream.status() == 0


# Infinite and overflowing r32 operands off the 16-byte boundary: one infinity in each operand (meeting zeros, values that the split's high
# part holds whole, and each other), a NaN, the largest float (which rounds up to infinity in 11 bits) and results beyond it.
# One k-block, several, a split of K, a batch; bias, matrix term and the old C on top.
@pytest.mark.parametrize("shape", [(1, 131, 97, 133), (1, 301, 999, 307), (1, 67, 16385, 67), (3, 131, 101, 99)])
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ij_kj_ik", "ji_jk_ik"])
def test_unaligned_r32_not_finite(mp, stream, shape, variant):
    import torch
    nb, m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    a, b = torch.randn(nb, m, n, generator=g, device="cuda"), torch.randn(nb, n, k, generator=g, device="cuda")
    inf, big = float("inf"), torch.finfo(torch.float32).max
    a[0, 3, 5], b[0, 5, 7], b[0, 5, 9], b[0, 5, 10] = inf, 0.0, 1.0, -0.5
    b[-1, n - 1, 20] = -inf
    a[-1, 40, n - 1], a[-1, 41, n - 1] = 0.0, 2.0
    a[0, 66, 11] = float("nan")
    a[0, 50], a[0, 50, 2], b[0, 2, 30], b[0, 2, 31] = 0.0, big, 0.5, 4.0
    ta, tb = variant[0] == "j", variant[3:5] == "kj"
    da, db = (a.transpose(1, 2) if ta else a).contiguous(), (b.transpose(1, 2) if tb else b).contiguous()
    name = "inner_product_" + ("_".join("b" + p for p in variant.split("_")) if nb > 1 else variant)
    dims = (nb, m, n, k) if nb > 1 else (m, n, k)
    # products and sums in r64, and what of it is beyond r32; no sum here comes near the limit without being far beyond it
    ref = (a.double() @ b.double()).float()
    scale = torch.where(torch.isfinite(ref), ref, torch.zeros_like(ref))
    scale[0, 50] = 0

    def check(c, want, what):
        assert torch.equal(torch.isnan(c), torch.isnan(want)), what
        sel = torch.isinf(want) | torch.isinf(c)
        assert torch.equal(c[sel], want[sel]), what
        fin = torch.isfinite(want)
        assert float((c - want)[fin].abs().max() / want[fin].abs().max()) <= 1e-5, what
        fin[0, 50] = False      # (the row with the largest float: the others are small against it)
        assert float((c - want)[fin].abs().max() / scale.abs().max()) <= 1e-5, what

    c = torch.full((nb, m, k), 3.0, device="cuda")
    run(mp, stream, name, "r32", da, db, 1.0, c, 0.0, *dims)
    check(c, ref, "plain")
    c = torch.full((nb, m, k), 3.0, device="cuda")
    run(mp, stream, name, "r32", da, db, 0.5, c, 1.0, *dims)
    check(c, 0.5 * ref + 3.0, "beta")
    if nb == 1 and variant == "ij_jk_ik":
        bias, mat = torch.randn(k, device="cuda"), torch.randn(m, k, device="cuda")
        run(mp, stream, "linear_ij_jk_ik", "r32", da, db, bias, 1.0, c, 0.0, *dims)
        check(c, ref + bias, "bias")
        run(mp, stream, "linear_ij_jk_ik_ik", "r32", da, db, mat, 1.0, c, 0.0, *dims)
        check(c, ref + mat, "matrix")
    assert stream.status() == 0


# r16 operands off the 16-byte boundary, of one sign, so that truncated additions do not cancel: enough 256 x 256 tiles for CTA pairs, a
# long K in few tiles, and one tile.  A sum that is off by at most 8 x 2^-24 of itself (the additions of one hand-over) comes to lie beyond
# the middle between two r16 values, which are 2^-11 to 2^-10 apart, in at most 8 x 2^-13 = 1e-3 of all cases; the fp32 additions of the
# hand-overs may add as much.
@pytest.mark.parametrize("shape", [(2571, 2049, 1993), (301, 4097, 307), (101, 513, 99)])
def test_unaligned_r16_keeps_fp32_sums(mp, stream, shape):
    import torch
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    a, b = (torch.randn(*s, generator=g, device="cuda").abs().half() for s in ((m, n), (n, k)))
    c = torch.empty(m, k, device="cuda", dtype=torch.float16)
    run(mp, stream, "inner_product_ij_jk_ik", "r16", a, b, 2.0 ** -6, c, 0.0, m, n, k)
    ref = (a.double() @ b.double()) * 2.0 ** -6
    assert float((c != ref.half()).double().mean()) <= 2e-3
    assert stream.status() == 0


# r32 contractions from three bf16 terms per value, at the edges of tiles (256 rows, 128 or 256 columns), k-blocks (64) and 16-byte pitches, and with a
# split of K.  Rows and columns are of sizes between 2^-40 and 2^40: values have exponents of their own, so every result is as exact as its own
# products: each is off by three roundings of 2^-23 at most, the sum by the truncated additions of 12 MMAs and a rounding per k-block.
@pytest.mark.parametrize("shape", [(1, 64, 1), (255, 63, 129), (256, 64, 256), (257, 65, 257), (300, 129, 520), (513, 777, 127), (66, 4097, 300)])
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ij_kj_ik", "ji_jk_ik"])
def test_r32_from_terms(mp, stream, monkeypatch, shape, variant):
    import torch
    monkeypatch.setenv("MP_GEMM_R32_TERMS", "1")      # read at every launch
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    power = lambda c: torch.exp2(torch.randint(-40, 41, (c,), generator=g, device="cuda").float())
    a = torch.randn(m, n, generator=g, device="cuda") * power(m)[:, None]
    b = torch.randn(n, k, generator=g, device="cuda") * power(k)[None, :]
    da = (a.t() if variant[0] == "j" else a).contiguous()
    db = (b.t() if variant[3:5] == "kj" else b).contiguous()
    ref, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    bound = (3 * 2.0 ** -23 + 13 * 2.0 ** -23) * size
    c = torch.full((m + 1, k), 7.0, device="cuda")
    run(mp, stream, "inner_product_" + variant, "r32", da, db, 1.0, c, 0.0, m, n, k)
    assert bool(((c[:m].double() - ref).abs() <= bound).all())
    assert bool((c[m] == 7).all())
    old = torch.randn(m, k, generator=g, device="cuda") * power(k)[None, :]
    c = old.clone()
    run(mp, stream, "inner_product_" + variant, "r32", da, db, 0.5, c, 2.0, m, n, k)
    assert bool(((c.double() - 0.5 * ref - 2 * old.double()).abs() <= bound + 2.0 ** -22 * old.double().abs()).all())
    if variant == "ij_jk_ik":
        bias = torch.randn(k, generator=g, device="cuda")
        run(mp, stream, "linear_ij_jk_ik", "r32", da, db, bias, 1.0, c, 0.0, m, n, k)
        assert bool(((c.double() - ref - bias.double()).abs() <= bound + 2.0 ** -22 * bias.double().abs()).all())
    assert stream.status() == 0


@pytest.mark.parametrize("shape", [(1, 131, 97, 133), (1, 301, 999, 307), (1, 67, 16385, 67)])
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ij_kj_ik", "ji_jk_ik"])
def test_r32_from_terms_not_finite(mp, stream, monkeypatch, shape, variant):
    monkeypatch.setenv("MP_GEMM_R32_TERMS", "1")
    test_unaligned_r32_not_finite(mp, stream, shape, variant)


# Values of one row that lie far apart along K, the large ones against zeros of the other operand: the small ones alone make the result and keep
# their bits (the bound is that of test_r32_from_terms).  One large value in each 64 of K, at another place in each; in A, then in B.
@pytest.mark.parametrize("shape", [(300, 129, 520), (256, 128, 256)])
@pytest.mark.parametrize("spread", [0, 10, 17, 24, 31, 45, 90])
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ij_kj_ik", "ji_jk_ik"])
def test_r32_terms_of_values_far_apart(mp, stream, monkeypatch, shape, spread, variant):
    import torch
    monkeypatch.setenv("MP_GEMM_R32_TERMS", "1")      # read at every launch
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    small, other = 0.1 + 0.9 * torch.rand(max(m, k), n, generator=g, device="cuda"), torch.randn(max(m, k), n, generator=g, device="cuda")
    at = torch.tensor([(i * 64 + (i * 23 + 5) % 64) % n for i in range((n + 63) // 64)], device="cuda")
    small[:, at], other[:, at] = 2.0 ** spread, 0.0
    for a, b in ((small[:m], other[:k].t()), (other[:m], small[:k].t())):
        da = (a.t() if variant[0] == "j" else a).contiguous()
        db = (b.t() if variant[3:5] == "kj" else b).contiguous()
        ref, size = a.double() @ b.double(), a.double().abs() @ b.double().abs()
        c = torch.full((m, k), 7.0, device="cuda")
        run(mp, stream, "inner_product_" + variant, "r32", da, db, 1.0, c, 0.0, m, n, k)
        assert bool(((c.double() - ref).abs() <= 16 * 2.0 ** -23 * size).all())
    assert stream.status() == 0


# The default rule: from 1e9 products on where the copies fit the workspace.  Which kernel ran shows in the bits, for the two differ in theirs.
@pytest.mark.parametrize("shape,terms", [((2048, 2048, 2048), True), ((2000, 999, 1501), True), ((1000, 1000, 999), False), ((4096, 1400, 4096), False)])
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ij_kj_ik", "ji_jk_ik"])
def test_r32_terms_by_default(mp, stream, monkeypatch, shape, terms, variant):
    import torch
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    a, b = torch.randn(m, n, generator=g, device="cuda"), torch.randn(n, k, generator=g, device="cuda")
    a[:, 7::64], b[7::64] = 2.0 ** 40, 0.0
    da = (a.t() if variant[0] == "j" else a).contiguous()
    db = (b.t() if variant[3:5] == "kj" else b).contiguous()

    def result(x, y):
        c = torch.full((m, k), 7.0, device="cuda")
        run(mp, stream, "inner_product_" + variant, "r32", x, y, 1.0, c, 0.0, m, n, k)
        return c

    c = result(da, db)
    bound = lambda x, y: 16 * 2.0 ** -23 * (x.double().abs() @ y.double().abs())
    assert bool(((c.double() - a.double() @ b.double()).abs() <= bound(a, b)).all()) or not terms
    # results near the smallest normal number, from products of the same size; and 1e24 where only a zero meets it
    tiny = result(torch.full_like(da, 2.0 ** -62), torch.full_like(db, 2.0 ** -61))
    assert bool(((tiny.double() - n * 2.0 ** -123).abs() <= 16 * 2.0 ** -23 * n * 2.0 ** -123).all())
    a, b = torch.zeros(m, n, device="cuda"), torch.zeros(n, k, device="cuda")
    a[:, 0], b[1], a[:, 2], b[2] = 1e24, 1e24, 3.0, 5.0
    huge = result((a.t() if variant[0] == "j" else a).contiguous(), (b.t() if variant[3:5] == "kj" else b).contiguous())
    assert bool((huge == 15.0).all())
    monkeypatch.setenv("MP_GEMM_R32_TERMS", "0")      # read at every launch
    assert torch.equal(c, result(da, db)) == (not terms)
    assert stream.status() == 0


# r16 results in a C with rows off the 16-byte boundary: written as words of two elements, whole rows and their odd ends.
@pytest.mark.parametrize("shape", [(33, 64, 1), (130, 64, 31), (129, 72, 33), (128, 64, 63), (300, 200, 65), (257, 64, 129), (40, 64, 258), (600, 128, 777)])
@pytest.mark.parametrize("off", [0, 1])
def test_r16_results_off_the_boundary(mp, stream, shape, off):
    import torch
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    a, b = torch.randn(m, n, generator=g, device="cuda").half(), torch.randn(n, k, generator=g, device="cuda").half()
    flat = torch.full((m * k + 16,), 7.0, device="cuda", dtype=torch.float16)
    c = flat[off:off + m * k].view(m, k)
    run(mp, stream, "inner_product_ij_jk_ik", "r16", a, b, 1.0, c, 0.0, m, n, k)
    ref = a.double() @ b.double()
    assert float((c.double() - ref).norm() / ref.norm()) <= 2.9e-4      # the rounding of an r16 result
    assert bool((flat[:off] == 7).all()) and bool((flat[off + m * k:] == 7).all())
    assert stream.status() == 0


def kernels(call):
    """The kernels a call launches, by name."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if "gemm" in e.name]
    assert names, "no kernel was recorded"
    return names


# r16 contractions with fewer 256 x 256 tiles than CTA pairs, which take the pairs where that saves rounds of tiles: ragged last tiles of both
# directions, one K block more than whole ones, a residual, a bias and the old C.  Bit for bit as the single CTAs' kernel has them, and that to the
# rounding of a result.
@pytest.mark.parametrize("shape,pairs", [((3000, 1000, 1000), True), ((2824, 1032, 776), True), ((4096, 1096, 520), True), ((2048, 2048, 2048), True),
                                         ((2570, 1032, 776), False)])      # (one round of single CTAs' tiles)
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ij_kj_ik", "ji_jk_ik"])
def test_pairs_on_few_tiles(mp, stream, monkeypatch, shape, pairs, variant):
    import torch
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    a, b = torch.randn(m, n, generator=g, device="cuda").half(), torch.randn(n, k, generator=g, device="cuda").half()
    term, bias = torch.randn(m, k, generator=g, device="cuda").half(), torch.randn(k, generator=g, device="cuda").half()
    da = (a.t() if variant[0] == "j" else a).contiguous()
    db = (b.t() if variant[3:5] == "kj" else b).contiguous()
    ref = a.double() @ b.double()

    def results():
        out = [torch.full((m, k), 3.0, device="cuda", dtype=torch.float16) for _ in range(4)]
        run(mp, stream, "inner_product_" + variant, "r16", da, db, 1.0, out[0], 0.0, m, n, k)
        run(mp, stream, "inner_product_" + variant, "r16", da, db, 0.5, out[1], 2.0, m, n, k)
        if variant == "ij_jk_ik":
            run(mp, stream, "linear_ij_jk_ik_ik", "r16", da, db, term, 1.0, out[2], 0.0, m, n, k)
            run(mp, stream, "linear_ij_jk_ik", "r16", da, db, bias, 1.0, out[3], 0.0, m, n, k)
        return out

    want = [ref, 0.5 * ref + 6.0, ref + term.double(), ref + bias.double()]
    got = results()
    assert all(("pair" in name) == pairs for name in kernels(results))
    monkeypatch.setenv("MP_GEMM_NO_PAIRS", "1")      # read at every launch
    single = results()
    assert not any("pair" in name for name in kernels(results))
    for c, s, w in list(zip(got, single, want))[:4 if variant == "ij_jk_ik" else 2]:
        assert torch.equal(c, s)
        assert float((s.double() - w).norm() / w.norm()) <= 2.9e-4      # the rounding of an r16 result
    assert stream.status() == 0


# CTA pairs on an A of more than 64 MB, where tiles come in groups of eight row blocks: 34 row blocks, so that the last group has two.
@pytest.mark.parametrize("variant", ["ij_jk_ik", "ji_jk_ik"])
def test_pairs_in_groups_of_row_blocks(mp, stream, monkeypatch, variant):
    import torch
    m, n, k = 8488, 4096, 1288
    g = torch.Generator(device="cuda").manual_seed(m)
    a, b = torch.randn(m, n, generator=g, device="cuda").half(), torch.randn(n, k, generator=g, device="cuda").half()
    da = (a.t() if variant[0] == "j" else a).contiguous()

    def result():
        c = torch.full((m, k), 3.0, device="cuda", dtype=torch.float16)
        run(mp, stream, "inner_product_" + variant, "r16", da, b, 1.0, c, 0.0, m, n, k)
        return c

    c = result()
    assert all("pair" in name for name in kernels(result))
    ref = a.double() @ b.double()
    assert bool(((c.double() - ref).norm(dim=1) <= 2.9e-4 * ref.norm(dim=1)).all())      # the rounding of an r16 result, every row
    monkeypatch.setenv("MP_GEMM_NO_PAIRS", "1")      # read at every launch
    assert torch.equal(c, result())
    assert stream.status() == 0


# CTA pairs into a C with rows off the 16-byte boundary, from aligned operands: whole words, odd ends, a last block of one column.
@pytest.mark.parametrize("shape", [(6000, 512, 1001), (5001, 128, 2049), (4870, 256, 1059)])
@pytest.mark.parametrize("off", [0, 1])
def test_pairs_into_rows_off_the_boundary(mp, stream, monkeypatch, shape, off):
    import torch
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    a, b = torch.randn(m, n, generator=g, device="cuda").half(), torch.randn(k, n, generator=g, device="cuda").half()

    def result():
        flat = torch.full((m * k + 16,), 7.0, device="cuda", dtype=torch.float16)
        run(mp, stream, "inner_product_ij_kj_ik", "r16", a, b, 1.0, flat[off:off + m * k].view(m, k), 0.0, m, n, k)
        return flat

    flat = result()
    assert all("pair" in name for name in kernels(result))
    ref = a.double() @ b.double().t()
    c = flat[off:off + m * k].view(m, k).double()
    assert bool(((c - ref).norm(dim=1) <= 2.9e-4 * ref.norm(dim=1)).all())      # the rounding of an r16 result, every row
    assert bool((flat[:off] == 7).all()) and bool((flat[off + m * k:] == 7).all())
    monkeypatch.setenv("MP_GEMM_NO_PAIRS", "1")      # read at every launch
    assert torch.equal(flat, result())
    assert stream.status() == 0
