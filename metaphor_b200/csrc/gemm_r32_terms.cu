// r32 contractions of some size: the operands are first written as two r16 terms each, and the products are r16 MMAs on CTA pairs.
//
// A value becomes hi + lo under a power of two that brings the largest value of its 64 along K below 2^15: 23 bits, and 40 binary
// orders below the largest value.  a b ~ hi_a hi_b + hi_a lo_b + lo_a hi_b, as in gemm_r32.cu; but an r16 MMA takes twice the K of a tf32 one
// in the same time, its operands are half as large in shared memory, and nothing is left to split in the kernel.  The scales of a
// k-block (64 of K) are undone when its accumulator is handed over to the epilogue warps, which add it up in registers with rounding; the
// small products of a k-block come before the large ones, so that only four additions truncate at full size.  2-norm of the error at
// [2000, 999, 1501], normal operands / operands of one sign: 1.5e-7 / 2.1e-7 (gemm_r32.cu for unaligned operands 1.7e-7 / 1.6e-7, for
// aligned ones 9.2e-7 / 1.65e-6).
//
// What bounds it is the tensor pipe: 1536 cycles of MMAs per k-block of a 256 x 256 tile, 1600 measured; beside that the pass over the operands,
// a tile's store (6 000 cycles, not hidden behind the next tile's first k-blocks) and waves that are not full.  us, all three forms of
// [2000, 999, 1501] with unaligned operands: 68 / 64 / 77 (gemm_r32.cu, copies included) -> 37 / 37 / 36;  [4001, 301, 2003] 54 / 52 / 58 -> 37 / 36 /
// 38;  [16384, 768, 3352] aligned 418 / 429 / 576 -> 324 / 330 / 295.
//
// The terms are copies in the stream's workspace: one pass over the operands, which also brings rows off the 16-byte boundary into line.
//   warp 0      TMA producer (one elected thread)
//   warp 1      MMA issuer (one elected thread of rank 0), owns the TMEM allocation; warps 2 and 3 only give their registers away
//   warps 4-11  accumulation and epilogue: warp w reads TMEM lane quarter w % 4 and one half of the columns
#include "mp_gemm.cuh"

namespace {

constexpr int H_THREADS = 384;
constexpr int H_EPI_FIRST = 4;
// registers a thread: 384 x 168 at launch = 128 x 56 (the first warpgroup) + 256 x 224
constexpr int H_REGS_FIRST = 56, H_REGS_EPI = 224;
constexpr int H_BK = 64, H_STAGES = 3, H_KSLICES = H_BK / 16;
constexpr int H_A = BM * SWIZZLE_BYTES;            // one term of 128 rows of A

template <int BN> struct TermsCfg {
  static constexpr int B = BN / 2 * SWIZZLE_BYTES;                 // one term of this CTA's half of the columns
  static constexpr int STAGE = 2 * (H_A + B);
  static constexpr int SCALES = 2 * (BN / 2) * 4;                  // per epilogue warp: its columns' scales of two k-blocks
  static constexpr int STORE = 16 * 32 * 4;                        // per epilogue warp: 16 rows of 32 columns
  static constexpr int SMEM = H_STAGES * STAGE + 1024 /*align*/ + 1024 /*barriers*/ + 8 * (SCALES + STORE);
};

// ---------------------------------------------------------------------------
// The terms of one operand: [rows][K] (K contiguous) or, MN, [K][rows].  Planes of the same order with a pitch of `ld`, scales [k-block][rows].
// ---------------------------------------------------------------------------
struct TermsJob {
  const float* src;
  __half *hi, *lo;
  float* scales;           // what a row's products of a k-block are multiplied by
  uint32_t rows, k;
  size_t src_ld, ld, scales_ld;
  uint32_t blocks;         // CTAs
  int mn, vec;             // vec: four (K contiguous) or two neighbouring values can be loaded at once
};
__device__ __forceinline__ uint32_t terms_bits(float v) {   // the scale is that of the finite values
  const uint32_t b = __float_as_uint(v) & 0x7fffffffu;
  return b < 0x7f800000u ? b : 0u;
}
__device__ __forceinline__ float terms_scale(uint32_t bits, float* inverse) {
  int e = 268 - static_cast<int>(bits >> 23);
  e = e < 253 ? e : 253;
  *inverse = __uint_as_float(static_cast<uint32_t>(254 - e) << 23);
  return __uint_as_float(static_cast<uint32_t>(e) << 23);
}
__device__ __forceinline__ void terms_of(float v0, float v1, float f, uint32_t& hi, uint32_t& lo) {
  v0 *= f;
  v1 *= f;
  const __half2 h = __floats2half2_rn(v0, v1);
  const float2 b = __half22float2(h);
  const __half2 l = __floats2half2_rn(v0 - b.x, v1 - b.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

__global__ void __launch_bounds__(256) r32_terms_kernel(const TermsJob ja, const TermsJob jb) {
  mp_grid_dependency();
  const bool second = blockIdx.x >= ja.blocks;
  const TermsJob& j = second ? jb : ja;
  const uint32_t block = second ? blockIdx.x - ja.blocks : blockIdx.x;
  const uint32_t kbs = (j.k + H_BK - 1) / H_BK;
  if (!j.mn) {   // eight values a thread, a k-block of a row on eight neighbouring threads
    const uint32_t id = block * 256u + threadIdx.x, row = id / (kbs * 8u), c = id - row * (kbs * 8u), k0 = c * 8u;
    const bool live = row < j.rows;
    float v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = 0.f;
    if (live && k0 < j.k) {
      const float* s = j.src + row * j.src_ld + k0;
      if (j.vec && k0 + 8u <= j.k) {
        const float4 p = *reinterpret_cast<const float4*>(s), r = *reinterpret_cast<const float4*>(s + 4);
        v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w; v[4] = r.x; v[5] = r.y; v[6] = r.z; v[7] = r.w;
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (k0 + e < j.k) v[e] = s[e];
      }
    }
    uint32_t m = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) m = max(m, terms_bits(v[e]));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    float inverse;
    const float f = terms_scale(m, &inverse);
    if (!live) return;
    if ((c & 7u) == 0) j.scales[(c >> 3) * j.scales_ld + row] = inverse;
    if (k0 >= j.ld) return;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) terms_of(v[2 * e], v[2 * e + 1], f, hi[e], lo[e]);
    *reinterpret_cast<uint4*>(j.hi + row * j.ld + k0) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(j.lo + row * j.ld + k0) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    return;
  }
  // a k-block of 64 rows: a warp takes eight steps of K, a lane two rows
  __shared__ uint32_t part[8][64];
  const uint32_t per = (j.rows + 63u) / 64u, kb = block / per, r0 = (block - kb * per) * 64u + 2u * (threadIdx.x & 31u);
  const uint32_t k0 = kb * H_BK + (threadIdx.x >> 5) * 8u;
  float v[8][2];
  uint32_t m0 = 0, m1 = 0;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    v[e][0] = v[e][1] = 0.f;
    if (k0 + e < j.k && r0 < j.rows) {
      const float* s = j.src + (k0 + e) * j.src_ld + r0;
      if (j.vec && r0 + 1u < j.rows) {
        const float2 p = *reinterpret_cast<const float2*>(s);
        v[e][0] = p.x;
        v[e][1] = p.y;
      } else {
        v[e][0] = s[0];
        if (r0 + 1u < j.rows) v[e][1] = s[1];
      }
    }
    m0 = max(m0, terms_bits(v[e][0]));
    m1 = max(m1, terms_bits(v[e][1]));
  }
  *reinterpret_cast<uint2*>(&part[threadIdx.x >> 5][2 * (threadIdx.x & 31)]) = make_uint2(m0, m1);
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    const uint2 p = *reinterpret_cast<const uint2*>(&part[w][2 * (threadIdx.x & 31)]);
    m0 = max(m0, p.x);
    m1 = max(m1, p.y);
  }
  float i0, i1;
  const float f0 = terms_scale(m0, &i0), f1 = terms_scale(m1, &i1);
  if (threadIdx.x < 32 && r0 < j.rows) {   // (scales_ld is even and covers the pair)
    j.scales[kb * j.scales_ld + r0] = i0;
    if (r0 + 1u < j.rows) j.scales[kb * j.scales_ld + r0 + 1u] = i1;
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (k0 + e >= j.k || r0 >= j.ld) continue;
    uint32_t hi, lo;
    terms_of(v[e][0] * f0, v[e][1] * f1, 1.f, hi, lo);
    *reinterpret_cast<uint32_t*>(j.hi + (k0 + e) * j.ld + r0) = hi;
    *reinterpret_cast<uint32_t*>(j.lo + (k0 + e) * j.ld + r0) = lo;
  }
}

// ---------------------------------------------------------------------------
// The contraction.  Barriers as in the r16 pair kernel (gemm.cu): full[s] on rank 0, credited by both ranks' loads; empty[s] and
// acc_full[b] on both, by the MMAs' commit; acc_empty[b] on rank 0, one arrival per epilogue warp of either rank.
// ---------------------------------------------------------------------------
struct TermsMaps { CUtensorMap a_hi, a_lo, b_hi, b_lo; };
struct TermsScales { const float *a, *b; size_t a_ld, b_ld; };

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(H_THREADS, 1)
    gemm_r32_terms_kernel(const __grid_constant__ TermsMaps maps, const GemmArgs g, const TermsScales sc, const Again again) {
  using Cfg = TermsCfg<BN>;
  extern __shared__ unsigned char gemm_smem_raw[];
  unsigned char* smem = mp_smem_align1024(gemm_smem_raw);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + H_STAGES * Cfg::STAGE);
  uint64_t* empty = full + H_STAGES;
  uint64_t* acc_full = empty + H_STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  unsigned char* epi = smem + H_STAGES * Cfg::STAGE + 1024;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int num_kb = (g.K + H_BK - 1) / H_BK;
  const int tiles_m = (g.M + 2 * BM - 1) / (2 * BM), tiles_n = (g.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int num_units = num_tiles * g.ksplit;   // unit = K split * tiles + tile
  const int kb_per = (num_kb + g.ksplit - 1) / g.ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < H_STAGES; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(acc_full + a, 1); mbar_init(acc_empty + a, 16); }
    *abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&maps.a_hi);
    tma_prefetch_desc(&maps.a_lo);
    tma_prefetch_desc(&maps.b_hi);
    tma_prefetch_desc(&maps.b_lo);
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 2 * BN);
  tcgen05_fence_before_sync();
  cluster_sync_all();   // both CTAs' barriers and TMEM exist before anything crosses the pair
  tcgen05_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  mp_grid_wait();

  if (warp < H_EPI_FIRST) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(H_REGS_FIRST));
  if (warp == 0) {
    // ------------------------------ TMA producer (both ranks) ------------------
    if (lane == 0) {
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = pair; unit < num_units && ok; unit += num_pairs) {
        const int tile = unit % num_tiles, sp = unit / num_tiles;
        const int m0 = (tile % tiles_m) * 2 * BM + static_cast<int>(rank) * BM;
        const int n0 = (tile / tiles_m) * BN + static_cast<int>(rank) * (BN / 2);
        const int kb0 = sp * kb_per, kb1 = min(num_kb, kb0 + kb_per);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_abortable(empty + s, phase ^ 1u, g.status, abort)) { ok = false; break; }
          if (rank == 0) mbar_arrive_expect_tx(full + s, 2 * Cfg::STAGE);
          unsigned char* dst = smem + s * Cfg::STAGE;
          const int k0 = kb * H_BK;
          auto load = [&](unsigned char* to, const CUtensorMap* map, bool mn, int x0, int rows) {
#pragma unroll 1
            for (int i = 0; i < (mn ? rows / H_BK : 1); ++i)
              tma_load_2d_pair(to + i * (H_BK * SWIZZLE_BYTES), map, mn ? x0 + i * H_BK : k0, mn ? k0 : x0, full + s);
          };
          load(dst, &maps.a_hi, g.a_mn != 0, m0, BM);
          load(dst + H_A, &maps.a_lo, g.a_mn != 0, m0, BM);
          load(dst + 2 * H_A, &maps.b_hi, g.b_mn != 0, n0, BN / 2);
          load(dst + 2 * H_A + Cfg::B, &maps.b_lo, g.b_mn != 0, n0, BN / 2);
          if (++s == H_STAGES) { s = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (rank 0) -------------------------
    if (rank == 0) {   // the warp as a whole, see elect_one
      const uint32_t idesc = umma_instr_desc(UMMA_FMT_F16, g.a_mn, g.b_mn, 2 * BM, BN);
      const uint32_t a_lbo = g.a_mn ? H_BK * SWIZZLE_BYTES : 16, b_lbo = g.b_mn ? H_BK * SWIZZLE_BYTES : 16;
      const uint32_t au = (g.a_mn ? 16 * SWIZZLE_BYTES : 32) >> 4, bu = (g.b_mn ? 16 * SWIZZLE_BYTES : 32) >> 4;
      const uint32_t base = mp_smem_u32(smem);
      const uint64_t ah0 = umma_smem_desc(base, a_lbo, 1024), bh0 = umma_smem_desc(base + 2 * H_A, b_lbo, 1024);
      int s = 0;
      uint32_t phase = 0, chunk = 0;
      bool ok = true;
      for (int unit = pair; unit < num_units && ok; unit += num_pairs) {
        const int sp = unit / num_tiles;
        const int kb0 = sp * kb_per, kb1 = min(num_kb, kb0 + kb_per);
        for (int kb = kb0; kb < kb1; ++kb, ++chunk) {
          const uint32_t buf = chunk & 1u;
          ok = mbar_wait_abortable(acc_empty + buf, ((chunk >> 1) & 1u) ^ 1u, g.status, abort) && mbar_wait_abortable(full + s, phase, g.status, abort);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tcgen05_fence_after_sync();
          const uint32_t acc = tmem_base + buf * BN, off = static_cast<uint32_t>(s * (Cfg::STAGE >> 4));
          const uint64_t ah = ah0 + off, al = ah + (H_A >> 4), bh = bh0 + off, bl = bh + (Cfg::B >> 4);
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < H_KSLICES; ++ks) {
              umma_pair_f16(acc, al + ks * au, bh + ks * bu, idesc, ks != 0 ? 1u : 0u);
              umma_pair_f16(acc, ah + ks * au, bl + ks * bu, idesc, 1u);
            }
#pragma unroll
            for (int ks = 0; ks < H_KSLICES; ++ks) umma_pair_f16(acc, ah + ks * au, bh + ks * bu, idesc, 1u);
            umma_commit_pair_to(empty + s, 3);
            umma_commit_pair_to(acc_full + buf, 3);
          }
          __syncwarp();
          if (++s == H_STAGES) { s = 0; phase ^= 1u; }
        }
      }
    }
    mp_launch_dependents();
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(H_REGS_EPI));
    // ------------------------------ accumulation and epilogue (both ranks) ------
    constexpr int NB = BN / 64;                   // 32-column blocks per warp
    const int quarter = warp & 3, half = (warp - H_EPI_FIRST) >> 2;
    const float* bias = static_cast<const float*>(g.bias);
    float* scales = reinterpret_cast<float*>(epi + (warp - H_EPI_FIRST) * (Cfg::SCALES + Cfg::STORE));   // [2][BN / 2]
    float* stage = scales + 2 * (BN / 2);
    uint32_t chunk = 0;
    bool ok = true;
    for (int unit = pair; unit < num_units && ok; unit += num_pairs) {
      const int tile = unit % num_tiles, sp = unit / num_tiles;
      const int row0 = (tile % tiles_m) * 2 * BM + static_cast<int>(rank) * BM + quarter * 32, row = row0 + lane;
      const int colw = (tile / tiles_m) * BN + half * (BN / 2);   // this warp's columns
      const int kb0 = sp * kb_per, kb1 = min(num_kb, kb0 + kb_per);
      // scales of a k-block: this lane's row, the warp's columns (their rows in memory are padded to whole tiles)
      auto fetch = [&](int kb, int slot) {
        if (lane * 4 < BN / 2) {
          const uint32_t dst = mp_smem_u32(scales + slot * (BN / 2) + lane * 4);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(sc.b + kb * sc.b_ld + colw + lane * 4) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        return sc.a[kb * sc.a_ld + row];
      };
      float acc[NB][32];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int e = 0; e < 32; ++e) acc[nb][e] = 0.f;
      float next = fetch(kb0, 0);
      for (int kb = kb0; kb < kb1; ++kb, ++chunk) {
        const uint32_t buf = chunk & 1u;
        const int slot = (kb - kb0) & 1;
        const float fa = next;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        if (kb + 1 < kb1) next = fetch(kb + 1, slot ^ 1);
        ok = mbar_wait_abortable(acc_full + buf, (chunk >> 1) & 1u, g.status, abort);
        ok = __all_sync(0xffffffffu, ok);   // tcgen05.ld is warp-collective
        if (!ok) break;
        tcgen05_fence_after_sync();
        const float4* fb = reinterpret_cast<const float4*>(scales + slot * (BN / 2));
        const uint32_t src = tmem_base + buf * BN + (static_cast<uint32_t>(quarter * 32) << 16) + half * (BN / 2);
#pragma unroll
        for (int nb = 0; nb < NB; nb += 2) {   // two loads in flight
          uint32_t v[2][32];
          tmem_ld_32x32(src + nb * 32, v[0]);
          if (nb + 1 < NB) tmem_ld_32x32(src + (nb + 1) * 32, v[1]);
          tmem_ld_wait();
#pragma unroll
          for (int u = 0; u < 2 && nb + u < NB; ++u)
#pragma unroll
            for (int p = 0; p < 8; ++p) {
              const float4 f = fb[(nb + u) * 8 + p];
              float* sum = acc[nb + u] + 4 * p;
              sum[0] = fmaf(__uint_as_float(v[u][4 * p]), fa * f.x, sum[0]);
              sum[1] = fmaf(__uint_as_float(v[u][4 * p + 1]), fa * f.y, sum[1]);
              sum[2] = fmaf(__uint_as_float(v[u][4 * p + 2]), fa * f.z, sum[2]);
              sum[3] = fmaf(__uint_as_float(v[u][4 * p + 3]), fa * f.w, sum[3]);
            }
        }
        tcgen05_fence_before_sync();
        __syncwarp();
        if (lane == 0) {
          if (rank == 0) mbar_arrive(acc_empty + buf);
          else mbar_arrive_cluster(acc_empty + buf, 0);
        }
      }
      if (!ok) break;
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const int col0 = colw + nb * 32;
        if (col0 >= g.N || row0 >= g.M) continue;   // uniform across the warp
        float* r = acc[nb];
        if (g.ksplit > 1) {   // raw partial sums; alpha, bias and beta are applied by the fold
          if (row < g.M) {
            float* prow = g.partial + (static_cast<size_t>(sp) * g.M + row) * g.partial_ld + col0;
            if (col0 + 32 <= g.N) {
#pragma unroll
              for (int p = 0; p < 8; ++p) *reinterpret_cast<float4*>(prow + p * 4) = make_float4(r[p * 4], r[p * 4 + 1], r[p * 4 + 2], r[p * 4 + 3]);
            } else {
#pragma unroll
              for (int e = 0; e < 32; ++e)
                if (col0 + e < g.N) prow[e] = r[e];
            }
          }
          continue;
        }
        bool nan = false;
        if (g.exact) {
#pragma unroll
          for (int e = 0; e < 32; ++e) nan = nan || r[e] != r[e];
          nan = __any_sync(0xffffffffu, nan);
        }
        // sixteen rows at a time through the staging, as in store_block_rows
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if ((lane >> 4) == h) {
#pragma unroll
            for (int e = 0; e < 32; ++e) stage[(lane & 15) * 32 + (e ^ (lane & 15))] = r[e];
          }
          __syncwarp();
          const int first = row0 + h * 16, col = col0 + lane;
          float* c = static_cast<float*>(g.c) + static_cast<size_t>(first) * g.ldc + col;
          const float* mat = bias != nullptr ? bias + static_cast<size_t>(first) * g.bias_pitch + col : nullptr;
#pragma unroll 1
          for (int i0 = 0; i0 < 16; i0 += 8) {
            const int n = col < g.N ? min(8, g.M - first - i0) : 0;
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = stage[(i0 + u) * 32 + (lane ^ (i0 + u))];
            if (nan) {   // rare, see dot_again (in line: a call would fix the registers of the whole kernel)
#pragma unroll 1
              for (int u = 0; u < n; ++u) {
                if (stage[(i0 + u) * 32 + (lane ^ (i0 + u))] == stage[(i0 + u) * 32 + (lane ^ (i0 + u))]) continue;
                const int m = first + i0 + u;
                const float *pa = again.a + (g.a_mn ? m : m * again.a_ld), *pb = again.b + (g.b_mn ? col : col * again.b_ld);
                float sum = 0.f;
#pragma unroll 1
                for (int k = 0; k < g.K && sum == sum; ++k) sum = fmaf(pa[k * (g.a_mn ? again.a_ld : 1)], pb[k * (g.b_mn ? again.b_ld : 1)], sum);
                stage[(i0 + u) * 32 + (lane ^ (i0 + u))] = sum;   // (read by this lane alone)
              }
#pragma unroll
              for (int u = 0; u < 8; ++u) v[u] = stage[(i0 + u) * 32 + (lane ^ (i0 + u))];
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] *= g.alpha;
            if (mat != nullptr) {
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (u < n) v[u] += mat[u * g.bias_pitch];
              mat += 8 * g.bias_pitch;
            }
            if (g.beta != 0.0f) {
#pragma unroll
              for (int u = 0; u < 8; ++u)
                if (u < n) v[u] += g.beta * c[u * g.ldc];
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (u < n) c[u * g.ldc] = v[u];
            c += 8 * g.ldc;
          }
          __syncwarp();
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  __syncwarp();         // the cluster barrier below is warp-aligned: lanes that skipped the role loops wait here
  tcgen05_fence_before_sync();
  cluster_sync_all();   // neither CTA frees TMEM or leaves while its partner may still read its memory
  if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * BN);
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
size_t up(size_t v, size_t to) { return (v + to - 1) / to * to; }

struct TermsPlan { int bn = 0, ksplit = 1; double cycles = 1e300; };
// The tile (256 x 256 or 256 x 128) and the number of K splits with the smallest estimate of
//     waves over the pairs x (k-blocks per unit x cycles per k-block + cycles to store a unit) + start  [+ the fold]
// with the cycles per k-block measured at [4096, 1024] x [1024, 4096] (the MMAs alone: 1536 and 768).
TermsPlan terms_plan(const GemmArgs& args, int sms, size_t partial_bytes) {
  TermsPlan best;
  const long num_kb = (args.K + H_BK - 1) / H_BK, pairs = sms / 2;
  const double mn_bytes = static_cast<double>(args.M) * args.partial_ld * 4.0;
  const int max_ks = env_flag("MP_GEMM_NO_SPLITK") ? 1 : 16;
  for (int bn = 256; bn >= 128; bn /= 2) {
    const double cycles = bn == 256 ? 1650.0 : 1100.0;
    const long tiles = static_cast<long>((args.M + 255) / 256) * ((args.N + bn - 1) / bn);
    for (int ks = 1; ks <= max_ks; ++ks) {
      const long per = (num_kb + ks - 1) / ks;
      if (ks > 1 && (per < 2 || (ks - 1) * per >= num_kb || ks * mn_bytes > static_cast<double>(partial_bytes))) continue;
      double cost = static_cast<double>((tiles * ks + pairs - 1) / pairs) * (per * cycles + 6000.0) + 15000.0;
      if (ks > 1) cost += 5000.0 + 2.0 * ks * mn_bytes / 3500.0;
      if (cost < best.cycles) { best.cycles = cost; best.bn = bn; best.ksplit = ks; }
    }
  }
  return best;
}

template <int BN>
void launch_terms(const TermsMaps& maps, const GemmArgs& g, const TermsScales& sc, const Again& again, int sms, cudaStream_t st) {
  MP_CUDA_CHECK(cudaFuncSetAttribute(gemm_r32_terms_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, TermsCfg<BN>::SMEM));
  const long units = static_cast<long>((g.N + BN - 1) / BN) * ((g.M + 2 * BM - 1) / (2 * BM)) * g.ksplit;
  const long pairs = units < sms / 2 ? units : sms / 2;
  MpLaunch(static_cast<unsigned>(2 * pairs), H_THREADS, TermsCfg<BN>::SMEM, st)(gemm_r32_terms_kernel<BN>, maps, g, sc, again);
  MP_LAUNCH_CHECK();
}

}  // namespace

// Runs the contraction when its terms fit the workspace and the estimate is below `limit_cycles` (that of the tf32 kernel); any operand
// alignment.
bool gemm_run_r32_terms(Operand<float> a, Operand<float> b, GemmArgs args, int sms, void* workspace, size_t workspace_bytes, double limit_cycles,
                        cudaStream_t st) {
  const size_t M = args.M, N = args.N, K = args.K, kbs = (K + H_BK - 1) / H_BK;
  args.partial_ld = (args.N + 3) & ~3;
  size_t used = 0;
  auto take = [&](size_t bytes) { void* p = static_cast<unsigned char*>(workspace) + used; used += up(bytes, 256); return p; };
  auto job = [&](const Operand<float>& o, size_t rows, int mn) {
    TermsJob j;
    j.src = o.p;
    j.src_ld = o.ld;
    j.rows = static_cast<uint32_t>(rows);
    j.k = static_cast<uint32_t>(K);
    j.mn = mn;
    j.ld = up(mn ? rows : K, 8);
    j.scales_ld = up(rows, 256);
    const size_t plane = (mn ? K : rows) * j.ld * sizeof(__half);
    j.hi = static_cast<__half*>(take(plane));
    j.lo = static_cast<__half*>(take(plane));
    j.scales = static_cast<float*>(take(kbs * j.scales_ld * sizeof(float)));
    j.vec = mn ? (reinterpret_cast<uintptr_t>(o.p) % 8 == 0 && o.ld % 2 == 0) : (mp_aligned16(o.p) && o.ld % 4 == 0);
    j.blocks = static_cast<uint32_t>(mn ? kbs * ((rows + 63) / 64) : (rows * kbs * 8 + 255) / 256);
    return j;
  };
  if (static_cast<double>(M + N) * K * 4.0 > static_cast<double>(workspace_bytes)) return false;
  const TermsJob ja = job(a, M, args.a_mn), jb = job(b, N, args.b_mn);
  if (used > workspace_bytes) return false;
  const TermsPlan plan = terms_plan(args, sms, workspace_bytes - used);
  // the terms: 8 bytes an element at 2.5 KB a cycle, and a launch
  if (plan.cycles + 5000.0 + static_cast<double>(M + N) * K * 8.0 / 2500.0 > limit_cycles) return false;
  args.ksplit = plan.ksplit;
  args.partial = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + used);
  MpLaunch(ja.blocks + jb.blocks, 256, 0, st)(r32_terms_kernel, ja, jb);
  MP_LAUNCH_CHECK();
  auto map = [&](const __half* p, const TermsJob& j, size_t rows, int mn, uint32_t box) {
    return mn ? make_map<__half>(p, K, rows, j.ld, H_BK, H_BK) : make_map<__half>(p, rows, K, j.ld, H_BK, box);
  };
  const uint32_t bbox = static_cast<uint32_t>(plan.bn / 2);
  const TermsMaps maps{map(ja.hi, ja, M, args.a_mn, BM), map(ja.lo, ja, M, args.a_mn, BM), map(jb.hi, jb, N, args.b_mn, bbox), map(jb.lo, jb, N, args.b_mn, bbox)};
  const TermsScales sc{ja.scales, jb.scales, ja.scales_ld, jb.scales_ld};
  const Again again{a.p, b.p, a.ld, b.ld};
  if (plan.bn == 256) launch_terms<256>(maps, args, sc, again, sms, st);
  else launch_terms<128>(maps, args, sc, again, sms, st);
  if (args.ksplit > 1) {
    if (args.exact) launch_fold<float>(args, AgainFold{again, args.a_mn, args.b_mn, args.K}, st);
    else launch_fold<float>(args, NoAgain{}, st);
  }
  return true;
}
