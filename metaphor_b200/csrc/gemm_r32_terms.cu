// r32 contractions of some size: the operands are first written as three bf16 terms each, and the products are bf16 MMAs on CTA pairs.
//
// A value becomes h0 + h1 + h2, each the rest of the one before rounded to bf16: 24 bits, all there are, and as bf16 has the exponents of fp32 every
// value keeps its own (the last terms of values below 2^-110 are rounded to multiples of 2^-133; gemm_r32.cu cuts them off at 2^-136).  Of the nine products the three of the smallest terms are left out:
//     a b ~ a0 b0 + (a0 b1 + a1 b0) + (a0 b2 + a2 b0 + a1 b1),    2^-26 of a product at most.
// The tensor core's accumulator truncates, so that it is handed over to the epilogue warps every 32 of K, which add it up in registers with
// rounding; the small products come before the large ones, so that only two additions truncate at full size.  2-norm of the error at
// [2000, 999, 1501], normal operands / operands of one sign: 1.2e-7 / 1.1e-7 (gemm_r32.cu for unaligned operands 1.7e-7 / 1.6e-7, for aligned
// ones 9.2e-7 / 1.65e-6).
//
// What bounds it is the tensor pipe: 3072 cycles of MMAs per 64 of K of a 256 x 256 tile, 3500 measured under the power they take; beside that the pass over
// the operands, the results' store (1.5 KB a cycle, not hidden behind the next tile's first k-blocks) and waves that are not full.  us, gemm_r32.cu
// (copies included) -> here, all three forms: [2000, 999, 1501] unaligned 64 / 64 / 74 -> 48 / 50 / 48; [4001, 301, 2003] 52 / 50 / 56 -> 45; [2048, 2048,
// 2048] aligned 101 / 96 / 129 -> 91.  Tried: four stages of 32 of K in the 64-byte swizzle (level, A or B along M or N 8 % slower); two r16 terms under
// a power of two per 64 of K, which are three products (37 us), but one exponent for 64 values: those far below the largest lost their bits.
//
// The terms are copies in the stream's workspace: one pass over the operands, which also brings rows off the 16-byte boundary into line.
//   warp 0      TMA producer (one elected thread)
//   warp 1      MMA issuer (one elected thread of rank 0), owns the TMEM allocation; warps 2 and 3 only give their registers away
//   warps 4-11  accumulation and epilogue: warp w reads TMEM lane quarter w % 4 and one half of the columns
#include "mp_gemm.cuh"

#include <cuda_bf16.h>

namespace {

constexpr int H_THREADS = 384;
constexpr int H_EPI_FIRST = 4;
// registers a thread: 384 x 168 at launch = 128 x 56 (the first warpgroup) + 256 x 224
constexpr int H_REGS_FIRST = 56, H_REGS_EPI = 224;
constexpr int H_BK = 64, H_STAGES = 2;             // of K per stage
constexpr int H_PART = 32, H_KSLICES = H_PART / 16;   // of K per hand-over
constexpr int H_A = BM * SWIZZLE_BYTES;            // one term of 128 rows of A

template <int BN> struct TermsCfg {
  static constexpr int B = BN / 2 * SWIZZLE_BYTES;                 // one term of this CTA's half of the columns
  static constexpr int STAGE = 3 * (H_A + B);
  static constexpr int STORE = 16 * 32 * 4;                        // per epilogue warp: 16 rows of 32 columns
  static constexpr int SMEM = H_STAGES * STAGE + 1024 /*align*/ + 1024 /*barriers*/ + 8 * STORE;
};

// ---------------------------------------------------------------------------
// The terms of one operand, [rows][cols] as it lies in memory: three planes with a pitch of `ld`.
// ---------------------------------------------------------------------------
struct TermsJob {
  const float* src;
  __nv_bfloat16* term[3];
  uint32_t rows, cols;
  size_t src_ld, ld;       // ld: a multiple of 8
  uint32_t blocks;         // CTAs
  int vec;                 // four neighbouring values can be loaded at once
};

__global__ void __launch_bounds__(256) r32_terms_kernel(const TermsJob ja, const TermsJob jb) {
  mp_grid_dependency();
  const bool second = blockIdx.x >= ja.blocks;
  const TermsJob& j = second ? jb : ja;
  const uint32_t per_row = static_cast<uint32_t>(j.ld / 4), id = (second ? blockIdx.x - ja.blocks : blockIdx.x) * 256u + threadIdx.x;
  const uint32_t row = id / per_row, c = (id - row * per_row) * 4u;   // four values a thread
  if (row >= j.rows) return;
  const float* s = j.src + row * j.src_ld + c;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (j.vec && c + 4u <= j.cols) {
    const float4 p = *reinterpret_cast<const float4*>(s);
    v[0] = p.x; v[1] = p.y; v[2] = p.z; v[3] = p.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (c + e < j.cols) v[e] = s[e];
  }
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    uint2 out;
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      // a finite value must not round up to infinity; an infinite or NaN one has a NaN as its last term
      constexpr float MAX = 3.38953139e38f;   // the largest bf16
      const __nv_bfloat162 h = t == 0 ? __floats2bfloat162_rn(fminf(fmaxf(v[e], -MAX), MAX), fminf(fmaxf(v[e + 1], -MAX), MAX))
                                      : __floats2bfloat162_rn(v[e], v[e + 1]);
      const float2 f = __bfloat1622float2(h);
      v[e] -= f.x;
      v[e + 1] -= f.y;
      (e == 0 ? out.x : out.y) = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint2*>(j.term[t] + row * j.ld + c) = out;
  }
}

// ---------------------------------------------------------------------------
// The contraction.  Barriers as in the r16 pair kernel (gemm.cu): full[s] on rank 0, credited by both ranks' loads; empty[s] and
// acc_full[b] on both, by the MMAs' commit; acc_empty[b] on rank 0, one arrival per epilogue warp of either rank.
// ---------------------------------------------------------------------------
struct TermsMaps { CUtensorMap a[3], b[3]; };

template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(H_THREADS, 1)
    gemm_r32_terms_kernel(const __grid_constant__ TermsMaps maps, const GemmArgs g, const Again again) {
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
  const int num_kb = (g.K + H_BK - 1) / H_BK, num_parts = (g.K + H_PART - 1) / H_PART;
  const int tiles_m = (g.M + 2 * BM - 1) / (2 * BM), tiles_n = (g.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int num_units = num_tiles * g.ksplit;   // unit = K split * tiles + tile
  const int kb_per = (num_kb + g.ksplit - 1) / g.ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < H_STAGES; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(acc_full + a, 1); mbar_init(acc_empty + a, 16); }
    *abort = 0;
    mbar_fence_init();
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      tma_prefetch_desc(&maps.a[t]);
      tma_prefetch_desc(&maps.b[t]);
    }
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
#pragma unroll
          for (int t = 2; t >= 0; --t) {
            load(dst + t * H_A, &maps.a[t], g.a_mn != 0, m0, BM);
            load(dst + 3 * H_A + t * Cfg::B, &maps.b[t], g.b_mn != 0, n0, BN / 2);
          }
          if (++s == H_STAGES) { s = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (rank 0) -------------------------
    if (rank == 0) {   // the warp as a whole, see elect_one
      const uint32_t idesc = umma_instr_desc(UMMA_FMT_BF16, g.a_mn, g.b_mn, 2 * BM, BN);
      const uint32_t a_lbo = g.a_mn ? H_BK * SWIZZLE_BYTES : 16, b_lbo = g.b_mn ? H_BK * SWIZZLE_BYTES : 16;
      const uint32_t au = (g.a_mn ? 16 * SWIZZLE_BYTES : 32) >> 4, bu = (g.b_mn ? 16 * SWIZZLE_BYTES : 32) >> 4;   // 16 of K
      const uint32_t base = mp_smem_u32(smem);
      const uint64_t a00 = umma_smem_desc(base, a_lbo, 1024), b00 = umma_smem_desc(base + 3 * H_A, b_lbo, 1024);
      constexpr uint32_t AT = H_A >> 4, BT = Cfg::B >> 4;   // from term to term
      int s = 0;
      uint32_t phase = 0, chunk = 0;
      bool ok = true;
      for (int unit = pair; unit < num_units && ok; unit += num_pairs) {
        const int sp = unit / num_tiles;
        const int part0 = 2 * sp * kb_per, part1 = min(num_parts, part0 + 2 * kb_per);
        for (int part = part0; part < part1; ++part, ++chunk) {
          const uint32_t buf = chunk & 1u;
          const bool first = (part & 1) == 0, last = !first || part + 1 == part1;   // of the stage
          ok = mbar_wait_abortable(acc_empty + buf, ((chunk >> 1) & 1u) ^ 1u, g.status, abort) &&
               (!first || mbar_wait_abortable(full + s, phase, g.status, abort));
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tcgen05_fence_after_sync();
          const uint32_t acc = tmem_base + buf * BN, off = static_cast<uint32_t>(s * (Cfg::STAGE >> 4)), half = first ? 0u : H_KSLICES;
          const uint64_t a0 = a00 + off + half * au, b0 = b00 + off + half * bu;
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < H_KSLICES; ++ks) {
              umma_pair_f16(acc, a0 + AT + ks * au, b0 + BT + ks * bu, idesc, ks != 0 ? 1u : 0u);
              umma_pair_f16(acc, a0 + 2 * AT + ks * au, b0 + ks * bu, idesc, 1u);
              umma_pair_f16(acc, a0 + ks * au, b0 + 2 * BT + ks * bu, idesc, 1u);
            }
#pragma unroll
            for (int ks = 0; ks < H_KSLICES; ++ks) {
              umma_pair_f16(acc, a0 + AT + ks * au, b0 + ks * bu, idesc, 1u);
              umma_pair_f16(acc, a0 + ks * au, b0 + BT + ks * bu, idesc, 1u);
            }
#pragma unroll
            for (int ks = 0; ks < H_KSLICES; ++ks) umma_pair_f16(acc, a0 + ks * au, b0 + ks * bu, idesc, 1u);
            if (last) umma_commit_pair_to(empty + s, 3);
            umma_commit_pair_to(acc_full + buf, 3);
          }
          __syncwarp();
          if (last && ++s == H_STAGES) { s = 0; phase ^= 1u; }
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
    float* stage = reinterpret_cast<float*>(epi + (warp - H_EPI_FIRST) * Cfg::STORE);
    uint32_t chunk = 0;
    bool ok = true;
    for (int unit = pair; unit < num_units && ok; unit += num_pairs) {
      const int tile = unit % num_tiles, sp = unit / num_tiles;
      const int row0 = (tile % tiles_m) * 2 * BM + static_cast<int>(rank) * BM + quarter * 32, row = row0 + lane;
      const int colw = (tile / tiles_m) * BN + half * (BN / 2);   // this warp's columns
      const int part0 = 2 * sp * kb_per, part1 = min(num_parts, part0 + 2 * kb_per);
      float acc[NB][32];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int e = 0; e < 32; ++e) acc[nb][e] = 0.f;
      for (int part = part0; part < part1; ++part, ++chunk) {
        const uint32_t buf = chunk & 1u;
        ok = mbar_wait_abortable(acc_full + buf, (chunk >> 1) & 1u, g.status, abort);
        ok = __all_sync(0xffffffffu, ok);   // tcgen05.ld is warp-collective
        if (!ok) break;
        tcgen05_fence_after_sync();
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
            for (int e = 0; e < 32; ++e) acc[nb + u][e] += __uint_as_float(v[u][e]);
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
//     waves over the pairs x (k-blocks per unit x cycles per k-block + cycles to fill and to drain a unit) + the results' bytes at 1.5 KB a cycle
// or, split, + the fold.  Cycles per k-block under load: the MMAs alone are 3072 and 1536, and the clock gives way to the power they take.  us, estimate
// (at 1.9 GHz) / measured: [2000, 999, 1501] 47 / 49, [2048, 2048, 2048] 89 / 92, [4096, 1024, 4096] 172 / 176, [4096, 256, 4096] 70 / 71, [2560, 1280, 1024]
// 56 / 56, [1500, 1501, 1499] 45 / 42 (split).
TermsPlan terms_plan(const GemmArgs& args, int sms, size_t partial_bytes) {
  TermsPlan best;
  const long num_kb = (args.K + H_BK - 1) / H_BK, pairs = sms / 2;
  const double mn_bytes = static_cast<double>(args.M) * args.partial_ld * 4.0;
  const int max_ks = env_flag("MP_GEMM_NO_SPLITK") ? 1 : 16;
  for (int bn = 256; bn >= 128; bn /= 2) {
    const double cycles = bn == 256 ? 3500.0 : 2000.0;
    const long tiles = static_cast<long>((args.M + 255) / 256) * ((args.N + bn - 1) / bn);
    for (int ks = 1; ks <= max_ks; ++ks) {
      const long per = (num_kb + ks - 1) / ks;
      if (ks > 1 && (per < 2 || (ks - 1) * per >= num_kb || ks * mn_bytes > static_cast<double>(partial_bytes))) continue;
      double cost = static_cast<double>((tiles * ks + pairs - 1) / pairs) * (per * cycles + 4000.0) + 8000.0;
      cost += ks > 1 ? 5000.0 + 2.0 * ks * mn_bytes / 3500.0 : mn_bytes / 1500.0;
      if (cost < best.cycles) { best.cycles = cost; best.bn = bn; best.ksplit = ks; }
    }
  }
  return best;
}

template <int BN>
void launch_terms(const TermsMaps& maps, const GemmArgs& g, const Again& again, int sms, cudaStream_t st) {
  MP_CUDA_CHECK(cudaFuncSetAttribute(gemm_r32_terms_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, TermsCfg<BN>::SMEM));
  const long units = static_cast<long>((g.N + BN - 1) / BN) * ((g.M + 2 * BM - 1) / (2 * BM)) * g.ksplit;
  const long pairs = units < sms / 2 ? units : sms / 2;
  MpLaunch(static_cast<unsigned>(2 * pairs), H_THREADS, TermsCfg<BN>::SMEM, st)(gemm_r32_terms_kernel<BN>, maps, g, again);
  MP_LAUNCH_CHECK();
}

}  // namespace

// Runs the contraction when its terms fit the workspace and the estimate is below `limit_cycles` (that of the tf32 kernel); any operand
// alignment.
bool gemm_run_r32_terms(Operand<float> a, Operand<float> b, GemmArgs args, int sms, void* workspace, size_t workspace_bytes, double limit_cycles,
                        cudaStream_t st) {
  const size_t M = args.M, N = args.N, K = args.K;
  args.partial_ld = (args.N + 3) & ~3;
  size_t used = 0;
  auto job = [&](const Operand<float>& o, size_t rows, size_t cols) {
    TermsJob j;
    j.src = o.p;
    j.src_ld = o.ld;
    j.rows = static_cast<uint32_t>(rows);
    j.cols = static_cast<uint32_t>(cols);
    j.ld = up(cols, 8);
    for (auto& t : j.term) {
      t = reinterpret_cast<__nv_bfloat16*>(static_cast<unsigned char*>(workspace) + used);
      used += up(rows * j.ld * sizeof(__nv_bfloat16), 256);
    }
    j.vec = mp_aligned16(o.p) && o.ld % 4 == 0;
    j.blocks = static_cast<uint32_t>((rows * (j.ld / 4) + 255) / 256);
    return j;
  };
  if (static_cast<double>(M + N) * K * 6.0 > static_cast<double>(workspace_bytes)) return false;
  const TermsJob ja = args.a_mn ? job(a, K, M) : job(a, M, K), jb = args.b_mn ? job(b, K, N) : job(b, N, K);
  if (used > workspace_bytes) return false;
  const TermsPlan plan = terms_plan(args, sms, workspace_bytes - used);
  // the terms: 10 bytes an element at 2.5 KB a cycle
  if (plan.cycles + static_cast<double>(M + N) * K * 10.0 / 2500.0 > limit_cycles) return false;
  args.ksplit = plan.ksplit;
  args.partial = reinterpret_cast<float*>(static_cast<unsigned char*>(workspace) + used);
  MpLaunch(ja.blocks + jb.blocks, 256, 0, st)(r32_terms_kernel, ja, jb);
  MP_LAUNCH_CHECK();
  auto map = [&](const TermsJob& j, int t, int mn, uint32_t box) {   // (bf16 is moved as 16-bit words)
    return make_map<__half>(j.term[t], j.rows, j.cols, j.ld, H_BK, mn ? H_BK : box);
  };
  TermsMaps maps;
  for (int t = 0; t < 3; ++t) {
    maps.a[t] = map(ja, t, args.a_mn, BM);
    maps.b[t] = map(jb, t, args.b_mn, static_cast<uint32_t>(plan.bn / 2));
  }
  const Again again{a.p, b.p, a.ld, b.ld};
  if (plan.bn == 256) launch_terms<256>(maps, args, again, sms, st);
  else launch_terms<128>(maps, args, again, sms, st);
  if (args.ksplit > 1) {
    if (args.exact) launch_fold<float>(args, AgainFold{again, args.a_mn, args.b_mn, args.K}, st);
    else launch_fold<float>(args, NoAgain{}, st);
  }
  return true;
}
