// r32 contractions on the tensor cores: every product is three tf32 MMAs on an error-compensated split of the operands,
//     x = hi + lo,   hi = the 19 high bits of x (what kind::tf32 reads of a 32-bit word), lo = x - hi (exact),
//     a b ~ hi_a hi_b + hi_a lo_b + lo_a hi_b.
// The tensor core's fp32 accumulation truncates: a sum of K / 8 x 3 MMAs drifts by up to 2^-24 of its size per MMA (measured
// 1.5e-5 at K = 1001, growing with K).  The accumulator is therefore handed over every CHUNK_KB k-blocks (24 MMAs) to the
// epilogue warps, which add it up in registers with rounding; two TMEM accumulators take turns.
//
// EXACT: problems that were summed on the FP pipe before (padded operands) keep its exactness.  What the form above loses there is
// the product lo_a lo_b and lo's own last bits, both of which have the sign of a b when hi is x cut off (up to 2^-20 and 2^-21 of a
// product), and the truncated additions.  So hi is x rounded to the nearest instead (lo takes both signs, the losses average out),
// the small products of a k-block come before the large ones (only whose four additions then truncate at full size), and
// every k-block is handed over.  2-norm of the error at [301, K, 307], normal operands, K = 65 / 1001 / 16385: FP pipe 1.5e-7 / 5.7e-7 /
// 2.3e-6, this 1.3e-7 / 1.5e-7 / 1.9e-7, the form above 9.2e-7 throughout.  It costs the write of B's hi tile and twice the
// hand-overs: 4096^3 719 instead of 659 us, [2000, 999, 1501] with its copies 73 instead of 68.
//
// What bounds the kernel is shared memory bandwidth: three MMAs on operands there read every tile three times, which at 128
// columns takes as long as the MMAs themselves (126 of 128 bytes a cycle), and the split comes on top.  A is therefore kept in TMEM:
// the split warps read its tile once and write the raw words (hi: the MMA ignores the low bits) and lo there with tcgen05.st, so
// that the MMAs read only B from shared memory, and of B only the lo tile is written.  Beyond that the single warps' latencies per
// k-block count: the issuing warp walks its loop as a whole (elect_one), the split warps keep the next k-block's loads in flight.
// 4096^3: 820 us (three MMAs on shared-memory operands, 256 columns) -> 608 us; a CTA pair on a 256 x 128 tile took 940 us (every
// k-block's hand-offs then cross the pair).
//   warp 0      TMA producer (one elected thread)
//   warp 1      MMA issuer (one elected thread), owns the TMEM allocation
//   warps 2-5   A: raw and lo words to TMEM (warp w: lane quarter w % 4); warps 6-7: lo tile of B
//   warps 8-15  accumulation and epilogue: warp w reads TMEM lane quarter w % 4 and one half of the columns
#include "mp_gemm.cuh"

namespace {

constexpr int R_THREADS = 512;
constexpr int R_BK = 32;              // elements per 128-byte row
constexpr int R_UMMA_K = 8;
constexpr int R_SPLIT_WARPS = 6, R_SPLIT_B_FIRST = 6, R_SPLIT_B_THREADS = 64, R_EPI_FIRST = 8, R_EPI_WARPS = 8;
constexpr int R_SLOTS = 4, R_MAX_STAGES = 8;      // slots: split k-blocks (A in TMEM, lo tile of B in shared memory)
constexpr int R_BOX_BYTES = 32 * 32 * 4;
template <bool EXACT> constexpr int CHUNK_KB = EXACT ? 1 : 2;   // k-blocks per TMEM accumulation

template <int BN> struct R32Cfg {
  static constexpr int A_BYTES = BM * SWIZZLE_BYTES, B_BYTES = BN * SWIZZLE_BYTES;
  static constexpr int RAW = A_BYTES + B_BYTES;
  static constexpr int FIXED = R_SLOTS * B_BYTES + 1024 + R_EPI_WARPS * R_BOX_BYTES + 1024;   // lo tiles, barriers, staging, alignment
  static constexpr int STAGES = (232448 - FIXED) / RAW < R_MAX_STAGES ? (232448 - FIXED) / RAW : R_MAX_STAGES;
  static constexpr int SMEM = STAGES * RAW + FIXED;
  static constexpr uint32_t TM_A = 2 * BN;                            // TMEM: two accumulators, then 32 raw + 32 lo columns of A per slot
  static constexpr uint32_t TM_COLS = 512;
};

// Position of a work unit: unit = (batch entry or K split) * tiles + tile, tiles of one column of tiles next to each other
// (they share the B tile, which then stays in L2).
struct R32Unit { int m0, n0, bz, sp, kb0, kb1; };
template <int BN>
__device__ __forceinline__ R32Unit r32_unit(const GemmArgs& g, int unit, int tiles_m, int num_tiles, int num_kb, int kb_per) {
  R32Unit u;
  const int outer = unit / num_tiles, tile = unit - outer * num_tiles;
  const int tn = tile / tiles_m;
  u.m0 = (tile - tn * tiles_m) * BM;
  u.n0 = tn * BN;
  u.bz = g.batch > 1 ? outer : 0;
  u.sp = g.batch > 1 ? 0 : outer;
  u.kb0 = u.sp * kb_per;
  u.kb1 = min(num_kb, u.kb0 + kb_per);
  return u;
}

template <int BN, bool EXACT>
__global__ void __launch_bounds__(R_THREADS, 1) gemm_r32_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                                                                const __grid_constant__ CUtensorMap tmap_c, const GemmArgs g, const Again again) {
  using Cfg = R32Cfg<BN>;
  constexpr int A_BYTES = Cfg::A_BYTES, B_BYTES = Cfg::B_BYTES, RAW = Cfg::RAW, STAGES = Cfg::STAGES;
  extern __shared__ unsigned char gemm_smem_raw[];
  unsigned char* smem = mp_smem_align1024(gemm_smem_raw);
  unsigned char* lo_ring = smem + STAGES * RAW;
  uint64_t* full = reinterpret_cast<uint64_t*>(lo_ring + R_SLOTS * B_BYTES);   // loads have arrived
  uint64_t* raw_empty = full + R_MAX_STAGES;
  uint64_t* ready = raw_empty + R_MAX_STAGES;       // k-block split
  uint64_t* slot_empty = ready + R_SLOTS;
  uint64_t* acc_full = slot_empty + R_SLOTS;        // [2] accumulator of a chunk complete
  uint64_t* acc_empty = acc_full + 2;               // [2] taken over by the epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  unsigned char* epi_stage = lo_ring + R_SLOTS * B_BYTES + 1024;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int worker = blockIdx.x, workers = gridDim.x;
  const int num_kb = (g.K + R_BK - 1) / R_BK;
  const int tiles_m = (g.M + BM - 1) / BM, tiles_n = (g.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  const int num_units = num_tiles * g.ksplit * g.batch;
  const int kb_per = (num_kb + g.ksplit - 1) / g.ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full + s, 1); mbar_init(raw_empty + s, 1); }
    for (int l = 0; l < R_SLOTS; ++l) { mbar_init(ready + l, R_SPLIT_WARPS); mbar_init(slot_empty + l, 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(acc_full + a, 1); mbar_init(acc_empty + a, R_EPI_WARPS); }
    *abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_c);
  }
  if (warp == 1) tmem_alloc(tmem_slot, Cfg::TM_COLS);
  tcgen05_fence_before_sync();
  __syncthreads();
  tcgen05_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  mp_grid_wait();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int unit = worker; unit < num_units && ok; unit += workers) {
        const R32Unit u = r32_unit<BN>(g, unit, tiles_m, num_tiles, num_kb, kb_per);
        for (int kb = u.kb0; kb < u.kb1; ++kb) {
          if (!mbar_wait_abortable(raw_empty + s, phase ^ 1u, g.status, abort)) { ok = false; break; }
          unsigned char* sa = smem + s * RAW;
          unsigned char* sb = sa + A_BYTES;
          mbar_arrive_expect_tx(full + s, RAW);
          const int k0 = kb * R_BK;
          // K-major: one box {32 along K, rows}; MN-major: boxes {32 along M or N, 32 k-rows}
          auto load = [&](unsigned char* dst, const CUtensorMap* map, bool mn, int x0, int rows) {
            for (int j = 0; j < (mn ? rows / R_BK : 1); ++j) {
              const int x = mn ? x0 + j * R_BK : k0, y = mn ? k0 : x0;
              if (g.batch > 1) tma_load_3d(dst + j * (R_BK * SWIZZLE_BYTES), map, x, y, u.bz, full + s);
              else tma_load_2d(dst + j * (R_BK * SWIZZLE_BYTES), map, x, y, full + s);
            }
          };
          load(sa, &tmap_a, g.a_mn != 0, u.m0, BM);
          load(sb, &tmap_b, g.b_mn != 0, u.n0, BN);
          if (++s == STAGES) { s = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ----------------------------------
    const uint32_t idesc = umma_instr_desc(UMMA_FMT_TF32, 0, g.b_mn, BM, BN);
    // B K-major: rows of 128 B, 8-row groups 1024 B apart, k-slice = +32 B.  MN-major: k-rows of 128 B in the 32-byte-atom swizzle
    // (groups of 4 k-rows, 512 B), 32-column blocks 4 KB apart, k-slice = +8 k-rows.
    const uint32_t lbo = g.b_mn ? R_BK * SWIZZLE_BYTES : 16, kstep = g.b_mn ? R_UMMA_K * SWIZZLE_BYTES : 32;
    const uint32_t lay = g.b_mn ? UMMA_LAYOUT_SW128_BASE32B : UMMA_LAYOUT_SW128, sbo = g.b_mn ? 512 : 1024;
    // descriptors of stage / slot 0 and k-slice 0; the others differ in the address field (16-byte units)
    const uint64_t bd0 = umma_smem_desc(mp_smem_u32(smem) + A_BYTES, lbo, sbo, lay), ld0 = umma_smem_desc(mp_smem_u32(lo_ring), lbo, sbo, lay);
    const uint32_t kunits = kstep >> 4;
    const bool split = g.split != 0;
    int s = 0;
    uint32_t it = 0, chunk = 0;
    bool ok = true;
    for (int unit = worker; unit < num_units && ok; unit += workers) {
      const R32Unit u = r32_unit<BN>(g, unit, tiles_m, num_tiles, num_kb, kb_per);
      for (int kb = u.kb0; kb < u.kb1 && ok; kb += CHUNK_KB<EXACT>, ++chunk) {
        const uint32_t buf = chunk & 1u;
        ok = mbar_wait_abortable(acc_empty + buf, ((chunk >> 1) & 1u) ^ 1u, g.status, abort);
        ok = __all_sync(0xffffffffu, ok);
        const uint32_t acc = tmem_base + buf * BN;
        const int kend = min(kb + CHUNK_KB<EXACT>, u.kb1);
        for (int k = kb; ok && k < kend; ++k, ++it) {
          const uint32_t l = it % R_SLOTS;
          ok = mbar_wait_abortable(ready + l, (it / R_SLOTS) & 1u, g.status, abort);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tcgen05_fence_after_sync();
          const uint64_t bd = bd0 + static_cast<uint32_t>(s * (RAW >> 4)), ld = ld0 + l * (B_BYTES >> 4);
          const uint32_t ta = tmem_base + Cfg::TM_A + l * 64;
          const uint32_t first = k != kb ? 1u : 0u;
          if (elect_one()) {
            if constexpr (EXACT) {   // one k-block per accumulation
#pragma unroll
              for (int ks = 0; ks < R_BK / R_UMMA_K; ++ks) {
                umma_tf32_ta(acc, ta + 32 + ks * R_UMMA_K, bd + ks * kunits, idesc, ks != 0 ? 1u : 0u);   // lo * hi
                umma_tf32_ta(acc, ta + ks * R_UMMA_K, ld + ks * kunits, idesc, 1u);                       // hi * lo
              }
#pragma unroll
              for (int ks = 0; ks < R_BK / R_UMMA_K; ++ks) umma_tf32_ta(acc, ta + ks * R_UMMA_K, bd + ks * kunits, idesc, 1u);
            } else {
#pragma unroll
              for (int ks = 0; ks < R_BK / R_UMMA_K; ++ks) {
                umma_tf32_ta(acc, ta + ks * R_UMMA_K, bd + ks * kunits, idesc, ks != 0 ? 1u : first);
                if (split) {
                  umma_tf32_ta(acc, ta + 32 + ks * R_UMMA_K, bd + ks * kunits, idesc, 1u);   // lo * hi
                  umma_tf32_ta(acc, ta + ks * R_UMMA_K, ld + ks * kunits, idesc, 1u);        // hi * lo
                }
              }
            }
            umma_commit(raw_empty + s);
            umma_commit(slot_empty + l);
            if (k + 1 == kend) umma_commit(acc_full + buf);
          }
          __syncwarp();
          if (++s == STAGES) s = 0;
        }
      }
    }
    mp_launch_dependents();
  } else if (warp < R_EPI_FIRST) {
    // ------------------------------ split ---------------------------------------
    const bool does_b = warp >= R_SPLIT_B_FIRST;
    const int tb = threadIdx.x - 32 * R_SPLIT_B_FIRST;
    const int quarter = warp & 3, arow = quarter * 32 + lane;
    // hi in its 19 high bits.  A NaN may lose its own (rounding can carry out of the exponent), lo = NaN - hi remains one.
    auto high = [](uint32_t v) { return (EXACT ? v + 0x1000u : v) & 0xFFFFE000u; };
    auto low = [&](uint32_t v) { return __float_as_uint(__uint_as_float(v) - __uint_as_float(high(v))); };
    // k-blocks that this CTA splits, over all of its units (they run through the rings without a break)
    uint32_t total = 0;
    for (int unit = worker; unit < num_units; unit += workers) {
      const R32Unit u = r32_unit<BN>(g, unit, tiles_m, num_tiles, num_kb, kb_per);
      total += static_cast<uint32_t>(u.kb1 - u.kb0);
    }
    int s = 0;
    uint32_t phase = 0;
    auto blocking = [&](uint32_t it) {
      const bool ok = mbar_wait_abortable(full + s, phase, g.status, abort) &&
                      mbar_wait_abortable(slot_empty + it % R_SLOTS, ((it / R_SLOTS) & 1u) ^ 1u, g.status, abort);
      return __all_sync(0xffffffffu, ok) != 0;   // tcgen05.st is warp-collective
    };
    auto arrive = [&](uint32_t it) {
      __syncwarp();
      if (lane == 0) mbar_arrive(ready + it % R_SLOTS);
    };
    auto advance = [&]() { if (++s == STAGES) { s = 0; phase ^= 1u; } };
    if (does_b) {
      for (uint32_t it = 0; it < total; ++it, advance()) {
        if (!blocking(it)) break;
        unsigned char* src = smem + s * RAW + A_BYTES;
        unsigned char* dst = lo_ring + (it % R_SLOTS) * B_BYTES;
        constexpr int STEP = R_SPLIT_B_THREADS * 16, BATCH = 8;
#pragma unroll
        for (int base = 0; base < B_BYTES; base += BATCH * STEP) {   // loads of a batch first: the compiler cannot move them over stores
          uint4 v[BATCH];
#pragma unroll
          for (int e = 0; e < BATCH; ++e) v[e] = *reinterpret_cast<const uint4*>(src + base + e * STEP + tb * 16);
#pragma unroll
          for (int e = 0; e < BATCH; ++e) {
            *reinterpret_cast<uint4*>(dst + base + e * STEP + tb * 16) = make_uint4(low(v[e].x), low(v[e].y), low(v[e].z), low(v[e].w));
            if (EXACT) *reinterpret_cast<uint4*>(src + base + e * STEP + tb * 16) = make_uint4(high(v[e].x), high(v[e].y), high(v[e].z), high(v[e].w));
          }
        }
        fence_proxy_async_smem();   // the tensor core reads the tiles through the async proxy
        arrive(it);
      }
    } else if (total > 0) {
      auto load_row = [&](uint32_t* v) {
        const unsigned char* raw = smem + s * RAW;
        if (g.a_mn) {               // unswizzled blocks of 32 k-rows x 32 rows of A
          const uint32_t* src = reinterpret_cast<const uint32_t*>(raw + quarter * (R_BK * SWIZZLE_BYTES)) + lane;
#pragma unroll
          for (int k = 0; k < 32; ++k) v[k] = src[k * 32];
        } else {
#pragma unroll
          for (int p = 0; p < 8; ++p) {
            const uint4 q = *reinterpret_cast<const uint4*>(raw + arow * SWIZZLE_BYTES + ((p ^ (arow & 7)) << 4));
            v[4 * p] = q.x; v[4 * p + 1] = q.y; v[4 * p + 2] = q.z; v[4 * p + 3] = q.w;
          }
        }
      };
      // One warp takes its rows through every k-block, so the latencies of a k-block (barriers, shared-memory loads, TMEM stores)
      // would add up to more than its MMAs take: the next k-block's loads are issued before this one's stores are waited for,
      // where it has arrived already.
      uint32_t v[32], w[32];
      bool ok = blocking(0);
      if (ok) load_row(v);
      for (uint32_t it = 0; ok && it < total; ++it) {
        tcgen05_fence_after_sync();
        const uint32_t ta = tmem_base + Cfg::TM_A + (it % R_SLOTS) * 64 + (static_cast<uint32_t>(quarter * 32) << 16);
        if constexpr (EXACT) {
#pragma unroll
          for (int k = 0; k < 32; ++k) w[k] = high(v[k]);
          tmem_st_32x32(ta, w);
        } else {
          tmem_st_32x32(ta, v);   // the MMA ignores the low bits
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = low(v[k]);
        tmem_st_32x32(ta + 32, v);
        advance();
        const bool more = it + 1 < total;
        bool early = more && mbar_try_wait(full + s, phase) && mbar_try_wait(slot_empty + (it + 1) % R_SLOTS, (((it + 1) / R_SLOTS) & 1u) ^ 1u);
        early = __all_sync(0xffffffffu, early) != 0;
        if (early) load_row(w);
        tmem_st_wait();
        tcgen05_fence_before_sync();
        arrive(it);
        if (more && !early) {
          ok = blocking(it + 1);
          if (ok) load_row(w);
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = w[k];
      }
    }
  } else {
    // ------------------------------ accumulation and epilogue ---------------------
    constexpr int NB = BN / 64;                   // 32-column blocks per warp
    const int quarter = warp & 3, half = (warp - R_EPI_FIRST) >> 2;
    const float* bias = static_cast<const float*>(g.bias);
    const bool vec_ok = (g.ldc * sizeof(float)) % 16 == 0 && mp_aligned16(g.c);
    const bool use_tma = vec_ok && g.beta == 0.0f && g.ksplit == 1;
    float* stage = reinterpret_cast<float*>(epi_stage + (warp - R_EPI_FIRST) * R_BOX_BYTES);
    uint32_t chunk = 0;
    bool ok = true;
    for (int unit = worker; unit < num_units && ok; unit += workers) {
      const R32Unit u = r32_unit<BN>(g, unit, tiles_m, num_tiles, num_kb, kb_per);
      float acc[NB][32];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[nb][j] = 0.f;
      for (int kb = u.kb0; kb < u.kb1; kb += CHUNK_KB<EXACT>, ++chunk) {
        const uint32_t buf = chunk & 1u;
        ok = mbar_wait_abortable(acc_full + buf, (chunk >> 1) & 1u, g.status, abort);
        ok = __all_sync(0xffffffffu, ok);   // tcgen05.ld is warp-collective
        if (!ok) break;
        tcgen05_fence_after_sync();
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
          uint32_t v[32];
          tmem_ld_32x32(tmem_base + buf * BN + (static_cast<uint32_t>(quarter * 32) << 16) + half * (BN / 2) + nb * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[nb][j] += __uint_as_float(v[j]);
        }
        tcgen05_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty + buf);
      }
      if (!ok) break;
      const int row0 = u.m0 + quarter * 32, row = row0 + lane;
      float* c0 = static_cast<float*>(g.c) + (static_cast<size_t>(u.bz) * g.M + row0) * g.ldc;
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        const int col0 = u.n0 + half * (BN / 2) + nb * 32;
        if (col0 < g.N) {   // uniform across the warp
          float* r = acc[nb];
          if (g.ksplit > 1) {   // raw partial sums; alpha, bias and beta are applied by the fold
            if (row < g.M) {
              float* prow = g.partial + (static_cast<size_t>(u.sp) * g.M + row) * g.partial_ld + col0;
              if (col0 + 32 <= g.N) {
#pragma unroll
                for (int p = 0; p < 8; ++p) *reinterpret_cast<float4*>(prow + p * 4) = make_float4(r[p * 4], r[p * 4 + 1], r[p * 4 + 2], r[p * 4 + 3]);
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (col0 + j < g.N) prow[j] = r[j];
              }
            }
          } else {
            const bool by_rows = !use_tma && !(vec_ok && col0 + 32 <= g.N);
            if constexpr (EXACT) {
              bool nan = false;
#pragma unroll
              for (int j = 0; j < 32; ++j) nan = nan || r[j] != r[j];
              if (__any_sync(0xffffffffu, nan)) {   // rare; the block goes through the staging, so that its elements can be walked by index
                if (lane == 0) bulk_wait_read<0>();
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 32; ++j) stage[j * 32 + lane] = r[j];
#pragma unroll 1
                for (int j = 0; j < 32; ++j)
                  if (row < g.M && col0 + j < g.N && stage[j * 32 + lane] != stage[j * 32 + lane]) stage[j * 32 + lane] = again(g, u.bz, row, col0 + j);
#pragma unroll
                for (int j = 0; j < 32; ++j) r[j] = stage[j * 32 + lane];
                __syncwarp();
              }
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) r[j] *= g.alpha;
            if (bias != nullptr && (g.bias_pitch == 0 || (row < g.M && !by_rows))) {
              const float* brow = bias + static_cast<size_t>(row) * g.bias_pitch;
              if (col0 + 32 <= g.N && g.bias_pitch % 4 == 0 && mp_aligned16(bias)) {
#pragma unroll
                for (int p = 0; p < 8; ++p) {
                  const float4 add = *reinterpret_cast<const float4*>(brow + col0 + 4 * p);
                  r[4 * p] += add.x; r[4 * p + 1] += add.y; r[4 * p + 2] += add.z; r[4 * p + 3] += add.w;
                }
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (col0 + j < g.N) r[j] += brow[col0 + j];
              }
            }
            if (use_tma) {
              if (lane == 0) bulk_wait_read<0>();   // the previous store has read the box
              __syncwarp();
#pragma unroll
              for (int p = 0; p < 8; ++p)   // 128-byte rows in the 128-byte swizzle
                *reinterpret_cast<float4*>(stage + lane * 32 + ((p ^ (lane & 7)) << 2)) = make_float4(r[p * 4], r[p * 4 + 1], r[p * 4 + 2], r[p * 4 + 3]);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                if (g.batch > 1) tma_store_3d(&tmap_c, stage, col0, row0, u.bz);
                else tma_store_2d(&tmap_c, stage, col0, row0);
                bulk_commit();
              }
            } else if (by_rows) {
              store_block_rows<float>(stage, r, lane, c0 + col0, g.ldc, min(32, g.M - row0), col0 + lane < g.N,
                                      bias != nullptr && g.bias_pitch != 0 ? bias + static_cast<size_t>(row0) * g.bias_pitch + col0 : nullptr,
                                      g.bias_pitch, g.beta);
            } else if (row < g.M) {
              float4* crow = reinterpret_cast<float4*>(c0 + lane * g.ldc + col0);
#pragma unroll
              for (int p = 0; p < 8; ++p) {
                const float4 o = crow[p];
                crow[p] = make_float4(r[p * 4] + g.beta * o.x, r[p * 4 + 1] + g.beta * o.y, r[p * 4 + 2] + g.beta * o.z, r[p * 4 + 3] + g.beta * o.w);
              }
            }
          }
        }
      }
    }
    if (use_tma && lane == 0) bulk_wait_all<0>();
  }
  __syncwarp();
  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, Cfg::TM_COLS);
}

template <int BN, bool EXACT>
void launch_r32(Operand<float> a, Operand<float> b, const GemmArgs& g, int sms, cudaStream_t st) {
  using Cfg = R32Cfg<BN>;
  const size_t nb = static_cast<size_t>(g.batch);
  const CUtensorMap ta = g.a_mn ? make_map<float>(a.p, g.K, g.M, a.ld, R_BK, R_BK, CU_TENSOR_MAP_SWIZZLE_NONE, nb) : make_map<float>(a.p, g.M, g.K, a.ld, R_BK, BM, CU_TENSOR_MAP_SWIZZLE_128B, nb);
  const CUtensorMap tb = g.b_mn ? make_map<float>(b.p, g.K, g.N, b.ld, R_BK, R_BK, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, nb) : make_map<float>(b.p, g.N, g.K, b.ld, R_BK, BN, CU_TENSOR_MAP_SWIZZLE_128B, nb);
  CUtensorMap tc = ta;
  if ((g.ldc * sizeof(float)) % 16 == 0 && mp_aligned16(g.c)) tc = make_store_map<float>(g.c, g.M, g.N, g.ldc, false, nb);
  MP_CUDA_CHECK(cudaFuncSetAttribute(gemm_r32_kernel<BN, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM));
  const long units = static_cast<long>((g.N + BN - 1) / BN) * ((g.M + BM - 1) / BM) * g.ksplit * g.batch;
  const Again again{a.p, b.p, a.ld, b.ld};
  MpLaunch(static_cast<unsigned>(units < sms ? units : sms), R_THREADS, Cfg::SMEM, st)(gemm_r32_kernel<BN, EXACT>, ta, tb, tc, g, again);
  MP_LAUNCH_CHECK();
  if (g.ksplit > 1) {
    if (EXACT) launch_fold<float>(g, AgainFold{again, g.a_mn, g.b_mn, g.K}, st);
    else launch_fold<float>(g, NoAgain{}, st);
  }
}

}  // namespace

// The tile (128 x 128 or 128 x 64) and the number of K splits with the smallest estimate of
//     waves over the SMs x (k-blocks per unit x cycles per k-block + cycles to fill and to drain a unit)  [+ the fold]
// with the cycles per k-block measured at 4096^3 (1330 and 890).
double gemm_r32_estimate(const GemmArgs& args, int sms, size_t workspace_bytes, int* bn, int* ksplit) {
  const long num_kb = (args.K + R_BK - 1) / R_BK;
  const double mn_bytes = static_cast<double>(args.M) * ((args.N + 3) & ~3) * 4.0;
  const bool may_split = args.batch == 1 && !env_flag("MP_GEMM_NO_SPLITK");
  double best = 1e300;
  for (int width = 128; width >= 64; width /= 2) {
    const double cycles = width == 128 ? 1330.0 : 890.0;
    const long n_tiles = static_cast<long>((args.M + BM - 1) / BM) * ((args.N + width - 1) / width) * args.batch;
    for (int ks = 1; ks <= (may_split ? 32 : 1); ++ks) {
      const long per = (num_kb + ks - 1) / ks;
      if (ks > 1 && (per < 2 || (ks - 1) * per >= num_kb || ks * mn_bytes > static_cast<double>(workspace_bytes))) continue;
      double cost = static_cast<double>((n_tiles * ks + sms - 1) / sms) * (per * cycles + 3000.0);
      if (ks > 1) cost += 5000.0 + 2.0 * ks * mn_bytes / 3500.0;   // the fold's launch; partials out and in at 3.5 KB a cycle
      if (cost < best) { best = cost; *bn = width; *ksplit = ks; }
    }
  }
  return best;
}

void gemm_run_r32(Operand<float> a, Operand<float> b, GemmArgs args, int sms, void* workspace, size_t workspace_bytes, cudaStream_t st) {
  args.partial_ld = (args.N + 3) & ~3;
  args.partial = static_cast<float*>(workspace);
  int bn = 128;
  gemm_r32_estimate(args, sms, workspace_bytes, &bn, &args.ksplit);
  const bool exact = args.exact != 0 && args.split != 0;
  if (bn == 128) {
    if (exact) launch_r32<128, true>(a, b, args, sms, st); else launch_r32<128, false>(a, b, args, sms, st);
  } else {
    if (exact) launch_r32<64, true>(a, b, args, sms, st); else launch_r32<64, false>(a, b, args, sms, st);
  }
}
