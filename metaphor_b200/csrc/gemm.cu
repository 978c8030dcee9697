// Contractions C[M,N] = alpha * op(A) * op(B) (+ bias) + beta * C, row-major.
//
//   launch_inner_product_ij_jk_ik : A[M,K]      B[K,N]       (reference: cuBLAS via
//                                                             inner_product_ij_jk_ik.cu:3-27)
//   launch_inner_product_ij_kj_ik : A[M,K]      B[N,K]^T     (reference: transpose to
//   launch_inner_product_ji_jk_ik : A[K,M]^T    B[K,N]        scratch + the call above)
//   launch_linear_ij_jk_ik        : A[M,K]      B[K,N] + bias[N]
//   launch_linear_ij_jk_ik_ik     : A[M,K]      B[K,N] + R[M,N]
//
// r16 and r32 run on the tcgen05 tensor cores: operand tiles are brought into
// 128-byte-swizzled shared memory by TMA (one warp's elected thread), a single
// thread issues tcgen05.mma with the fp32 accumulator tile in TMEM, and four
// epilogue warps read the accumulator back with tcgen05.ld and apply alpha,
// beta, bias on the way to global memory.  The kernel is persistent (one CTA per
// SM walking the output tiles) with two TMEM accumulators, so one tile's
// epilogue overlaps the next tile's main loop.  Transposed operands need no scratch
// copy: the shared-memory descriptor and the instruction descriptor carry the
// operand's major-ness.  r32 has a kernel of its own (gemm_r32.cu: three tf32 MMAs per
// product on an error-compensated split).  Operands TMA cannot address
// (row pitch not a multiple of 16 bytes) are copied into aligned rows first; r64 and
// those of them with a short K use an FP-pipe tile kernel.
#include "mp_gemm.cuh"

namespace {

// ---------------------------------------------------------------------------
// SIMT tile kernel: any dtype, any shape.  64x64 output tile, 16-deep k-slices
// through shared memory, 4x4 outputs per thread, accumulation in Acc<T>.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const T* __restrict__ a, const T* __restrict__ b,
                                                        const T* __restrict__ bias, typename Acc<T>::type alpha, T* c,
                                                        typename Acc<T>::type beta, size_t M, size_t N, size_t K, int a_mn,
                                                        int b_mn, size_t bias_pitch) {
  mp_grid_dependency();
  using A = typename Acc<T>::type;
  constexpr int TS = 64, KS = 16;
  a += static_cast<size_t>(blockIdx.z) * M * K;   // batch entries are densely packed
  b += static_cast<size_t>(blockIdx.z) * K * N;
  c += static_cast<size_t>(blockIdx.z) * M * N;
  __shared__ A sa[KS][TS + 1];
  __shared__ A sb[KS][TS + 1];
  const size_t m0 = static_cast<size_t>(blockIdx.y) * TS, n0 = static_cast<size_t>(blockIdx.x) * TS;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  A acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = A(0);
  for (size_t k0 = 0; k0 < K; k0 += KS) {
    for (int idx = threadIdx.x; idx < TS * KS; idx += 256) {
      // A element (m, k): a_mn ? a[k*M + m] : a[m*K + k]
      int kk, mm;
      if (a_mn) { mm = idx % TS; kk = idx / TS; } else { kk = idx % KS; mm = idx / KS; }
      const size_t gm = m0 + mm, gk = k0 + kk;
      sa[kk][mm] = (gm < M && gk < K) ? mp_up(a_mn ? a[gk * M + gm] : a[gm * K + gk]) : A(0);
      int kb, nb;
      if (b_mn) { nb = idx % TS; kb = idx / TS; } else { kb = idx % KS; nb = idx / KS; }
      const size_t gn = n0 + nb, gkb = k0 + kb;
      sb[kb][nb] = (gn < N && gkb < K) ? mp_up(b_mn ? b[gkb * N + gn] : b[gn * K + gkb]) : A(0);
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
      A av[4], bv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) av[i] = sa[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) bv[j] = sb[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += av[i] * bv[j];
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const size_t gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const size_t gn = n0 + tx * 4 + j;
      if (gn >= N) continue;
      A r = alpha * acc[i][j];
      if (bias != nullptr) r += mp_up(bias[gm * bias_pitch + gn]);
      if (beta != A(0)) r += beta * mp_up(c[gm * N + gn]);
      c[gm * N + gn] = mp_down<T>(r);
    }
  }
}

// ---------------------------------------------------------------------------
// tcgen05 kernel.
// ---------------------------------------------------------------------------
constexpr int GEMM_THREADS = 320;     // warp 0: TMA, warp 1: MMA + TMEM, warps 2-9: epilogue
constexpr int EPI_THREADS = 256;      // two epilogue warps per TMEM lane quarter, each takes half of the columns
constexpr int MAX_STAGES = 8;

// 32-column staging blocks per epilogue warp: one per block of the warp's half tile (4 at BN = 256), so a tile's TMA stores are
// issued back to back and the staging is only waited for at the next tile.
constexpr int EPI_BUFS = 4;

struct GemmT {
  static constexpr int BK = 64;       // elements per 128-byte row
  static constexpr int UMMA_K = 16;
};

template <int BN> constexpr int stage_bytes() { return BM * SWIZZLE_BYTES + BN * SWIZZLE_BYTES; }

// Persistent kernel: grid = min(tiles, SMs); every CTA walks output tiles
// t = blockIdx.x, blockIdx.x + gridDim.x, ... (consecutive tiles share the B
// tile, which therefore stays in L2).  The shared-memory ring runs across tile
// boundaries and there are two TMEM accumulators, so the epilogue of tile i
// (tcgen05.ld -> registers -> global) overlaps the main loop of tile i+1.
//   warp 0      TMA producer (one elected thread)
//   warp 1      MMA issuer (one elected thread), owns the TMEM allocation
//   warps 2-9   epilogue: warp w reads TMEM lane quarter w % 4 and one half of the tile's columns;
//               32x32 blocks go registers -> shared staging -> TMA store (coalesced, edge-clipped)
//
// EXACT: the tensor core's fp32 accumulation truncates, which drifts by up to 2^-24 of the sum per MMA.  Problems that were
// summed on the FP pipe before (padded operands) keep its exactness: the accumulator is handed over every CHUNK_KB k-blocks
// (8 MMAs) and added up in the epilogue warps' registers with rounding.  That leaves the pair kernel out.  Results that are not the r16
// nearest to the exact sum, operands of one sign, [5001, 4097, 5001]: 0.1 % on the FP pipe, 0.07 % here, 3.4 % with the pair kernel; times
// 9 733, 431 and 317 us.
constexpr int CHUNK_KB = 2;
template <int BN, bool EXACT>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a,
                                                                      const __grid_constant__ CUtensorMap tmap_b,
                                                                      const __grid_constant__ CUtensorMap tmap_c, const GemmArgs g) {
  using T = __half;
  using G = GemmT;
  constexpr int BK = G::BK;
  constexpr int A_BYTES = BM * SWIZZLE_BYTES, B_BYTES = BN * SWIZZLE_BYTES;
  constexpr int KSLICES = BK / G::UMMA_K;  // 4
  constexpr int ACC_BUFS = 2;
  constexpr int EPI_TILE_BYTES = 32 * 32 * sizeof(T);   // one 32 x 32 staging block for the TMA store
  // BN >= 128: two 32-column blocks share one [32 rows][64 columns] staging box in the 128-byte swizzle,
  // written out by one TMA store with full 128-byte rows (64-byte rows halve the store engine's throughput)
  constexpr bool WIDE_STORE = BN >= 128;
  extern __shared__ unsigned char gemm_smem_raw[];
  // 1024-byte alignment: swizzle atoms are 8 rows x 128 bytes
  unsigned char* smem = mp_smem_align1024(gemm_smem_raw);
  const int stages = g.stages;
  constexpr int stage_sz = A_BYTES + B_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(stages) * stage_sz);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* acc_full = empty + MAX_STAGES;  // [2] accumulator complete
  uint64_t* acc_empty = acc_full + ACC_BUFS;  // [2] accumulator drained by the epilogue
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + ACC_BUFS);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  unsigned char* epi_stage = smem + static_cast<size_t>(stages) * stage_sz + 1024;   // 8 warps x EPI_BUFS x EPI_TILE_BYTES, 1024-aligned

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_kb = (g.K + BK - 1) / BK;
  const int tiles_m = (g.M + BM - 1) / BM, tiles_n = (g.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  // work unit u = (tile u % num_tiles, K split u / num_tiles) covering k-blocks [kb0, kb1)
  // batched: unit = batch entry * num_tiles + tile (ksplit is 1)
  const int num_units = num_tiles * g.ksplit * g.batch;
  const int kb_per = (num_kb + g.ksplit - 1) / g.ksplit;
  const bool batched = g.batch > 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(full + s, 1);
      mbar_init(empty + s, 1);
    }
    for (int a = 0; a < ACC_BUFS; ++a) { mbar_init(acc_full + a, 1); mbar_init(acc_empty + a, EPI_THREADS); }
    *abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_c);
  }
  if (warp == 1) tmem_alloc(tmem_slot, ACC_BUFS * BN);
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
      for (int unit = blockIdx.x; unit < num_units && ok; unit += gridDim.x) {
        const int bz = batched ? unit / num_tiles : 0;
        const int tile = batched ? unit - bz * num_tiles : unit % num_tiles, sp = batched ? 0 : unit / num_tiles;
        const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * BN;
        const int kb0 = sp * kb_per, kb1 = min(num_kb, kb0 + kb_per);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_abortable(empty + s, phase ^ 1u, g.status, abort)) { ok = false; break; }
          unsigned char* sa = smem + static_cast<size_t>(s) * stage_sz;
          unsigned char* sb = sa + A_BYTES;
          mbar_arrive_expect_tx(full + s, A_BYTES + B_BYTES);
          const int k0 = kb * BK;
          if (batched) {   // the same boxes over 3-D maps
            if (!g.a_mn) {
              tma_load_3d(sa, &tmap_a, k0, m0, bz, full + s);
            } else {
#pragma unroll 1
              for (int j = 0; j < BM / BK; ++j) tma_load_3d(sa + j * (BK * SWIZZLE_BYTES), &tmap_a, m0 + j * BK, k0, bz, full + s);
            }
            if (!g.b_mn) {
              tma_load_3d(sb, &tmap_b, k0, n0, bz, full + s);
            } else {
#pragma unroll 1
              for (int j = 0; j < BN / BK; ++j) tma_load_3d(sb + j * (BK * SWIZZLE_BYTES), &tmap_b, n0 + j * BK, k0, bz, full + s);
            }
          } else {
            if (!g.a_mn) {
              tma_load_2d(sa, &tmap_a, k0, m0, full + s);            // box {BK, BM}
            } else {
#pragma unroll 1
              for (int j = 0; j < BM / BK; ++j)                        // boxes {BK along M, BK k-rows}
                tma_load_2d(sa + j * (BK * SWIZZLE_BYTES), &tmap_a, m0 + j * BK, k0, full + s);
            }
            if (!g.b_mn) {
              tma_load_2d(sb, &tmap_b, k0, n0, full + s);            // box {BK, BN}
            } else {
#pragma unroll 1
              for (int j = 0; j < BN / BK; ++j)
                tma_load_2d(sb + j * (BK * SWIZZLE_BYTES), &tmap_b, n0 + j * BK, k0, full + s);
            }
          }
          if (++s == stages) { s = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (the warp as a whole, see elect_one) ----
    const uint32_t idesc = umma_instr_desc(UMMA_FMT_F16, g.a_mn, g.b_mn, BM, BN);
    // K-major: rows of 128 B, 8-row groups 1024 B apart, k-slice = +32 B.
    // MN-major: k-rows of 128 B, 64-column blocks BK*128 B apart, k-slice = +UMMA_K*128 B.
    const uint32_t a_lbo = g.a_mn ? BK * SWIZZLE_BYTES : 16, b_lbo = g.b_mn ? BK * SWIZZLE_BYTES : 16;
    const uint32_t a_kunits = (g.a_mn ? G::UMMA_K * SWIZZLE_BYTES : 32) >> 4, b_kunits = (g.b_mn ? G::UMMA_K * SWIZZLE_BYTES : 32) >> 4;
    // descriptors of stage 0, k-slice 0; the others differ in the address field (16-byte units)
    const uint64_t ad0 = umma_smem_desc(mp_smem_u32(smem), a_lbo, 1024), bd0 = umma_smem_desc(mp_smem_u32(smem) + A_BYTES, b_lbo, 1024);
    int s = 0;
    uint32_t phase = 0, chunk = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < num_units && ok; unit += gridDim.x) {
      const int sp = batched ? 0 : unit / num_tiles;
      const int kb0 = sp * kb_per, kb1 = min(num_kb, kb0 + kb_per);
      for (int kc = kb0; kc < kb1 && ok; ++chunk) {
        const int kend = EXACT ? min(kb1, kc + CHUNK_KB) : kb1;
        const uint32_t buf = chunk & 1u;
        // the epilogue must have drained this accumulator (passes at once on its first use)
        ok = mbar_wait_abortable(acc_empty + buf, ((chunk >> 1) & 1u) ^ 1u, g.status, abort);
        ok = __all_sync(0xffffffffu, ok);
        const uint32_t tmem_acc = tmem_base + buf * BN;
        for (int kb = kc; ok && kb < kend; ++kb) {
          ok = mbar_wait_abortable(full + s, phase, g.status, abort);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tcgen05_fence_after_sync();
          const uint64_t ad = ad0 + static_cast<uint32_t>(s * (stage_sz >> 4)), bd = bd0 + static_cast<uint32_t>(s * (stage_sz >> 4));
          const uint32_t first = kb != kc ? 1u : 0u;
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < KSLICES; ++ks) umma<false>(tmem_acc, ad + ks * a_kunits, bd + ks * b_kunits, idesc, ks != 0 ? 1u : first);
            umma_commit(empty + s);  // the stage may be refilled once these MMAs have read it
            if (kb + 1 == kend) umma_commit(acc_full + buf);
          }
          __syncwarp();
          if (++s == stages) { s = 0; phase ^= 1u; }
        }
        kc = kend;
      }
    }
    mp_launch_dependents();
  } else {
    // ------------------------------ epilogue -----------------------------------
    const int quarter = warp & 3;                 // TMEM lanes this warp may read
    const int half = (warp - 2) >> 2;             // which half of the tile's columns
    const T* bias = static_cast<const T*>(g.bias);
    const bool vec_ok = (g.ldc * sizeof(T)) % 16 == 0 && mp_aligned16(g.c);
    const bool use_tma = vec_ok && g.beta == 0.0f && g.ksplit == 1;   // overwrite: stage 32x32 blocks and let TMA write them
    unsigned char* stage_base = epi_stage + (warp - 2) * (EPI_BUFS * EPI_TILE_BYTES);
    constexpr int BLOCKS = BN / 64;   // 32-column blocks of a warp's half tile
    const uint32_t tmem_lane = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * (BN / 2);
    uint32_t chunk = 0;
    bool ok = true;
    // hands an accumulator back to the MMA warp
    auto release = [&]() {
      tcgen05_fence_before_sync();
      mbar_arrive(acc_empty + (chunk & 1u));
      ++chunk;
    };
    auto acquire = [&]() {   // tcgen05.ld is warp-collective
      const bool ready = mbar_wait_abortable(acc_full + (chunk & 1u), (chunk >> 1) & 1u, g.status, abort);
      ok = __all_sync(0xffffffffu, ready) != 0;
      tcgen05_fence_after_sync();
      return ok;
    };
    for (int unit = blockIdx.x; unit < num_units; unit += gridDim.x) {
      const int bz = batched ? unit / num_tiles : 0;
      const int tile = batched ? unit - bz * num_tiles : unit % num_tiles, sp = batched ? 0 : unit / num_tiles;
      const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * BN;
      float sum[EXACT ? BLOCKS : 1][32];
      if constexpr (EXACT) {
#pragma unroll
        for (int q = 0; q < BLOCKS; ++q)
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[q][j] = 0.f;
        const int kb0 = sp * kb_per, kb1 = min(num_kb, kb0 + kb_per);
        for (int kc = kb0; kc < kb1 && acquire(); kc += CHUNK_KB) {
#pragma unroll
          for (int q = 0; q < BLOCKS; ++q) {
            uint32_t v[32];
            tmem_ld_32x32(tmem_lane + (chunk & 1u) * BN + q * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) sum[q][j] += __uint_as_float(v[j]);
          }
          release();
        }
      } else {
        acquire();
      }
      if (!ok) break;
      const uint32_t tmem_acc = tmem_lane + (chunk & 1u) * BN;
      const int row = m0 + quarter * 32 + lane;
      T* crow = static_cast<T*>(g.c) + (static_cast<size_t>(bz) * g.M + row) * g.ldc;
#pragma unroll(EXACT ? BLOCKS : 1)
      for (int blk = 0; blk < BLOCKS; ++blk) {
        const int col0 = n0 + half * (BN / 2) + blk * 32;
        if (col0 >= g.N) break;   // uniform across the warp
        unsigned char* stage = stage_base + (blk % EPI_BUFS) * EPI_TILE_BYTES;
        uint32_t v[32];
        if constexpr (EXACT) {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(sum[blk][j]);
        } else {
          tmem_ld_32x32(tmem_acc + blk * 32, v);
          tmem_ld_wait();
        }
        if (g.ksplit > 1) {   // raw partial sums; alpha, bias and beta are applied by the fold
          if (row < g.M) {
            float* prow = g.partial + (static_cast<size_t>(sp) * g.M + row) * g.partial_ld + col0;
            if (col0 + 32 <= g.N) {
#pragma unroll
              for (int p = 0; p < 8; ++p) *reinterpret_cast<uint4*>(prow + p * 4) = make_uint4(v[p * 4], v[p * 4 + 1], v[p * 4 + 2], v[p * 4 + 3]);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + j < g.N) prow[j] = __uint_as_float(v[j]);
            }
          }
          continue;
        }
        float r[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = g.alpha * __uint_as_float(v[j]);
        const bool by_rows = !use_tma && !(vec_ok && col0 + 32 <= g.N);   // store_block_rows; it adds a matrix term itself
        if (bias != nullptr && (g.bias_pitch == 0 || (row < g.M && !by_rows))) {
          const T* brow = bias + static_cast<size_t>(row) * g.bias_pitch;
          if (col0 + 32 <= g.N && (g.bias_pitch * sizeof(T)) % 16 == 0 && mp_aligned16(bias)) {
            // the lane's 32 values in four loads ([512, 512] x [512, 256] with a residual, one at a time / so: 15.2 / 7.1 us)
            constexpr int PN = Pack<T>::N;
#pragma unroll
            for (int p = 0; p < 32 / PN; ++p) {
              float add[PN];
              unpack<T>(ld_pack(brow + col0, p), add);
#pragma unroll
              for (int e = 0; e < PN; ++e) r[p * PN + e] += add[e];
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (col0 + j < g.N) r[j] += mp_up(brow[col0 + j]);
          }
        }
        if (use_tma) {
          constexpr int PN = Pack<T>::N;
          if constexpr (WIDE_STORE) {
            if (blk == 0) {   // the previous tile's stores have finished reading the staging boxes
              if (lane == 0) bulk_wait_read<0>();
              __syncwarp();
            }
            const int in_box = blk & 1;
            unsigned char* box = stage_base + (blk >> 1) * (2 * EPI_TILE_BYTES);
#pragma unroll
            for (int p = 0; p < 4; ++p)   // 16-byte chunk (4 in_box + p) of this lane's 128-byte row, XOR-swizzled
              *reinterpret_cast<Pack<T>*>(box + lane * 128 + (((4 * in_box + p) ^ (lane & 7)) << 4)) = pack<T>(r + p * PN);
            if (in_box == 1 || col0 + 32 >= g.N) {   // box complete (columns past N are clipped by the store)
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                if (batched) tma_store_3d(&tmap_c, box, col0 - 32 * in_box, m0 + quarter * 32, bz);
                else tma_store_2d(&tmap_c, box, col0 - 32 * in_box, m0 + quarter * 32);
                bulk_commit();
              }
            }
            continue;
          }
          // the store that last used this staging block has finished reading it
          if (lane == 0) { if (blk < EPI_BUFS) { if (blk == 0) bulk_wait_read<0>(); } else bulk_wait_read<EPI_BUFS - 1>(); }
          __syncwarp();
          // BN = 64: linear 64-byte rows
          unsigned char* srow = stage + lane * (32 * sizeof(T));
#pragma unroll
          for (int p = 0; p < 32 / PN; ++p) *reinterpret_cast<Pack<T>*>(srow + p * 16) = pack<T>(r + p * PN);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (batched) tma_store_3d(&tmap_c, stage, col0, m0 + quarter * 32, bz);
            else tma_store_2d(&tmap_c, stage, col0, m0 + quarter * 32);
            bulk_commit();
          }
        } else if (by_rows && g.beta == 0.0f && (bias == nullptr || g.bias_pitch == 0)) {   // (nothing is aligned: all blocks come here)
          uint32_t* words = reinterpret_cast<uint32_t*>(stage_base);
          stage_half_words(words, r, lane, blk & 1);
          if ((blk & 1) != 0 || blk + 1 == BLOCKS || col0 + 32 >= g.N) {
            const int row0 = m0 + quarter * 32, colb = col0 - 32 * (blk & 1);
            store_half_rows(words, lane, crow - static_cast<size_t>(lane) * g.ldc + colb, g.ldc, min(32, g.M - row0),
                            min(32 * (blk & 1) + 32, g.N - colb));
          }
        } else if (by_rows) {
          const int row0 = m0 + quarter * 32;
          store_block_rows<T>(reinterpret_cast<float*>(stage_base), r, lane, crow - static_cast<size_t>(lane) * g.ldc + col0, g.ldc,
                              min(32, g.M - row0), col0 + lane < g.N,
                              bias != nullptr && g.bias_pitch != 0 ? bias + static_cast<size_t>(row0) * g.bias_pitch + col0 : nullptr, g.bias_pitch,
                              g.beta);
        } else if (row < g.M) {
          constexpr int PN = Pack<T>::N;
          if (g.beta != 0.0f) {
#pragma unroll
            for (int p = 0; p < 32 / PN; ++p) {
              float old[PN];
              unpack<T>(ld_pack(crow + col0, p), old);
#pragma unroll
              for (int e = 0; e < PN; ++e) r[p * PN + e] += g.beta * old[e];
            }
          }
#pragma unroll
          for (int p = 0; p < 32 / PN; ++p) st_pack(crow + col0, p, pack<T>(r + p * PN));
        }
      }
      if constexpr (!EXACT) release();
    }
    if (use_tma && lane == 0) bulk_wait_all<0>();   // all of this warp's stores have completed
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, ACC_BUFS * BN);
}


// ---------------------------------------------------------------------------
// CTA-pair kernel (r16): a cluster of two CTAs owns a 256 x 256 output tile.  Rank r loads its 128 rows of
// A and columns [128 r, 128 r + 128) of B, so every CTA moves 32 KB per 64-deep k-block for a 128 x 256
// accumulator instead of 48 KB: the single-CTA kernel is bound by the L2 -> shared-memory feed, not by the
// tensor pipe (measured 1.25-1.7 k cycles per k-block against 0.5 k at the tensor peak).
//   both ranks  warp 0: TMA producer; warps 2-9: epilogue of the rank's own 128 rows
//   rank 0      warp 1: issues the pair MMAs, commits to its own barriers
// Barriers live at the same offsets in both CTAs.  full[s]: rank 0 only, credited by both ranks' loads.
// empty[s] / acc_full[b]: the MMA commit arrives on both CTAs' barriers (tcgen05.commit to a CTA mask).
// acc_empty[b]: rank 0 only, one arrival per epilogue warp of both ranks.  Every wait is bounded and suspends between
// polls: polling the ring barriers without a suspend hint (as the scan's chunk walk does) made every shape 5 - 8 % slower.
// ---------------------------------------------------------------------------
constexpr int PAIR_BN = 256;
// Tiles in the order of their rows, column by column: the pairs at work share a tile of B and read all of A once per column.  Where A does not
// stay in the L2 that long, eight row blocks at a time: A is read once, B once per group.  us, all rows / eight at a time: [16384, 3352] x
// [3352, 768] 88 / 81, [16384, 50280] x [50280, 768] 1196 / 1058, 8192^3 891 / 818 (24 at a time: 82, 1071, 862); where A takes 25 - 50 MB
// the two are level or all rows are ahead ([16384, 768] x [768, 3352] 84.8 / 84.6, [16384, 768] x [768, 50280] 1042 / 1074).
constexpr int PAIR_GROUP = 8;
constexpr double PAIR_GROUP_BYTES = 64e6;   // half of the L2
__device__ __forceinline__ void pair_tile(const GemmArgs& g, int tile, int tiles_m, int tiles_n, int& tm, int& tn) {
  if (g.group == 0) {
    tm = tile % tiles_m;
    tn = tile / tiles_m;
    return;
  }
  const int per = g.group * tiles_n, first = tile / per * g.group, in = tile % per, rows = min(g.group, tiles_m - first);
  tm = first + in % rows;
  tn = in / rows;
}
constexpr int PAIR_STAGE_BYTES = BM * SWIZZLE_BYTES + (PAIR_BN / 2) * SWIZZLE_BYTES;   // 32 KB

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
    gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                             const __grid_constant__ CUtensorMap tmap_c, const GemmArgs g) {
  using T = __half;
  using G = GemmT;
  constexpr int BK = G::BK, BN = PAIR_BN;
  constexpr int A_BYTES = BM * SWIZZLE_BYTES, B_BYTES = (BN / 2) * SWIZZLE_BYTES;
  constexpr int KSLICES = BK / G::UMMA_K;
  constexpr int ACC_BUFS = 2;
  constexpr int BOX_BYTES = 32 * 64 * sizeof(T);   // one [32 rows][64 columns] staging box
  extern __shared__ unsigned char gemm_smem_raw[];
  unsigned char* smem = mp_smem_align1024(gemm_smem_raw);
  const int stages = g.stages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + static_cast<size_t>(stages) * PAIR_STAGE_BYTES);
  uint64_t* empty = full + MAX_STAGES;
  uint64_t* acc_full = empty + MAX_STAGES;
  uint64_t* acc_empty = acc_full + ACC_BUFS;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + ACC_BUFS);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  unsigned char* epi_stage = smem + static_cast<size_t>(stages) * PAIR_STAGE_BYTES + 1024;   // 8 warps x 1 or 2 boxes
  const int epi_boxes = g.epi_boxes;   // 1: a deeper operand ring; every box then waits for the previous store's read

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int num_kb = (g.K + BK - 1) / BK;
  const int tiles_m = (g.M + 2 * BM - 1) / (2 * BM), tiles_n = (g.N + BN - 1) / BN;
  const int num_tiles = tiles_m * tiles_n;
  // work unit u = (tile u % num_tiles, K split u / num_tiles) covering k-blocks [kb0, kb1)
  const int num_units = num_tiles * g.ksplit;
  const int kb_per = (num_kb + g.ksplit - 1) / g.ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
    for (int a = 0; a < ACC_BUFS; ++a) { mbar_init(acc_full + a, 1); mbar_init(acc_empty + a, 16); }
    *abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
    tma_prefetch_desc(&tmap_c);
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, ACC_BUFS * BN);
  tcgen05_fence_before_sync();
  cluster_sync_all();   // both CTAs' barriers and TMEM exist before anything crosses the pair
  tcgen05_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  mp_grid_wait();

  if (warp == 0) {
    // ------------------------------ TMA producer (both ranks) ------------------
    if (lane == 0) {
      int s = 0;
      uint32_t phase = 0;
      long it = 0;
      bool ok = true;
      for (int unit = pair; unit < num_units && ok; unit += num_pairs) {
        const int tile = unit % num_tiles, sp = unit / num_tiles;
        int tm, tn;
        pair_tile(g, tile, tiles_m, tiles_n, tm, tn);
        const int m0 = tm * 2 * BM + static_cast<int>(rank) * BM, n0 = tn * BN + static_cast<int>(rank) * (BN / 2);
        const int kb0 = sp * kb_per, kb1 = min(num_kb, kb0 + kb_per);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          if (!mbar_wait_abortable(empty + s, phase ^ 1u, g.status, abort)) { ok = false; break; }
          if (rank == 0) mbar_arrive_expect_tx(full + s, 2 * (A_BYTES + B_BYTES));
          unsigned char* sa = smem + static_cast<size_t>(s) * PAIR_STAGE_BYTES;
          unsigned char* sb = sa + A_BYTES;
          const int k0 = kb * BK;
          if (!g.a_mn) {
            tma_load_2d_pair(sa, &tmap_a, k0, m0, full + s);
          } else {
#pragma unroll 1
            for (int j = 0; j < BM / BK; ++j) tma_load_2d_pair(sa + j * (BK * SWIZZLE_BYTES), &tmap_a, m0 + j * BK, k0, full + s);
          }
          if (!g.b_mn) {
            tma_load_2d_pair(sb, &tmap_b, k0, n0, full + s);
          } else {
#pragma unroll 1
            for (int j = 0; j < (BN / 2) / BK; ++j) tma_load_2d_pair(sb + j * (BK * SWIZZLE_BYTES), &tmap_b, n0 + j * BK, k0, full + s);
          }
          if (++s == stages) { s = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (rank 0) -------------------------
    if (rank == 0) {   // the warp as a whole, see elect_one
      const uint32_t idesc = umma_instr_desc(UMMA_FMT_F16, g.a_mn, g.b_mn, 2 * BM, BN);
      const uint32_t a_lbo = g.a_mn ? BK * SWIZZLE_BYTES : 16, b_lbo = g.b_mn ? BK * SWIZZLE_BYTES : 16;
      const uint32_t a_kunits = (g.a_mn ? G::UMMA_K * SWIZZLE_BYTES : 32) >> 4, b_kunits = (g.b_mn ? G::UMMA_K * SWIZZLE_BYTES : 32) >> 4;
      const uint64_t ad0 = umma_smem_desc(mp_smem_u32(smem), a_lbo, 1024), bd0 = umma_smem_desc(mp_smem_u32(smem) + A_BYTES, b_lbo, 1024);
      int s = 0;
      uint32_t phase = 0;
      bool ok = true;
      int local = 0;
      for (int unit = pair; unit < num_units && ok; unit += num_pairs, ++local) {
        const int buf = local & 1;
        const uint32_t use = static_cast<uint32_t>(local >> 1);
        ok = mbar_wait_abortable(acc_empty + buf, (use & 1u) ^ 1u, g.status, abort);
        ok = __all_sync(0xffffffffu, ok);
        const uint32_t tmem_acc = tmem_base + buf * BN;
        const int sp = unit / num_tiles;
        const int kb0 = sp * kb_per, kb1 = min(num_kb, kb0 + kb_per);
        for (int kb = kb0; ok && kb < kb1; ++kb) {
          ok = mbar_wait_abortable(full + s, phase, g.status, abort);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tcgen05_fence_after_sync();
          const uint64_t ad = ad0 + static_cast<uint32_t>(s * (PAIR_STAGE_BYTES >> 4)), bd = bd0 + static_cast<uint32_t>(s * (PAIR_STAGE_BYTES >> 4));
          const uint32_t first = kb != kb0 ? 1u : 0u;
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < KSLICES; ++ks) umma_pair_f16(tmem_acc, ad + ks * a_kunits, bd + ks * b_kunits, idesc, ks != 0 ? 1u : first);
            umma_commit_pair_to(empty + s, 3);   // the stage is free in both CTAs
            if (kb + 1 == kb1) umma_commit_pair_to(acc_full + buf, 3);
          }
          __syncwarp();
          if (++s == stages) { s = 0; phase ^= 1u; }
        }
      }
    }
    mp_launch_dependents();
  } else {
    // ------------------------------ epilogue (both ranks) -----------------------
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const T* bias = static_cast<const T*>(g.bias);
    const bool vec_ok = (g.ldc * sizeof(T)) % 16 == 0 && mp_aligned16(g.c);
    const bool use_tma = vec_ok && g.beta == 0.0f && g.ksplit == 1;
    unsigned char* stage_base = epi_stage + (warp - 2) * (epi_boxes * BOX_BYTES);
    int local = 0;
    for (int unit = pair; unit < num_units; unit += num_pairs, ++local) {
      const int tile = unit % num_tiles, sp = unit / num_tiles;
      const int buf = local & 1;
      const uint32_t use = static_cast<uint32_t>(local >> 1);
      int tm, tn;
      pair_tile(g, tile, tiles_m, tiles_n, tm, tn);
      const int m0 = tm * 2 * BM + static_cast<int>(rank) * BM, n0 = tn * BN;
      const bool acc_ready = mbar_wait_abortable(acc_full + buf, use & 1u, g.status, abort);
      __syncwarp();
      if (!acc_ready) break;
      tcgen05_fence_after_sync();
      const uint32_t tmem_acc = tmem_base + buf * BN;
      const int row = m0 + quarter * 32 + lane;
      T* crow = static_cast<T*>(g.c) + static_cast<size_t>(row) * g.ldc;
      // one staging box (64 columns) per iteration: both TMEM loads are in flight before the wait
      int boxi = 0;
#pragma unroll 1
      for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 64, ++boxi) {
        const int col0 = n0 + c0;
        if (col0 >= g.N) break;
        uint32_t v[2][32];
        tmem_ld_32x32(tmem_acc + (static_cast<uint32_t>(quarter * 32) << 16) + c0, v[0]);
        tmem_ld_32x32(tmem_acc + (static_cast<uint32_t>(quarter * 32) << 16) + c0 + 32, v[1]);
        tmem_ld_wait();
        if (g.ksplit > 1) {   // raw partial sums; alpha, bias and beta are applied by the fold
          if (row < g.M) {
#pragma unroll
            for (int hb = 0; hb < 2; ++hb) {
              const int colb = col0 + 32 * hb;
              float* prow = g.partial + (static_cast<size_t>(sp) * g.M + row) * g.partial_ld + colb;
              if (colb + 32 <= g.N) {
#pragma unroll
                for (int p = 0; p < 8; ++p)
                  *reinterpret_cast<uint4*>(prow + p * 4) = make_uint4(v[hb][p * 4], v[hb][p * 4 + 1], v[hb][p * 4 + 2], v[hb][p * 4 + 3]);
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (colb + j < g.N) prow[j] = __uint_as_float(v[hb][j]);
              }
            }
          }
          continue;
        }
        constexpr int PN = Pack<T>::N;
        unsigned char* box = stage_base + (epi_boxes == 2 ? boxi : 0) * BOX_BYTES;
        if (use_tma && (boxi == 0 || epi_boxes == 1)) {   // the earlier stores have finished reading the staging box(es)
          if (lane == 0) bulk_wait_read<0>();
          __syncwarp();
        }
#pragma unroll
        for (int hb = 0; hb < 2; ++hb) {   // (no early exit: the register arrays must stay statically indexed)
          const int colb = col0 + 32 * hb;
          if (colb < g.N) {
          float r[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = g.alpha * __uint_as_float(v[hb][j]);
          const bool by_rows = !use_tma && !(vec_ok && colb + 32 <= g.N);
          if (bias != nullptr && (g.bias_pitch == 0 || (row < g.M && !by_rows))) {
            const T* brow = bias + static_cast<size_t>(row) * g.bias_pitch;
            if (colb + 32 <= g.N && (g.bias_pitch * sizeof(T)) % 16 == 0 && mp_aligned16(bias)) {
              // the lane's 32 values are one contiguous 64-byte piece (of its row, where the term is a full matrix)
#pragma unroll
              for (int p = 0; p < 32 / PN; ++p) {
                float add[PN];
                unpack<T>(ld_pack(brow + colb, p), add);
#pragma unroll
                for (int e = 0; e < PN; ++e) r[p * PN + e] += add[e];
              }
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (colb + j < g.N) r[j] += mp_up(brow[colb + j]);
            }
          }
          if (use_tma) {
#pragma unroll
            for (int p = 0; p < 4; ++p)
              *reinterpret_cast<Pack<T>*>(box + lane * 128 + (((4 * hb + p) ^ (lane & 7)) << 4)) = pack<T>(r + p * PN);
          } else if (by_rows && g.beta == 0.0f && (bias == nullptr || g.bias_pitch == 0)) {   // (nothing is aligned: all blocks come here)
            uint32_t* words = reinterpret_cast<uint32_t*>(stage_base);
            stage_half_words(words, r, lane, hb);
            if (hb == 1 || colb + 32 >= g.N) {
              const int row0 = m0 + quarter * 32;
              store_half_rows(words, lane, crow - static_cast<size_t>(lane) * g.ldc + col0, g.ldc, min(32, g.M - row0), min(32 * hb + 32, g.N - col0));
            }
          } else if (by_rows) {
            const int row0 = m0 + quarter * 32;
            store_block_rows<T>(reinterpret_cast<float*>(stage_base), r, lane, crow - static_cast<size_t>(lane) * g.ldc + colb, g.ldc,
                                min(32, g.M - row0), colb + lane < g.N,
                                bias != nullptr && g.bias_pitch != 0 ? bias + static_cast<size_t>(row0) * g.bias_pitch + colb : nullptr,
                                g.bias_pitch, g.beta);
          } else if (row < g.M) {
            if (g.beta != 0.0f) {
#pragma unroll
              for (int p = 0; p < 32 / PN; ++p) {
                float old[PN];
                unpack<T>(ld_pack(crow + colb, p), old);
#pragma unroll
                for (int e = 0; e < PN; ++e) r[p * PN + e] += g.beta * old[e];
              }
            }
#pragma unroll
            for (int p = 0; p < 32 / PN; ++p) st_pack(crow + colb, p, pack<T>(r + p * PN));
          }
          }
        }
        if (use_tma) {   // columns past N are clipped by the store
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmap_c, box, col0, m0 + quarter * 32);
            bulk_commit();
          }
        }
      }
      // hand the accumulator back to rank 0's MMA thread: one arrival per warp of either rank
      tcgen05_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        if (rank == 0) mbar_arrive(acc_empty + buf);
        else mbar_arrive_cluster(acc_empty + buf, 0);
      }
    }
    if (use_tma && lane == 0) bulk_wait_all<0>();
  }
  __syncwarp();         // the cluster barrier below is warp-aligned: lanes that skipped the role loops wait here
  tcgen05_fence_before_sync();
  cluster_sync_all();   // neither CTA frees TMEM or leaves while its partner may still read its memory
  if (warp == 1) tmem_dealloc_pair(tmem_base, ACC_BUFS * BN);
}

// ---------------------------------------------------------------------------
// Operands that TMA cannot address (a row pitch or a base that is no multiple of 16 bytes: odd widths) are copied into rows of
// a 16-byte pitch in the stream's workspace and multiplied from there.  The copy moves each element twice against the tensor
// pipe's M or N uses of it; the FP-pipe kernel that served these shapes before reached 16 TFLOP/s ([2000, 999] x [999, 1501] and
// the two contractions of its reverse in r32: 1148 us there, 196 us from copies, 15 us of them the copies).  Every contraction copies the
// operands it reads: a training step of a dense block copies x, its weights and the upstream gradient twice each.  One thread makes one
// 16-byte chunk of a destination row from 2- or 4-byte loads (neighbouring threads share the sectors); the bytes of the last
// chunk past the row's end are zeros that the tensor map does not read.
// ---------------------------------------------------------------------------
struct PadJob {
  const unsigned char* src;
  unsigned char* dst;
  size_t src_pitch;        // bytes
  uint32_t row_bytes;      // bytes of a row that are copied
  uint32_t chunks;         // 16-byte chunks of a destination row
  uint32_t total;          // chunks of all rows
};
__global__ void __launch_bounds__(256) pad_rows_kernel(const PadJob ja, const PadJob jb, uint32_t blocks_a) {
  mp_grid_dependency();
  const bool second = blockIdx.x >= blocks_a;
  const PadJob j = second ? jb : ja;
  const uint32_t id = (second ? blockIdx.x - blocks_a : blockIdx.x) * 256u + threadIdx.x;
  if (id >= j.total) return;
  const uint32_t row = id / j.chunks, off = (id - row * j.chunks) * 16u;
  const unsigned char* s = j.src + row * j.src_pitch + off;
  uint32_t w[4];
  if (off + 16u <= j.row_bytes) {
    if ((reinterpret_cast<uintptr_t>(s) & 3u) == 0) {
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = *reinterpret_cast<const uint32_t*>(s + 4 * e);
    } else {   // r16 at an odd element: half words at both ends, words between
      const uint32_t h0 = *reinterpret_cast<const uint16_t*>(s), h7 = *reinterpret_cast<const uint16_t*>(s + 14);
      const uint32_t a = *reinterpret_cast<const uint32_t*>(s + 2), b = *reinterpret_cast<const uint32_t*>(s + 6), c = *reinterpret_cast<const uint32_t*>(s + 10);
      w[0] = h0 | (a << 16);
      w[1] = (a >> 16) | (b << 16);
      w[2] = (b >> 16) | (c << 16);
      w[3] = (c >> 16) | (h7 << 16);
    }
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      w[e] = 0u;
      if (off + 4 * e + 2 <= j.row_bytes) w[e] = *reinterpret_cast<const uint16_t*>(s + 4 * e);
      if (off + 4 * e + 4 <= j.row_bytes) w[e] |= static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(s + 4 * e + 2)) << 16;
    }
  }
  *reinterpret_cast<uint4*>(j.dst + static_cast<size_t>(id) * 16u) = make_uint4(w[0], w[1], w[2], w[3]);
}

// ---------------------------------------------------------------------------
// Host side: tensor maps and dispatch.
// ---------------------------------------------------------------------------
template <int BN, bool EXACT>
void launch_tc(Operand<__half> a, Operand<__half> b, const GemmArgs& args, int sm_count, cudaStream_t st) {
  using T = __half;
  using G = GemmT;
  const int M = args.M, N = args.N, K = args.K;
  // A: K-major [M,K] box {BK, BM};  MN-major [K,M] box {BK (along M), BK (k-rows)}
  const size_t nb = static_cast<size_t>(args.batch);
  const CUtensorMap ta = args.a_mn ? make_map<T>(a.p, K, M, a.ld, G::BK, G::BK, CU_TENSOR_MAP_SWIZZLE_128B, nb) : make_map<T>(a.p, M, K, a.ld, G::BK, BM, CU_TENSOR_MAP_SWIZZLE_128B, nb);
  const CUtensorMap tb = args.b_mn ? make_map<T>(b.p, K, N, b.ld, G::BK, G::BK, CU_TENSOR_MAP_SWIZZLE_128B, nb) : make_map<T>(b.p, N, K, b.ld, G::BK, BN, CU_TENSOR_MAP_SWIZZLE_128B, nb);
  // C as a TMA store target: 32 x 32 blocks, no swizzle (only used when the row pitch is a multiple of 16 bytes)
  CUtensorMap tc = ta;
  if ((args.ldc * sizeof(T)) % 16 == 0 && mp_aligned16(args.c)) tc = make_store_map<T>(args.c, M, N, args.ldc, BN >= 128, nb);
  const size_t smem = static_cast<size_t>(args.stages) * stage_bytes<BN>() + 1024 /*align*/ + 1024 /*barriers*/ +
                      8 * EPI_BUFS * 32 * 32 * sizeof(T) /*epilogue staging*/;
  MP_CUDA_CHECK(cudaFuncSetAttribute(gemm_tcgen05_kernel<BN, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     static_cast<int>(smem)));
  const long tiles = static_cast<long>((N + BN - 1) / BN) * ((M + BM - 1) / BM) * args.ksplit * args.batch;
  const int grid = tiles < sm_count ? static_cast<int>(tiles) : sm_count;   // persistent: one CTA per SM
  MpLaunch(grid, GEMM_THREADS, smem, st)(gemm_tcgen05_kernel<BN, EXACT>, ta, tb, tc, args);
  MP_LAUNCH_CHECK();
  if (args.ksplit > 1) launch_fold<T>(args, NoAgain{}, st);
}

void launch_pair(Operand<__half> a, Operand<__half> b, GemmArgs args, int sm_count, cudaStream_t st) {
  using T = __half;
  using G = GemmT;
  const int M = args.M, N = args.N, K = args.K;
  const CUtensorMap ta = args.a_mn ? make_map<T>(a.p, K, M, a.ld, G::BK, G::BK) : make_map<T>(a.p, M, K, a.ld, G::BK, BM);
  const CUtensorMap tb = args.b_mn ? make_map<T>(b.p, K, N, b.ld, G::BK, G::BK) : make_map<T>(b.p, N, K, b.ld, G::BK, PAIR_BN / 2);
  CUtensorMap tc = ta;
  if ((args.ldc * sizeof(T)) % 16 == 0 && mp_aligned16(args.c)) tc = make_store_map<T>(args.c, M, N, args.ldc, true);
  // 227 KB: six 32 KB stages + one 4 KB staging box per epilogue warp, or five stages + two boxes.  The ring depth is what
  // feeds the tensor pipe: a stage is refilled only after its MMAs have completed, so (stages - 1) x 32 KB are in flight
  // per SM against an L2 latency of 2 - 3 k cycles under load (measured: the MMA thread waited for operands 35 - 40 % of
  // every tile with five stages).
  args.group = 2.0 * M * K > PAIR_GROUP_BYTES ? PAIR_GROUP : 0;
  args.stages = 6;
  args.epi_boxes = 1;
  if (const char* e = getenv("MP_GEMM_PAIR_STAGES")) { if (atoi(e) == 5) { args.stages = 5; args.epi_boxes = 2; } }
  const size_t smem = static_cast<size_t>(args.stages) * PAIR_STAGE_BYTES + 1024 /*align*/ + 1024 /*barriers*/ +
                      8 * args.epi_boxes * 32 * 64 * sizeof(T);
  MP_CUDA_CHECK(cudaFuncSetAttribute(gemm_tcgen05_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  const int tiles = ((N + PAIR_BN - 1) / PAIR_BN) * ((M + 2 * BM - 1) / (2 * BM)) * args.ksplit;
  const int pairs = tiles < sm_count / 2 ? tiles : sm_count / 2;
  MpLaunch(2 * pairs, GEMM_THREADS, smem, st)(gemm_tcgen05_pair_kernel, ta, tb, tc, args);
  MP_LAUNCH_CHECK();
  if (args.ksplit > 1) launch_fold<T>(args, NoAgain{}, st);
}

// Output-tile width: wide tiles for wide problems, narrower ones when they are
// needed to put at least ~one CTA on every SM.
int pick_bn(int M, int N, int sms, int batch = 1) {
  const long tiles_m = static_cast<long>((M + BM - 1) / BM) * batch;
  if (N > 128 && tiles_m * ((N + 255) / 256) >= sms) return 256;
  if (N > 64 && tiles_m * ((N + 127) / 128) >= sms / 2) return 128;
  return N > 64 && tiles_m * ((N + 127) / 128) >= 4 ? 128 : 64;
}

// Split-K: contractions with few output tiles and a long K (weight gradients: K = tokens) leave SMs
// idle or run a mostly empty last wave.  Cost model in k-block steps of one CTA:
//   waves(tiles * ks / SMs) * (k-blocks per unit + fixed cost per unit) * step time(BN)  [+ fold traffic]
// The unsplit choice of pick_bn stays unless a split is predicted to be at least 15 % faster.
void pick_split_k(GemmArgs& args, int sms, size_t workspace_bytes, int* bn_io) {
  constexpr int bk = GemmT::BK;
  const long num_kb = (args.K + bk - 1) / bk;
  if (num_kb < 32) return;
  const double mn_bytes = static_cast<double>(args.M) * args.partial_ld * 4.0;
  auto cost = [&](int bn, int ks) {
    const long tiles = static_cast<long>((args.M + BM - 1) / BM) * ((args.N + bn - 1) / bn);
    const long waves = (tiles * ks + sms - 1) / sms;
    // one k-block step of a CTA at ~1000 TFLOP/s over all SMs, in microseconds
    const double step_us = 2.0 * BM * bn * bk / (1000.0e6 / sms);
    double t = waves * ((num_kb + ks - 1) / ks + 8.0) * step_us;
    if (ks > 1) t += 2.0 * ks * mn_bytes / 6.0e6 + 3.0;   // partial write + read at ~6 TB/s, one more launch
    return t;
  };
  const double base = cost(*bn_io, 1);
  double best = base;
  int best_bn = *bn_io, best_ks = 1;
  const int bns[2] = {128, 256};
  for (int bi = 0; bi < 2; ++bi) {
    const int bn = bns[bi];
    if (bn == 256 && (args.N <= 128 || args.exact)) continue;
    for (int ks = 2; ks <= 16; ++ks) {
      if (static_cast<double>(ks) * mn_bytes > static_cast<double>(workspace_bytes)) break;
      if (num_kb / ks < 8) break;
      if ((ks - 1) * ((num_kb + ks - 1) / ks) >= num_kb) continue;   // the last unit would be empty
      const double t = cost(bn, ks);
      if (t < best) { best = t; best_bn = bn; best_ks = ks; }
    }
  }
  if (best_ks > 1 && best < 0.85 * base) { args.ksplit = best_ks; *bn_io = best_bn; }
}

// Fewer 256 x 256 tiles than pairs: still faster where the single CTAs' tiles take more rounds.  Estimate of both in cycles: rounds x (k-blocks x
// cycles per k-block under load + cycles to fill and to drain a tile).  us, single CTAs / pairs: [4096, 3352] x [3352, 768] 45.3 / 27.4, with a
// residual [4096, 1536] x [1536, 768] 31.2 / 16.4, 2048^3 25.6 / 17.2, [2048, 512] x [512, 2048] 9.6 / 8.9; where a tile has few k-blocks the pairs'
// hand-shakes cost more than a round ([8192, 256] x [256, 512] 7.1 / 7.6).
bool pair_saves_rounds(const GemmArgs& args, int bn, long pair_tiles, int sms) {
  const long num_kb = (args.K + GemmT::BK - 1) / GemmT::BK, tiles = static_cast<long>((args.M + BM - 1) / BM) * ((args.N + bn - 1) / bn);
  const double one = static_cast<double>((tiles + sms - 1) / sms) * (num_kb * (bn == 256 ? 950.0 : bn == 128 ? 590.0 : 430.0) + 1500.0);
  const double pair = static_cast<double>((pair_tiles + sms / 2 - 1) / (sms / 2)) * (num_kb * 800.0 + 4500.0);
  return pair < 0.9 * one;
}

// One r16 contraction whose operands TMA can address.  `args` carries the problem; the tile width, the K split and the ring depth
// are chosen here.  workspace: room for split-K partials.
void gemm_run_r16(Operand<__half> a, Operand<__half> b, GemmArgs args, int sms, void* workspace, size_t workspace_bytes, cudaStream_t st) {
  args.partial_ld = (args.N + 3) & ~3;
  int bn = pick_bn(args.M, args.N, sms, args.batch);
  if (args.exact && bn == 256) bn = 128;   // the widest tile whose sums the epilogue warps can hold
  args.ksplit = 1;
  args.partial = static_cast<float*>(workspace);
  if (args.batch == 1 && !env_flag("MP_GEMM_NO_SPLITK")) pick_split_k(args, sms, workspace_bytes, &bn);
  // shared memory of the ring: 227 KB per CTA minus alignment slack, barriers and the epilogue staging (64 KB)
  const int budget = 159 * 1024;
  auto stages_for = [&](int per_stage) {   // the ring runs across tiles, so depth is bounded by memory only
    int s = budget / per_stage;
    if (s > MAX_STAGES) s = MAX_STAGES;
    return s < 2 ? 2 : s;
  };
  // CTA pairs for wide problems with enough 256 x 256 tiles to fill the pairs (their accumulators are handed over once per tile: not EXACT)
  const long pair_tiles = static_cast<long>((args.M + 255) / 256) * ((args.N + 255) / 256);
  if (args.batch == 1 && !args.exact && !env_flag("MP_GEMM_NO_PAIRS") && args.M >= 256 && args.N >= 256) {
    if (args.ksplit == 1 && ((bn == 256 && pair_tiles >= sms / 2) || pair_saves_rounds(args, bn, pair_tiles, sms))) {
      launch_pair(a, b, args, sms, st);
      return;
    }
    if (args.ksplit > 1) {
      // long K, few tiles: 256 x 256 pair tiles with the K range cut so that the units fill the pairs about evenly
      const long num_kb = (args.K + 63) / 64;
      const int pairs = sms / 2;
      int best = 0; double best_cost = 1e30;
      for (int ks = 1; ks <= 16; ++ks) {
        if (num_kb / ks < 8 || (ks - 1) * ((num_kb + ks - 1) / ks) >= num_kb) continue;
        if (static_cast<double>(ks) * args.M * args.partial_ld * 4.0 > static_cast<double>(workspace_bytes)) break;
        const long waves = (pair_tiles * ks + pairs - 1) / pairs;
        const double cost = waves * ((num_kb + ks - 1) / ks + 10.0) + (ks > 1 ? 2.0 * ks * args.M * args.N * 4.0 / 6.0e6 / 0.5 : 0.0);
        if (cost < best_cost) { best_cost = cost; best = ks; }
      }
      if (best >= 1) {
        args.ksplit = best;
        launch_pair(a, b, args, sms, st);
        return;
      }
    }
  }
  if (bn == 256) {
    args.stages = stages_for(stage_bytes<256>());
    launch_tc<256, false>(a, b, args, sms, st);
  } else if (bn == 128) {
    args.stages = stages_for(stage_bytes<128>());
    if (args.exact) launch_tc<128, true>(a, b, args, sms, st); else launch_tc<128, false>(a, b, args, sms, st);
  } else {
    args.stages = stages_for(stage_bytes<64>());
    if (args.exact) launch_tc<64, true>(a, b, args, sms, st); else launch_tc<64, false>(a, b, args, sms, st);
  }
}

inline void gemm_run(Operand<__half> a, Operand<__half> b, const GemmArgs& args, int sms, void* ws, size_t ws_bytes, cudaStream_t st) {
  gemm_run_r16(a, b, args, sms, ws, ws_bytes, st);
}
inline void gemm_run(Operand<float> a, Operand<float> b, const GemmArgs& args, int sms, void* ws, size_t ws_bytes, cudaStream_t st) {
  gemm_run_r32(a, b, args, sms, ws, ws_bytes, st);
}

// Up to here two launches and the pass over the operands leave no gain over the tf32 kernel (us, that / from terms: [1024, 1024, 1024] 22 / 25,
// [777, 777, 777] 19 / 23, with A along M 21 / 23).
constexpr double TERMS_MIN_VOLUME = 1e9;

// The FP-pipe kernel: r64, and what does not pay on the tensor cores.
template <typename T>
void gemm_simt(const T* a, const T* b, const T* bias, double alpha, T* c, double beta, len_t M, len_t N, len_t K, int a_mn, int b_mn, len_t batch,
               len_t bias_pitch, cudaStream_t st) {
  using A = typename Acc<T>::type;
  if ((M + 63) / 64 > 65535) MP_FATAL("inner_product: M too large for the FP-pipe kernel");
  for (len_t b0 = 0; b0 < batch; b0 += 65535) {   // grid.z carries the batch index
    const len_t nb = batch - b0 < 65535 ? batch - b0 : 65535;
    const dim3 grid(static_cast<unsigned>((N + 63) / 64), static_cast<unsigned>((M + 63) / 64), static_cast<unsigned>(nb));
    MpLaunch(grid, 256, 0, st)(gemm_simt_kernel<T>, a + b0 * M * K, b + b0 * K * N, bias, static_cast<A>(alpha), c + b0 * M * N, static_cast<A>(beta), M,
                                              N, K, a_mn, b_mn, bias_pitch);
    MP_LAUNCH_CHECK();
  }
}

// A contraction with operands that need a copy into aligned rows (see pad_rows_kernel).  Where the copies of whole operands do
// not fit three quarters of the workspace (the rest is left to split-K partials), the batch, then the rows of C, then its
// columns are worked off in slabs.  Returns false where even the smallest slab does not fit (a K of tens of thousands with a
// small MP_WORKSPACE_MB).
template <typename T>
bool gemm_padded(const T* a, const T* b, bool pad_a, bool pad_b, GemmArgs args, MpStreamState* state, cudaStream_t st) {
  const size_t M = args.M, N = args.N, K = args.K, batch = args.batch;
  const size_t limit = state->workspace_bytes / 4 * 3;
  constexpr size_t LINE = 16 / sizeof(T);
  auto up = [](size_t v, size_t to) { return (v + to - 1) / to * to; };
  auto bytes_a = [&](size_t m) { return pad_a ? up((args.a_mn ? K * up(m, LINE) : m * up(K, LINE)) * sizeof(T), 256) : 0; };
  auto bytes_b = [&](size_t n) { return pad_b ? up((args.b_mn ? K * up(n, LINE) : n * up(K, LINE)) * sizeof(T), 256) : 0; };
  size_t ms = M, ns = N, bs = batch;
  if (bytes_a(M) + bytes_b(N) > limit) {
    bs = 1;
    while (bytes_a(ms) + bytes_b(ns) > limit) {
      size_t* cut = (bytes_a(ms) >= bytes_b(ns) && ms > 256) || ns <= 256 ? &ms : &ns;
      if (*cut <= 256) return false;
      *cut = up((*cut + 1) / 2, 256);
    }
  } else if (batch > 1) {
    const size_t per = bytes_a(M) + bytes_b(N);
    if (per * batch > limit) bs = limit / per;
  }
  unsigned char* ws = static_cast<unsigned char*>(state->workspace);
  const T* bias = static_cast<const T*>(args.bias);
  T* c = static_cast<T*>(args.c);
  for (size_t b0 = 0; b0 < batch; b0 += bs) {
    const size_t nb = batch - b0 < bs ? batch - b0 : bs;
    for (size_t n0 = 0; n0 < N; n0 += ns) {
      for (size_t m0 = 0; m0 < M; m0 += ms) {
        const size_t m = M - m0 < ms ? M - m0 : ms, n = N - n0 < ns ? N - n0 : ns;
        size_t used = 0;
        PadJob jobs[2] = {};
        uint32_t blocks[2] = {0, 0};
        auto place = [&](int which, const T* src, bool pad, bool mn, size_t ext, size_t full) {   // ext of `full` rows resp. columns
          const size_t rows = (mn ? K : ext) * nb, cols = mn ? ext : K, src_ld = mn ? full : K;
          if (!pad) return Operand<T>{src, src_ld};
          const size_t ld = up(cols, LINE);
          PadJob& j = jobs[which];
          j.src = reinterpret_cast<const unsigned char*>(src);
          j.dst = ws + used;
          j.src_pitch = src_ld * sizeof(T);
          j.row_bytes = static_cast<uint32_t>(cols * sizeof(T));
          j.chunks = static_cast<uint32_t>(ld / LINE);
          j.total = static_cast<uint32_t>(rows * (ld / LINE));
          blocks[which] = (j.total + 255) / 256;
          used += up(rows * ld * sizeof(T), 256);
          return Operand<T>{reinterpret_cast<const T*>(j.dst), ld};
        };
        // (slabs inside an entry only with bs = 1, so a copy of several entries is always of whole, densely packed ones)
        const Operand<T> oa = place(0, a + b0 * M * K + (args.a_mn ? m0 : m0 * K), pad_a, args.a_mn != 0, m, M);
        const Operand<T> ob = place(1, b + b0 * N * K + (args.b_mn ? n0 : n0 * K), pad_b, args.b_mn != 0, n, N);
        MpLaunch(blocks[0] + blocks[1], 256, 0, st)(pad_rows_kernel, jobs[0], jobs[1], blocks[0]);
        MP_LAUNCH_CHECK();
        GemmArgs s = args;
        s.exact = 1;
        s.M = static_cast<int>(m);
        s.N = static_cast<int>(n);
        s.batch = static_cast<int>(nb);
        s.c = c + b0 * M * N + m0 * args.ldc + n0;
        if (bias != nullptr) s.bias = bias + m0 * args.bias_pitch + n0;
        gemm_run(oa, ob, s, state->sm_count, ws + used, state->workspace_bytes - used, st);
      }
    }
  }
  return true;
}

template <typename T>
void gemm_dispatch(const void* a_, const void* b_, const void* bias, double alpha, void* c_, double beta, len_t M, len_t N,
                   len_t K, int a_mn, int b_mn, StreamContext ctx, len_t batch = 1, len_t bias_pitch = 0) {
  if (M == 0 || N == 0 || batch == 0) return;
  cudaStream_t st = mp_stream(ctx);
  const T* a = static_cast<const T*>(a_);
  const T* b = static_cast<const T*>(b_);
  T* c = static_cast<T*>(c_);
  if constexpr (!std::is_same<T, double>::value) {
    // tiles are counted, and TMA addressed, in 32 bits
    const double units = static_cast<double>((M + BM - 1) / BM) * static_cast<double>((N + 63) / 64) * static_cast<double>(batch);
    MpStreamState* state = mp_state_or_null(ctx);
    bool tensor_path = state != nullptr && K > 0 && M < (1ull << 31) && N < (1ull << 31) && K < (1ull << 31) && units < 2.0e9 &&
                       !env_flag("MP_GEMM_FORCE_SIMT");
    // TMA needs 16-byte aligned bases, row pitches and batch pitches
    const size_t a_pitch = (a_mn ? M : K) * sizeof(T), b_pitch = (b_mn ? N : K) * sizeof(T);
    const bool pad_a = !mp_aligned16(a) || a_pitch % 16 != 0, pad_b = !mp_aligned16(b) || b_pitch % 16 != 0;
    if (pad_a || pad_b) {
      // r16: the copies, the launch and a tile's way through TMEM take 8 - 12 us whatever the size.  The FP pipe takes 2.4 us and 0.11 us per step of
      // K where the output is small, and 16 TFLOP/s where it is not; with few steps of K it is bound by the output.  FP pipe / tensor cores in
      // us: [9, 301, 9] 35 / 9.5, [65, 65, 65] 10.9 / 9.2, [257, 17, 257] 5.8 / 11.4, [1001, 33, 1003] 10.4 / 12.3, [1501, 33, 1503] 15.6 / 13.3,
      // [2001, 17, 2003] 18 / 20, [3001, 9, 3003] 25 / 32.
      // r32: with a short K the FP pipe's sum has seen few roundings, the split's own losses are larger.  2-norm of the error at [301, K, 307],
      // FP pipe / split: normal operands K = 33 1.04e-7 / 1.32e-7, 53 1.32e-7 / 1.29e-7, 129 2.0e-7 / 1.4e-7; operands of one sign 65 1.23e-7 /
      // 1.38e-7, 129 1.58e-7 / 1.35e-7.  (Up to there the FP pipe takes 13 us where the output is small; [4097, 63, 4099] 121 against 64 us.)
      const double volume = static_cast<double>(M) * N * K * batch;
      const bool too_tall = (M + 63) / 64 > 65535;   // for the FP-pipe kernel's grid
      tensor_path = tensor_path && (too_tall || (sizeof(T) == 4 ? K >= 96 : K >= 64 || (K >= 16 && volume > 6.0e7)));
    }
    if (tensor_path) {
      GemmArgs args;
      args.bias = bias;
      args.bias_pitch = bias_pitch;
      args.c = c;
      args.ldc = N;
      args.alpha = static_cast<float>(alpha);
      args.beta = static_cast<float>(beta);
      args.M = static_cast<int>(M);
      args.N = static_cast<int>(N);
      args.K = static_cast<int>(K);
      args.a_mn = a_mn;
      args.b_mn = b_mn;
      args.split = (std::is_same<T, float>::value && !env_flag("MP_GEMM_TF32X1")) ? 1 : 0;
      args.status = state->status_dev;
      args.batch = static_cast<int>(batch);
      if constexpr (sizeof(T) == 4) {
        const char* forced = getenv("MP_GEMM_R32_TERMS");   // a test switch: 0 never, 1 wherever the terms fit
        if (batch == 1 && args.split != 0 && (forced != nullptr || static_cast<double>(M) * N * K > TERMS_MIN_VOLUME)) {
          int bn, ks;
          double cycles = gemm_r32_estimate(args, state->sm_count, state->workspace_bytes, &bn, &ks);
          if (a_mn) cycles *= 1.2;   // (A goes through TMEM: [2048, 2048, 2048] 101 us, and 127 where its rows are contiguous along M)
          if (pad_a || pad_b) cycles = 1.1 * cycles + 5000.0 + 8.0 * K * (pad_a ? M : 0) / 2500.0 + 8.0 * K * (pad_b ? N : 0) / 2500.0;   // EXACT; the copies
          if (forced != nullptr) cycles = forced[0] == '0' ? 0.0 : 1e300;
          args.exact = pad_a || pad_b;
          if (gemm_run_r32_terms(Operand<T>{a, a_mn ? M : K}, Operand<T>{b, b_mn ? N : K}, args, state->sm_count, state->workspace,
                                 state->workspace_bytes, cycles, st))
            return;
          args.exact = 0;
        }
      }
      if (!pad_a && !pad_b) {
        gemm_run(Operand<T>{a, a_mn ? M : K}, Operand<T>{b, b_mn ? N : K}, args, state->sm_count, state->workspace, state->workspace_bytes, st);
        return;
      }
      if (gemm_padded<T>(a, b, pad_a, pad_b, args, state, st)) return;
    }
  }
  gemm_simt<T>(a, b, static_cast<const T*>(bias), alpha, c, beta, M, N, K, a_mn, b_mn, batch, bias_pitch, st);
}

}  // namespace

template <typename T>
static void inner_product_ij_jk_ik_impl(const void* a, const void* b, double alpha, void* c, double beta, len_t m, len_t n,
                                        len_t k, StreamContext ctx) {
  gemm_dispatch<T>(a, b, nullptr, alpha, c, beta, m, k, n, 0, 1, ctx);  // A[m,n] K-major, B[n,k] N-contiguous
}
template <typename T>
static void inner_product_ij_kj_ik_impl(const void* a, const void* b, double alpha, void* c, double beta, len_t m, len_t n,
                                        len_t k, StreamContext ctx) {
  gemm_dispatch<T>(a, b, nullptr, alpha, c, beta, m, k, n, 0, 0, ctx);  // B[k,n] K-major
}
template <typename T>
static void inner_product_ji_jk_ik_impl(const void* a, const void* b, double alpha, void* c, double beta, len_t m, len_t n,
                                        len_t k, StreamContext ctx) {
  gemm_dispatch<T>(a, b, nullptr, alpha, c, beta, m, k, n, 1, 1, ctx);  // A[n,m] M-contiguous
}
// C = alpha * A B + R + beta * C with a full [m, k] term R (a residual stream: R may be C itself when beta = 0)
template <typename T>
static void linear_ij_jk_ik_ik_impl(const void* a, const void* b, const void* r, double alpha, void* c, double beta, len_t m, len_t n, len_t k,
                                    StreamContext ctx) {
  gemm_dispatch<T>(a, b, r, alpha, c, beta, m, k, n, 0, 1, ctx, 1, r != nullptr ? k : 0);
}

template <typename T>
static void linear_ij_jk_ik_impl(const void* a, const void* b, const void* bias, double alpha, void* c, double beta, len_t m,
                                 len_t n, len_t k, StreamContext ctx) {
  gemm_dispatch<T>(a, b, bias, alpha, c, beta, m, k, n, 0, 1, ctx);
}

// Batched forms ("_ij,_jk->_ik" of the reference's roadmap, NOTES.md:18): densely packed [batch, ., .] operands.
template <typename T>
static void inner_product_bij_bjk_bik_impl(const void* a, const void* b, double alpha, void* c, double beta, len_t batch, len_t m,
                                           len_t n, len_t k, StreamContext ctx) {
  gemm_dispatch<T>(a, b, nullptr, alpha, c, beta, m, k, n, 0, 1, ctx, batch);
}
template <typename T>
static void inner_product_bij_bkj_bik_impl(const void* a, const void* b, double alpha, void* c, double beta, len_t batch, len_t m,
                                           len_t n, len_t k, StreamContext ctx) {
  gemm_dispatch<T>(a, b, nullptr, alpha, c, beta, m, k, n, 0, 0, ctx, batch);
}
template <typename T>
static void inner_product_bji_bjk_bik_impl(const void* a, const void* b, double alpha, void* c, double beta, len_t batch, len_t m,
                                           len_t n, len_t k, StreamContext ctx) {
  gemm_dispatch<T>(a, b, nullptr, alpha, c, beta, m, k, n, 1, 1, ctx, batch);
}

MP_STAMP3(inner_product_bij_bjk_bik, (const void* a, const void* b, const double alpha, void* c, const double beta, len_t batch, len_t m, len_t n, len_t k, StreamContext s), (a, b, alpha, c, beta, batch, m, n, k, s))
MP_STAMP3(inner_product_bij_bkj_bik, (const void* a, const void* b, const double alpha, void* c, const double beta, len_t batch, len_t m, len_t n, len_t k, StreamContext s), (a, b, alpha, c, beta, batch, m, n, k, s))
MP_STAMP3(inner_product_bji_bjk_bik, (const void* a, const void* b, const double alpha, void* c, const double beta, len_t batch, len_t m, len_t n, len_t k, StreamContext s), (a, b, alpha, c, beta, batch, m, n, k, s))
MP_STAMP3(inner_product_ij_jk_ik, (const void* a, const void* b, const double alpha, void* c, const double beta, len_t m, len_t n, len_t k, StreamContext s), (a, b, alpha, c, beta, m, n, k, s))
MP_STAMP3(inner_product_ij_kj_ik, (const void* a, const void* b, const double alpha, void* c, const double beta, len_t m, len_t n, len_t k, StreamContext s), (a, b, alpha, c, beta, m, n, k, s))
MP_STAMP3(inner_product_ji_jk_ik, (const void* a, const void* b, const double alpha, void* c, const double beta, len_t m, len_t n, len_t k, StreamContext s), (a, b, alpha, c, beta, m, n, k, s))
MP_STAMP3(linear_ij_jk_ik_ik, (const void* a, const void* b, const void* r, const double alpha, void* c, const double beta, len_t m, len_t n, len_t k, StreamContext s), (a, b, r, alpha, c, beta, m, n, k, s))
MP_STAMP3(linear_ij_jk_ik, (const void* a, const void* b, const void* bias, const double alpha, void* c, const double beta, len_t m, len_t n, len_t k, StreamContext s), (a, b, bias, alpha, c, beta, m, n, k, s))
