// Mamba-2 SSD scan as a chunk walk: a CTA goes through a (batch, head) sequence
// 128 steps at a time and keeps the carried state on chip, so no chunk state is
// written to or scanned from global memory.  The grid is one CTA per SM slot and
// every CTA walks the same number of chunks: where a CTA's range ends inside a
// sequence, the state crosses to the next CTA once, through global memory
// (walk_segment).  The same kernel evaluates the operator in both directions,
//     out_i = r_i * sum_j mask(i,j) * decay(i,j) * c_j * <q_i, k_j> * v_j
//   causal      : j <= i, decay = exp(cum_i - cum_j), c_j = dt_j, r_i = 1       (chunks first to last)
//   anti-causal : j >= i, decay = exp(cum_j - cum_i), c_j = 1,    r_i = dt_i    (chunks last to first)
// with cum the inclusive prefix sum of dt*A inside the 128-step chunk:
//   forward pass   y  = causal(q, k, v) = (C, B, x)
//   reverse pass   gx = anti(q, k, v)   = (B, C, gy),   v_t = <gx_t, x_t>
//                  u_t = <gy_t, y_t> from a second causal walk that keeps the row dots and drops y.
// Per chunk (all on the 5th-generation tensor core, operands in 128-byte
// swizzled shared memory, fp32 accumulators in TMEM):
//   G   = q k^T                         128 x 128, K = 128   -> TMEM
//   P   = G o F  (mask, decay, c_j)     TMEM -> registers -> r16 operand tile in shared memory
//   Yd  = P v                           128 x 64,  K = 128
//   Yo  = q H                           128 x 64,  K = 128   (H = state received by the chunk, r16 copy in smem)
//   S   = k^T (w o v)                   128 x 64,  K = 128   (w_j = decay of step j to the chunk's far end)
//   out = r o (Yd + f o Yo),  H' = D H + S   (H in fp32 registers of the eight worker warps)
// Warp 0 feeds the two-stage ring by TMA, one thread of warp 1 issues the MMAs, warps 2-9
// (two warps per TMEM lane quarter, one per half of the columns) do the element-wise parts.
// The chunk length of the walk is fixed (128); the `chunk` argument of the public launcher
// only selects the evaluation order of a result that does not depend on it.
#include "mp_tcgen05.cuh"

#include <cuda.h>
#include <mutex>
#include <type_traits>

namespace {

constexpr int WQ = 128;                       // steps per chunk
constexpr int WN = 128;                       // state size (columns of q and k)
constexpr int WP = 64;                        // head size (columns of v)
constexpr int W_THREADS = 320;        // warps 0-1 control (TMA, MMA), warps 2-9 workers
constexpr int W_TILE_QK = 2 * WQ * 128;       // [2 k-blocks][128 rows][128 B]
constexpr int W_TILE_V = WQ * 128;            // [128 rows][128 B]
constexpr int W_STAGE = 2 * W_TILE_QK + W_TILE_V;
constexpr int W_OFF_P = 2 * W_STAGE;
constexpr int W_OFF_H = W_OFF_P + W_TILE_QK;
constexpr int W_OFF_VS = W_OFF_H + W_TILE_V;
constexpr int W_OFF_TAIL = W_OFF_VS + W_TILE_V;   // 229376
constexpr int W_TAIL_BYTES = 2048;
constexpr int W_SMEM_BYTES = W_OFF_TAIL + W_TAIL_BYTES + 1024;   // + alignment slack = 232448 (the per-CTA maximum)
// TMEM columns
constexpr uint32_t TC_G = 0, TC_S = 128, TC_Y = 192, TC_COLS = 512;   // Yd / Yo of chunk parity p at TC_Y + p * 128 (+ 64)

enum { B_FULL0 = 0, B_FULL1, B_EMPTY0, B_EMPTY1, B_GFULL, B_PREADY, B_VSREADY, B_HREADY, B_YFULL, B_SFULL, B_SCAL, B_COUNT };

struct WalkArgs {
  int B, L, H, G, nc;
  const float* cum;        // [B, H, L] inclusive prefix sums of dt*A inside each 128-step chunk
  const float* dtt;        // [B, H, L] dt
  const float* colf;       // [B, H, L] column factor of every step relative to the far end of its 8-step piece
  __half* out;             // [B*L, H*64] or null
  const __half* z;         // dot partner, same indexing as out, or null
  float* dot_out;          // [2][B, H, L] row dots <z, out> from the fp32 accumulators, one array per half of the columns, or null
  __half* hs_out;          // [B, H, nc][128][64]: state every chunk receives, or null
  float* carry;            // [B * H][128][64] fp32: state handed from the CTA that walked the first part of a sequence to the next
  int* carry_flag;         // [B * H]: number of worker warps (of 8) that have written their part of `carry`; zero before the launch
  uint32_t* status;
};

// A CTA walks a contiguous range of the B * H * nc chunk positions (position = index in walk order, so that every CTA
// gets the same number of chunks whatever B * H is against the number of SMs).  A range is at least one sequence
// long, hence: the last part of one sequence, whole sequences, the first part of another.  The first part is walked
// FIRST and leaves its final state in `carry`; the last part is walked LAST and starts from the state the
// neighbouring CTA left there - long before, so the wait on `carry_flag` does not hold anything up (it is bounded).
struct WalkSeg { int seq, p0, n, cin, cout; };
__host__ __device__ __forceinline__ bool walk_segment(int cta, int ncta, int nseq, int nc, int idx, WalkSeg& sg) {
  const long long U = static_cast<long long>(nseq) * nc;
  const long long lo = cta * U / ncta, hi = (cta + 1) * U / ncta;
  const int s_lo = static_cast<int>(lo / nc), j_lo = static_cast<int>(lo % nc);
  const int s_hi = static_cast<int>(hi / nc), j_hi = static_cast<int>(hi % nc);
  const int first_whole = s_lo + (j_lo != 0 ? 1 : 0), n_whole = s_hi - first_whole;
  int i = idx;
  if (j_hi != 0) {
    if (i == 0) { sg.seq = s_hi; sg.p0 = 0; sg.n = j_hi; sg.cin = 0; sg.cout = 1; return true; }
    --i;
  }
  if (i < n_whole) { sg.seq = first_whole + i; sg.p0 = 0; sg.n = nc; sg.cin = 0; sg.cout = 0; return true; }
  i -= n_whole;
  if (j_lo != 0 && i == 0) { sg.seq = s_lo; sg.p0 = j_lo; sg.n = nc - j_lo; sg.cin = 1; sg.cout = 0; return true; }
  return false;
}

// Eight floats -> eight r16.
__device__ __forceinline__ uint4 walk_pack8(const float* f) {
  uint4 pk;
  uint32_t* w = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const __half2 hv = __floats2half2_rn(f[2 * e], f[2 * e + 1]);
    w[e] = *reinterpret_cast<const uint32_t*>(&hv);
  }
  return pk;
}

__device__ __forceinline__ float w_exp(float x) { return __expf(x); }

// One arrival per warp: every lane has made its shared-memory writes visible to the asynchronous proxy (and
// finished its TMEM reads) before lane 0 arrives for the warp.
__device__ __forceinline__ void warp_arrive(uint64_t* bar, int lane) {
  fence_proxy_async_smem();
  tcgen05_fence_before_sync();
  __syncwarp();
  if (lane == 0) mbar_arrive(bar);
}

// The hand-offs of the walk sit on its critical path: poll without a suspend hint first (a suspended warp
// wakes up hundreds of cycles after the phase completes), then fall back to the bounded, abortable wait.
__device__ __forceinline__ bool walk_wait(uint64_t* bar, uint32_t parity, uint32_t* status, volatile int* abort) {
#pragma unroll 1
  for (int i = 0; i < 4096; ++i) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mp_smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return mbar_wait_abortable(bar, parity, status, abort);
}

// DOT: the row dots <z, out> are wanted (the reverse pass); a template parameter, so that the forward pass does not carry the
// registers of the dot partner's rows.
template <int ANTI, bool DOT>
__global__ void __launch_bounds__(W_THREADS, 1) ssd_walk_kernel(const __grid_constant__ CUtensorMap map_q,
                                                               const __grid_constant__ CUtensorMap map_k,
                                                               const __grid_constant__ CUtensorMap map_v,
                                                               const __grid_constant__ CUtensorMap map_hs, const WalkArgs g) {
  extern __shared__ unsigned char walk_smem_raw[];
  unsigned char* smem = mp_smem_align1024(walk_smem_raw);
  unsigned char* sP = smem + W_OFF_P;
  unsigned char* sH = smem + W_OFF_H;
  unsigned char* sVs = smem + W_OFF_VS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + W_OFF_TAIL);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + W_OFF_TAIL + 112);
  volatile int* abort = reinterpret_cast<volatile int*>(smem + W_OFF_TAIL + 116);
  float* s_cum = reinterpret_cast<float*>(smem + W_OFF_TAIL + 128);   // [128]
  float* s_colf = s_cum + WQ;                                         // [128]
  float* s_dt = s_colf + WQ;                                          // [128]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nc = g.nc;
  const int nseq = g.B * g.H, cta = blockIdx.x, ncta = gridDim.x;

  if (threadIdx.x == 0) {
    mbar_init(bars + B_FULL0, 1); mbar_init(bars + B_FULL1, 1);
    mbar_init(bars + B_EMPTY0, 1); mbar_init(bars + B_EMPTY1, 1);
    mbar_init(bars + B_GFULL, 1); mbar_init(bars + B_YFULL, 1); mbar_init(bars + B_SFULL, 1);
    mbar_init(bars + B_PREADY, 8); mbar_init(bars + B_VSREADY, 8); mbar_init(bars + B_HREADY, 8);
    mbar_init(bars + B_SCAL, 4);
    *abort = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, TC_COLS);
  tcgen05_fence_before_sync();
  __syncthreads();
  tcgen05_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  mp_grid_wait();


  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      WalkSeg sg;
      int qb = 0;   // chunks walked by this CTA before the segment in hand: the barriers' phases run on across segments
      bool ok = true;
      for (int si = 0; ok && walk_segment(cta, ncta, nseq, nc, si, sg); ++si) {
        const int h = sg.seq % g.H, b = sg.seq / g.H;
        const int grp = h / (g.H / g.G);
        for (int k = 0; k < sg.n; ++k) {
          const int q = qb + k;
          const int c = ANTI ? nc - 1 - (sg.p0 + k) : sg.p0 + k;
          const int s = q & 1;
          if (!walk_wait(bars + B_EMPTY0 + s, ((q >> 1) & 1) ^ 1u, g.status, abort)) { ok = false; break; }
          unsigned char* st = smem + s * W_STAGE;
          const int row0 = c * WQ;
          mbar_arrive_expect_tx(bars + B_FULL0 + s, W_STAGE);
          tma_load_3d(st, &map_q, grp * WN, row0, b, bars + B_FULL0 + s);
          tma_load_3d(st + WQ * 128, &map_q, grp * WN + 64, row0, b, bars + B_FULL0 + s);
          tma_load_3d(st + W_TILE_QK, &map_k, grp * WN, row0, b, bars + B_FULL0 + s);
          tma_load_3d(st + W_TILE_QK + WQ * 128, &map_k, grp * WN + 64, row0, b, bars + B_FULL0 + s);
          tma_load_3d(st + 2 * W_TILE_QK, &map_v, h * WP, row0, b, bars + B_FULL0 + s);
        }
        qb += sg.n;
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer --------------------------------
    // Order per chunk k: Yd(k) as soon as its P tile is written, Yo(k) as soon as the state the chunk
    // receives is in shared memory, S(k), then the scores of chunk k+1.  The warp walks the loop as a whole, one elected lane
    // issues (see elect_one): a chunk's 32 MMAs are on the critical path of the hand-offs, and under `lane == 0` each of them
    // cost about 65 cycles of moving its descriptors into uniform registers.
    const uint32_t id_g = umma_instr_desc(UMMA_FMT_F16, 0u, 0u, 128, 128);   // q (K-major) x k (K-major)
    const uint32_t id_y = umma_instr_desc(UMMA_FMT_F16, 0u, 1u, 128, 64);    // K-major A x MN-major B
    const uint32_t id_s = umma_instr_desc(UMMA_FMT_F16, 1u, 1u, 128, 64);    // k^T (MN-major A) x MN-major B
    // descriptors of ring stage 0; stage 1 and the k-slices differ in the address field (16-byte units)
    const uint32_t s0 = mp_smem_u32(smem);
    const uint64_t d_q = umma_smem_desc(s0, 16, 1024), d_k = umma_smem_desc(s0 + W_TILE_QK, 16, 1024);
    const uint64_t d_kt = umma_smem_desc(s0 + W_TILE_QK, WQ * 128, 1024), d_v = umma_smem_desc(s0 + 2 * W_TILE_QK, W_TILE_V, 1024);
    const uint64_t d_p = umma_smem_desc(mp_smem_u32(sP), 16, 1024), d_h = umma_smem_desc(mp_smem_u32(sH), W_TILE_V, 1024);
    const uint64_t d_vs = umma_smem_desc(mp_smem_u32(sVs), W_TILE_V, 1024);
    constexpr uint32_t STAGE_U = W_STAGE >> 4, ROWS_U = 2048 >> 4;           // MN-major k-slice: 16 rows of 128 bytes
    auto kslice = [](int ks) { return static_cast<uint32_t>(((ks >> 2) * (WQ * 128) + (ks & 3) * 32) >> 4); };   // K-major: two 64-column blocks
    auto issue_g = [&](int s) {
      tcgen05_fence_after_sync();
      if (elect_one()) {
        const uint64_t dq = d_q + s * STAGE_U, dk = d_k + s * STAGE_U;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma<false>(tmem + TC_G, dq + kslice(ks), dk + kslice(ks), id_g, ks != 0 ? 1u : 0u);
        umma_commit(bars + B_GFULL);
      }
      __syncwarp();
    };
    WalkSeg sg;
    int qb = 0;          // chunks walked before this segment
    uint32_t hq = 0;     // completions of B_HREADY consumed so far (one per received state, incl. a carried-in one)
    bool ok = true;
    auto await = [&](int bar, uint32_t parity) {
      ok = walk_wait(bars + bar, parity, g.status, abort);
      ok = __all_sync(0xffffffffu, ok) != 0;
      return ok;
    };
    for (int si = 0; ok && walk_segment(cta, ncta, nseq, nc, si, sg); ++si) {
      if (await(B_FULL0 + (qb & 1), (qb >> 1) & 1)) issue_g(qb & 1);
      for (int k = 0; ok && k < sg.n; ++k) {
        const int q = qb + k;
        const int s = q & 1;
        const uint32_t ty = tmem + TC_Y + (q & 1) * 128;
        if (!await(B_PREADY, q & 1)) break;
        tcgen05_fence_after_sync();
        const uint64_t dv = d_v + s * STAGE_U;
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma<false>(ty, d_p + kslice(ks), dv + ks * ROWS_U, id_y, ks != 0 ? 1u : 0u);
        }
        __syncwarp();
        const bool has_state = k > 0 || sg.cin != 0;
        if (has_state) {
          if (!await(B_HREADY, hq & 1u)) break;
          ++hq;
          tcgen05_fence_after_sync();
        }
        if (elect_one()) {
          if (has_state) {
            if (g.hs_out != nullptr) {   // the state this chunk receives, straight from its operand tile
              const int c = ANTI ? nc - 1 - (sg.p0 + k) : sg.p0 + k;
              tma_store_2d(&map_hs, sH, 0, static_cast<int>((static_cast<size_t>(sg.seq) * nc + c) * WN));
              bulk_commit();
            }
            const uint64_t dq = d_q + s * STAGE_U;
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) umma<false>(ty + 64, dq + kslice(ks), d_h + ks * ROWS_U, id_y, ks != 0 ? 1u : 0u);
          }
          umma_commit(bars + B_YFULL);
        }
        __syncwarp();
        // scores of the next chunk (its stage was released by S(k-1); the workers are past G(k))
        if (k + 1 < sg.n) {
          const int s1 = (q + 1) & 1;
          if (!await(B_FULL0 + s1, ((q + 1) >> 1) & 1)) break;
          issue_g(s1);
        }
        if (!await(B_VSREADY, q & 1)) break;
        tcgen05_fence_after_sync();
        const uint64_t dkt = d_kt + s * STAGE_U;
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma<false>(tmem + TC_S, dkt + ks * ROWS_U, d_vs + ks * ROWS_U, id_s, ks != 0 ? 1u : 0u);
          // The workers rewrite the state tile once S(k) is complete: the store issued above must have read it by then.
          // (Waiting here, behind the next chunk's score MMAs, costs nothing; waiting right after the store held back
          // the commit of the output accumulators by the store's whole latency in every chunk.)
          if (g.hs_out != nullptr && has_state) bulk_wait_read<0>();
          umma_commit(bars + B_SFULL);
          umma_commit(bars + B_EMPTY0 + s);
        }
        __syncwarp();
      }
      qb += sg.n;
    }
    mp_launch_dependents();
    if (g.hs_out != nullptr) bulk_wait_all<0>();
  } else {
    // ------------------------------ workers -----------------------------------
    // Software pipeline: in iteration k the warps write the P tile of chunk k+1, fold S(k) into the carried
    // state, scale the values of chunk k+1 and only then read chunk k's accumulators, so that every MMA of
    // chunk k+1 is in flight while chunk k's epilogue runs.
    const int quarter = warp & 3;              // TMEM lane quarter this warp may read
    const int ch = (warp - 2) >> 2;            // column half
    const int r = quarter * 32 + lane;         // row of every 128-row tile
    const uint32_t tl = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    const int pitch = g.H * WP;
    WalkSeg sg;
    int qb = 0;          // chunks walked before this segment (barrier phases run on across segments)
    bool alive = true;
    for (int si = 0; alive && walk_segment(cta, ncta, nseq, nc, si, sg); ++si) {
    const int n = sg.n;
    const int h = sg.seq % g.H, b = sg.seq / g.H;
    const size_t bh = static_cast<size_t>(sg.seq);
    // this thread's step in the first chunk of the sequence, in the arrays per step (one offset, not one pointer per array:
    // the loop below is short of registers)
    const size_t step0 = bh * (static_cast<size_t>(g.nc) * WQ) + r;
    float state[32];
    const int c_first = ANTI ? nc - 1 - sg.p0 : sg.p0;
    if (sg.cin) {
      // the state the first part of this sequence ended with: written by all eight worker warps of the CTA that walked it
      if (lane == 0) {
        const uint64_t t0 = mp_globaltimer_ns();
        const uint64_t limit = mp_wait_limit_ns(g.status);
        while (true) {
          int seen;
          asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(g.carry_flag + sg.seq) : "memory");
          if (seen >= 8) break;
          if (*abort != 0) break;
          if (mp_globaltimer_ns() - t0 > limit) {
            *abort = 1;
            if (g.status != nullptr) atomicExch(g.status, MP_STATUS_WAIT_TIMEOUT);
            break;
          }
          __nanosleep(200);
        }
      }
      __syncwarp();
      if (*abort != 0) { alive = false; break; }
      const float4* src = reinterpret_cast<const float4*>(g.carry + (bh * WN + r) * WP + ch * 32);
#pragma unroll
      for (int q4 = 0; q4 < 8; ++q4) {
        const float4 v4 = __ldcg(src + q4);
        state[q4 * 4] = v4.x; state[q4 * 4 + 1] = v4.y; state[q4 * 4 + 2] = v4.z; state[q4 * 4 + 3] = v4.w;
      }
      // its r16 copy is the operand of the first chunk's q H (the tile is free: the previous segment's last readers,
      // q H and the state store, were complete before that segment's last S accumulator was released)
#pragma unroll
      for (int q4 = 0; q4 < 4; ++q4) {
        uint4 pk;
        uint32_t* ow = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __half2 hv = __floats2half2_rn(state[q4 * 8 + 2 * e], state[q4 * 8 + 2 * e + 1]);
          ow[e] = *reinterpret_cast<const uint32_t*>(&hv);
        }
        *reinterpret_cast<uint4*>(sH + r * 128 + (((ch * 4 + q4) ^ (r & 7)) << 4)) = pk;
      }
      warp_arrive(bars + B_HREADY, lane);
    } else {
#pragma unroll
      for (int e = 0; e < 32; ++e) state[e] = 0.f;
      if (g.hs_out != nullptr) {   // the first chunk of a sequence's walk receives nothing
        uint4* dst = reinterpret_cast<uint4*>(g.hs_out + ((bh * nc + c_first) * WN + r) * WP + ch * 32);
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) dst[q4] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    // scalars of the walk: chunk in hand (cur), the one after it (nxt), and one more in flight (pre), so that
    // their loads are never waited for
    float cum_cur = 0.f, dt_cur = 0.f, last_cur = 0.f;
    float cum_nxt = g.cum[step0 + c_first * WQ], dt_nxt = g.dtt[step0 + c_first * WQ], colf_nxt = g.colf[step0 + c_first * WQ];
    float last_nxt = 0.f;
    float cum_pre = 0.f, dt_pre = 0.f, colf_pre = 0.f;
    if (n > 1) {
      const int c1 = ANTI ? c_first - 1 : c_first + 1;
      cum_pre = g.cum[step0 + c1 * WQ]; dt_pre = g.dtt[step0 + c1 * WQ]; colf_pre = g.colf[step0 + c1 * WQ];
    }

    // Iteration k finishes chunk k of the segment and prepares chunk k+1; k = -1 is the lead-in that only prepares chunk 0.
#pragma unroll 1
    for (int k = -1; k < n; ++k) {
      const bool cur = k >= 0;
      const bool more = k + 1 < n;
      const int c = ANTI ? c_first - k : c_first + k;      // chunk in hand (meaningless in the lead-in)
      const int q = qb + k;                                // its index among the chunks this CTA walks
      const uint32_t par = static_cast<uint32_t>(q) & 1u;
      const uint32_t parn = static_cast<uint32_t>(q + 1) & 1u;
      const bool has_state = k > 0 || sg.cin != 0;         // the chunk in hand received a state
      uint4 zc[4];
      if (cur) {
        cum_cur = cum_nxt; dt_cur = dt_nxt; last_cur = last_nxt;
        if (more) {
          cum_nxt = cum_pre; dt_nxt = dt_pre; colf_nxt = colf_pre;
          if (k + 2 < n) {
            const int c2 = ANTI ? c_first - k - 2 : c_first + k + 2;
            cum_pre = g.cum[step0 + c2 * WQ]; dt_pre = g.dtt[step0 + c2 * WQ]; colf_pre = g.colf[step0 + c2 * WQ];
          }
        }
        // Yd(k) has consumed the P tile, and every warp is past the shared scalars of chunk k
        if (!walk_wait(bars + B_YFULL, par, g.status, abort)) { alive = false; break; }
      }
      if (more) {
        // ---- scalars of chunk k+1 into shared memory ------------------------------------------
        if (ch == 0) {
          s_cum[r] = cum_nxt; s_colf[r] = colf_nxt; s_dt[r] = dt_nxt;
          __syncwarp();
          if (lane == 0) mbar_arrive(bars + B_SCAL);
        }
        if (!walk_wait(bars + B_SCAL, parn, g.status, abort)) { alive = false; break; }
        last_nxt = s_cum[WQ - 1];
        // ---- P = G o F of chunk k+1 ----------------------------------------------------------------
        if (!walk_wait(bars + B_GFULL, parn, g.status, abort)) { alive = false; break; }
        tcgen05_fence_after_sync();
#pragma unroll 1
        for (int pp = 0; pp < 2; ++pp) {
          const int pc = ch * 2 + pp;              // 32-column piece of the chunk
          const int j0 = pc * 32;
          unsigned char* prow = sP + ch * (WQ * 128) + r * 128;
          const bool zero = ANTI ? (pc < quarter) : (pc > quarter);   // warp-uniform: the whole piece is masked
          if (zero) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) *reinterpret_cast<uint4*>(prow + (((pp * 4 + q4) ^ (r & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
            continue;
          }
          uint32_t v[32];
          tmem_ld_32x32(tl + TC_G + j0, v);
          // F = row factor x column factor, both relative to the far end of the 8-column sub-piece, so that neither
          // leaves the fp32 range unless eight steps decay by more than e^-80; there (rare, and only on the
          // diagonal sub-piece) the exponent is taken per element.
          const bool diag = pc == quarter;
          tmem_ld_wait();
          float rarg[4];   // <= 0 off the diagonal
#pragma unroll
          for (int sp = 0; sp < 4; ++sp) {
            const float cref = s_cum[j0 + sp * 8 + (ANTI ? 0 : 7)];
            rarg[sp] = ANTI ? cref - cum_nxt : cum_nxt - cref;
          }
          uint32_t po[16];
          if (!__any_sync(0xffffffffu, fmaxf(fmaxf(rarg[0], rarg[1]), fmaxf(rarg[2], rarg[3])) > 80.f)) {
#pragma unroll
            for (int sp = 0; sp < 4; ++sp) {   // no branch in here: the exponentials and loads of all four overlap
              const float rowf = w_exp(rarg[sp]);
              const float4 c0 = *reinterpret_cast<const float4*>(s_colf + j0 + sp * 8);
              const float4 c1 = *reinterpret_cast<const float4*>(s_colf + j0 + sp * 8 + 4);
              const float f[8] = {c0.x * rowf, c0.y * rowf, c0.z * rowf, c0.w * rowf, c1.x * rowf, c1.y * rowf, c1.z * rowf, c1.w * rowf};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const __half2 hv = __floats2half2_rn(__uint_as_float(v[sp * 8 + 2 * e]) * f[2 * e], __uint_as_float(v[sp * 8 + 2 * e + 1]) * f[2 * e + 1]);
                po[sp * 4 + e] = *reinterpret_cast<const uint32_t*>(&hv);
              }
            }
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              float f[2];
#pragma unroll
              for (int t = 0; t < 2; ++t) {
                const float cj = s_cum[j0 + 2 * e + t];
                f[t] = ANTI ? w_exp(fminf(cj - cum_nxt, 0.f)) : w_exp(fminf(cum_nxt - cj, 0.f)) * s_dt[j0 + 2 * e + t];
              }
              const __half2 hv = __floats2half2_rn(__uint_as_float(v[2 * e]) * f[0], __uint_as_float(v[2 * e + 1]) * f[1]);
              po[e] = *reinterpret_cast<const uint32_t*>(&hv);
            }
          }
          if (diag) {   // word e holds steps 2e and 2e + 1 of the piece
#pragma unroll
            for (int e = 0; e < 16; ++e)
              po[e] &= ANTI ? (2 * e >= lane ? 0xffffffffu : (2 * e + 1 >= lane ? 0xffff0000u : 0u))
                            : (2 * e + 1 <= lane ? 0xffffffffu : (2 * e <= lane ? 0xffffu : 0u));
          }
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4)
            *reinterpret_cast<uint4*>(prow + (((pp * 4 + q4) ^ (r & 7)) << 4)) = make_uint4(po[q4 * 4], po[q4 * 4 + 1], po[q4 * 4 + 2], po[q4 * 4 + 3]);
        }
        warp_arrive(bars + B_PREADY, lane);
      }
      if (cur) {
        if (DOT) {    // the dot partner's rows of chunk k, whole 64-byte row pieces per load
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const size_t zrow = static_cast<size_t>(b) * g.L + c * WQ + quarter * 32 + it * 8 + (lane >> 2);
            zc[it] = *reinterpret_cast<const uint4*>(g.z + zrow * pitch + h * WP + ch * 32 + (lane & 3) * 8);
          }
        }
        // ---- H' = D H + S ---------------------------------------------------------------
        if (!walk_wait(bars + B_SFULL, par, g.status, abort)) { alive = false; break; }
        tcgen05_fence_after_sync();
        if (more || sg.cout) {
          uint32_t sv[32];
          tmem_ld_32x32(tl + TC_S + ch * 32, sv);
          const float D = w_exp(last_cur);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; ++e) state[e] = D * state[e] + __uint_as_float(sv[e]);
          if (more) {
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              uint4 pk;
              uint32_t* ow = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const __half2 hv = __floats2half2_rn(state[q4 * 8 + 2 * e], state[q4 * 8 + 2 * e + 1]);
                ow[e] = *reinterpret_cast<const uint32_t*>(&hv);
              }
              *reinterpret_cast<uint4*>(sH + r * 128 + (((ch * 4 + q4) ^ (r & 7)) << 4)) = pk;
            }
            warp_arrive(bars + B_HREADY, lane);
          } else {
            // the first part of a sequence ends here: its state goes to the CTA that walks the rest
            float4* dst = reinterpret_cast<float4*>(g.carry + (bh * WN + r) * WP + ch * 32);
#pragma unroll
            for (int q4 = 0; q4 < 8; ++q4) __stcg(dst + q4, make_float4(state[q4 * 4], state[q4 * 4 + 1], state[q4 * 4 + 2], state[q4 * 4 + 3]));
            __threadfence();
            __syncwarp();
            if (lane == 0) atomicAdd(g.carry_flag + sg.seq, 1);
          }
        }
        // ---- out = r o (Yd + f o Yo) of chunk k -------------------------------------------
        // staging = this warp's own positions of the scaled-value tile (S(k), its last reader, has completed, and the
        // warp refills exactly these positions for chunk k+1 right after the epilogue)
        unsigned char* stg = sVs;
        if (DOT) {
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int lr = quarter * 32 + it * 8 + (lane >> 2), cc = ch * 4 + (lane & 3);
            *reinterpret_cast<uint4*>(stg + lr * 128 + ((cc ^ (lr & 7)) << 4)) = zc[it];
          }
          __syncwarp();
        }
        uint32_t yd[32], yo[32];
        const uint32_t ty = tl + TC_Y + par * 128 + ch * 32;
        tmem_ld_32x32(ty, yd);
        if (has_state) tmem_ld_32x32(ty + 64, yo);
        const float fo = has_state ? (ANTI ? w_exp(last_cur - cum_cur) : w_exp(cum_cur)) : 0.f;
        const float ro = ANTI ? dt_cur : 1.f;
        tmem_ld_wait();
        if (!has_state) {
#pragma unroll
          for (int e = 0; e < 32; ++e) yo[e] = 0u;
        }
        tcgen05_fence_before_sync();
        float o[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) o[e] = ro * (__uint_as_float(yd[e]) + fo * __uint_as_float(yo[e]));
        if (DOT) {   // this thread's row of z comes back from the staging positions before the output overwrites them
          float dot = 0.f;
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            const uint4 zq = *reinterpret_cast<const uint4*>(stg + r * 128 + (((ch * 4 + q4) ^ (r & 7)) << 4));
            const __half2* z2 = reinterpret_cast<const __half2*>(&zq);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float2 zf = __half22float2(z2[e]);
              const int k0 = q4 * 8 + 2 * e;
              dot += zf.x * o[k0] + zf.y * o[k0 + 1];
            }
          }
          g.dot_out[static_cast<size_t>(ch) * g.B * g.H * (static_cast<size_t>(g.nc) * WQ) + step0 + c * WQ] = dot;
          __syncwarp();
        }
        if (g.out != nullptr) {
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint4 pk;
            uint32_t* ow = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const __half2 hv = __floats2half2_rn(o[q4 * 8 + 2 * e], o[q4 * 8 + 2 * e + 1]);
              ow[e] = *reinterpret_cast<const uint32_t*>(&hv);
            }
            *reinterpret_cast<uint4*>(stg + r * 128 + (((ch * 4 + q4) ^ (r & 7)) << 4)) = pk;
          }
          __syncwarp();
          // whole 64-byte row pieces per store instruction
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const int lr = quarter * 32 + it * 8 + (lane >> 2), cc = ch * 4 + (lane & 3);
            const uint4 val = *reinterpret_cast<const uint4*>(stg + lr * 128 + ((cc ^ (lr & 7)) << 4));
            const size_t orow = static_cast<size_t>(b) * g.L + c * WQ + lr;
            *reinterpret_cast<uint4*>(g.out + orow * pitch + h * WP + cc * 8) = val;
          }
          __syncwarp();
        }
      }
      if (more) {
        // ---- w o v of chunk k+1 -> operand of its state update ------------------------------------
        const int s1 = (q + 1) & 1;
        if (!walk_wait(bars + B_FULL0 + s1, static_cast<uint32_t>((q + 1) >> 1) & 1u, g.status, abort)) { alive = false; break; }
        const float wt = ANTI ? w_exp(cum_nxt) : w_exp(last_nxt - cum_nxt) * dt_nxt;
        const __half2 wt2 = __float2half2_rn(wt);
        const unsigned char* src = smem + s1 * W_STAGE + 2 * W_TILE_QK + r * 128;
        unsigned char* dst = sVs + r * 128;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const int off = ((ch * 4 + q4) ^ (r & 7)) << 4;
          uint4 v = *reinterpret_cast<const uint4*>(src + off);
          __half2* h2 = reinterpret_cast<__half2*>(&v);
#pragma unroll
          for (int e = 0; e < 4; ++e) h2[e] = __hmul2(h2[e], wt2);
          *reinterpret_cast<uint4*>(dst + off) = v;
        }
        warp_arrive(bars + B_VSREADY, lane);
      }
    }
    qb += n;
    }
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, TC_COLS);
}

// ---------------------------------------------------------------------------
// The walk for two neighbouring heads of a group at once.  They share q and k (B and C belong to the group), so a chunk of both loads
// them once and its scores are computed once; Yo and S of both are single MMAs with 128 columns.  What this buys is the chain: with
// one head a chunk is a sequence of hand-offs between the tensor core and the worker warps that leaves both idle most of the time,
// with two the workers have twice the work per hand-off.
// Order of a chunk k for the workers: epilogue of Y(k-1), scale the values of chunk k, write P(k), fold S(k) into the states; for the
// MMA warp: [values and states of k written] Yo(k), S(k), [P(k) written, S(k) read] Yd(k), G(k+1).
// Shared memory has room for one v tile of each head only: v(k+1) is requested when Yd(k) has read v(k).  P lies in TMEM, in the columns
// of the scores it is made from (16 score columns become 8 + 8 columns of packed r16 pairs, one block per head): Yd reads its
// A operand there.  The fp32 states lie in TMEM as well, S and Yd share columns.  (Letting S add to D H inside its accumulator
// leaves Yd columns of its own and is 10 % faster, but rounds differently from the fused multiply-add of the one-head kernel: every
// result here is bit for bit that kernel's.)
// q and k of a chunk are read once S(k) is complete, so that their tiles take the dot partner's rows (TMA load) and the output's
// (TMA store, 32 columns a warp) before the stage goes back to the ring.
// Bound: the latency of the workers' steps, about 8000 cycles a chunk pair (state 1000, epilogue 1500, scaled values 1000, P 1900,
// Yd 900, the rest hand-offs) beside 2100 cycles of MMAs; four worker warps a scheduler hide part of it.  What counts there is registers
// (shared memory leaves L1 next to nothing, so a spill is an L2 access; hence the split below) and straight-line code in P, whose
// exponentials and shared-memory loads then overlap (one exponent-per-element path for a block as a whole, not one per 8 steps).
// 8 x 8192 steps x 32 heads, one head -> two heads at a time: forward 346 -> 281 us, reverse 1168 -> 923 us; 8 x 2048 x 24 reverse 249 ->
// 203 us.  On the way: eight worker warps with the states in registers 396 us forward; the output and the dot partner by loads and
// stores of 64-byte row pieces 44 us more forward and reverse (1500 cycles a chunk in the load/store unit).
// ---------------------------------------------------------------------------
constexpr int WP2_QK = 2 * W_TILE_QK;              // q and k of a chunk, 64 KB; two stages
constexpr int WP2_HALF = W_TILE_V / 2;             // 32 columns of one head
constexpr int WP2_OFF_V = 2 * WP2_QK;              // v of both heads
constexpr int WP2_OFF_H = WP2_OFF_V + 2 * W_TILE_V;
constexpr int WP2_OFF_VS = WP2_OFF_H + 2 * W_TILE_V;
constexpr int WP2_OFF_TAIL = WP2_OFF_VS + 2 * W_TILE_V;   // 229376
constexpr int WP2_SMEM_BYTES = WP2_OFF_TAIL + 2048 + 1024;
constexpr uint32_t TP_G = 0, TP_S = 128, TP_YD = 128, TP_H = 256, TP_YO = 384;   // TMEM columns; head h of a pair at + 64 h
constexpr int WP2_THREADS = 32 * 20;   // warps 0-1 control (2-3 idle), warps 4-19 workers: 640 threads are launched with 96 registers each,
                                       // of which the control warpgroup keeps 64 and the workers take 104 (128 * 64 + 512 * 104 = 640 * 96)
enum { PB_FULL0 = 0, PB_FULL1, PB_EMPTY0, PB_EMPTY1, PB_VFULL, PB_GFULL, PB_PREADY, PB_VSREADY, PB_YFULL, PB_SFULL, PB_SCAL, PB_ZFULL, PB_COUNT };

template <int ANTI, bool DOT>
__global__ void __launch_bounds__(WP2_THREADS, 1) ssd_walk_pair_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                    const __grid_constant__ CUtensorMap map_k,
                                                                    const __grid_constant__ CUtensorMap map_v,
                                                                    const __grid_constant__ CUtensorMap map_hs, const __grid_constant__ CUtensorMap map_z,
                                                                    const __grid_constant__ CUtensorMap map_out, const WalkArgs g) {
  constexpr bool OUT = ANTI != 0 || !DOT;   // the causal form with row dots has no other output
  extern __shared__ unsigned char walk_smem_raw[];
  unsigned char* smem = mp_smem_align1024(walk_smem_raw);
  unsigned char* sV = smem + WP2_OFF_V;
  unsigned char* sH = smem + WP2_OFF_H;
  unsigned char* sVs = smem + WP2_OFF_VS;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + WP2_OFF_TAIL);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + WP2_OFF_TAIL + 112);
  volatile int* abort = reinterpret_cast<volatile int*>(smem + WP2_OFF_TAIL + 116);
  float* s_colf = reinterpret_cast<float*>(smem + WP2_OFF_TAIL + 128);   // [2][128]
  float* s_ref = s_colf + 2 * WQ;                                        // [2][16]: cum at the far end of every 8-step piece
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nc = g.nc, hp = g.H / 2;
  const int nseq = g.B * hp, cta = blockIdx.x, ncta = gridDim.x;

  if (threadIdx.x == 0) {
    for (int i = 0; i < PB_COUNT; ++i) mbar_init(bars + i, i == PB_PREADY || i == PB_VSREADY || i == PB_SCAL || i == PB_EMPTY0 || i == PB_EMPTY1 ? 16 : 1);
    *abort = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, TC_COLS);
  tcgen05_fence_before_sync();
  __syncthreads();
  tcgen05_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  mp_grid_wait();

  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      WalkSeg sg;
      int qb = 0;   // chunks walked by this CTA before the segment in hand: the barriers' phases run on across segments
      bool ok = true;
      for (int si = 0; ok && walk_segment(cta, ncta, nseq, nc, si, sg); ++si) {
        const int h = 2 * (sg.seq % hp), b = sg.seq / hp;
        const int grp = h / (g.H / g.G);
        auto load_qk = [&](int k) {
          const int q = qb + k, s = q & 1, row0 = (ANTI ? nc - 1 - (sg.p0 + k) : sg.p0 + k) * WQ;
          if (!walk_wait(bars + PB_EMPTY0 + s, ((q >> 1) & 1) ^ 1u, g.status, abort)) return false;
          unsigned char* st = smem + s * WP2_QK;
          uint64_t* full = bars + PB_FULL0 + s;
          mbar_arrive_expect_tx(full, WP2_QK);
          tma_load_3d(st, &map_q, grp * WN, row0, b, full);
          tma_load_3d(st + WQ * 128, &map_q, grp * WN + 64, row0, b, full);
          tma_load_3d(st + W_TILE_QK, &map_k, grp * WN, row0, b, full);
          tma_load_3d(st + W_TILE_QK + WQ * 128, &map_k, grp * WN + 64, row0, b, full);
          return true;
        };
        auto load_v = [&](int k) {   // Yd of the previous chunk has read the v tiles (the workers scaled them before they wrote its P)
          const int q = qb + k, row0 = (ANTI ? nc - 1 - (sg.p0 + k) : sg.p0 + k) * WQ;
          if (q > 0 && !walk_wait(bars + PB_YFULL, (q - 1) & 1, g.status, abort)) return false;
          mbar_arrive_expect_tx(bars + PB_VFULL, 2 * W_TILE_V);
          tma_load_3d(sV, &map_v, h * WP, row0, b, bars + PB_VFULL);
          tma_load_3d(sV + W_TILE_V, &map_v, (h + 1) * WP, row0, b, bars + PB_VFULL);
          return true;
        };
        ok = load_qk(0) && load_v(0);
        for (int k = 0; ok && k < sg.n; ++k) {
          const int q = qb + k, row0 = (ANTI ? nc - 1 - (sg.p0 + k) : sg.p0 + k) * WQ;
          if (k + 1 < sg.n) ok = load_qk(k + 1);
          if (DOT && ok) {   // the dot partner's rows into the k tile that S(k) has read
            ok = walk_wait(bars + PB_SFULL, q & 1, g.status, abort);
            if (!ok) break;
            mbar_arrive_expect_tx(bars + PB_ZFULL, 2 * W_TILE_V);
            for (int t = 0; t < 4; ++t)
              tma_load_3d(smem + (q & 1) * WP2_QK + W_TILE_QK + t * WP2_HALF, &map_z, h * WP + t * 32, row0, b, bars + PB_ZFULL);
          }
          if (ok && k + 1 < sg.n) ok = load_v(k + 1);
        }
        qb += sg.n;
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (the warp as a whole, see elect_one) ----
    const uint32_t id_g = umma_instr_desc(UMMA_FMT_F16, 0u, 0u, 128, 128);    // q (K-major) x k (K-major)
    const uint32_t id_yd = umma_instr_desc(UMMA_FMT_F16, 0u, 1u, 128, 64);    // P (TMEM) x MN-major v
    const uint32_t id_yo = umma_instr_desc(UMMA_FMT_F16, 0u, 1u, 128, 128);   // q (K-major) x MN-major states of both heads
    const uint32_t id_s = umma_instr_desc(UMMA_FMT_F16, 1u, 1u, 128, 128);    // k^T (MN-major A) x MN-major scaled values of both
    const uint32_t s0 = mp_smem_u32(smem);
    const uint64_t d_q = umma_smem_desc(s0, 16, 1024);
    const uint64_t d_kt = umma_smem_desc(s0 + W_TILE_QK, WQ * 128, 1024), d_v = umma_smem_desc(mp_smem_u32(sV), W_TILE_V, 1024);
    const uint64_t d_h = umma_smem_desc(mp_smem_u32(sH), W_TILE_V, 1024);   // the scaled values follow the states
    constexpr uint32_t STAGE_U = WP2_QK >> 4, QK_U = W_TILE_QK >> 4, ROWS_U = 2048 >> 4, HEAD_U = W_TILE_V >> 4;
    auto kslice = [](int ks) { return static_cast<uint32_t>(((ks >> 2) * (WQ * 128) + (ks & 3) * 32) >> 4); };   // K-major: two 64-column blocks
    // The operands' steps are added up where they are used: hoisted out of the walk's loop they take more registers than this role has.
    auto fresh = [](uint64_t d) {
      asm volatile("" : "+l"(d));
      return d;
    };
    bool ok = true;
    auto await = [&](int bar, uint32_t parity) {
      ok = walk_wait(bars + bar, parity, g.status, abort);
      ok = __all_sync(0xffffffffu, ok) != 0;
      tcgen05_fence_after_sync();
      return ok;
    };
    auto issue_g = [&](int q) {
      if (!await(PB_FULL0 + (q & 1), (q >> 1) & 1)) return;
      const uint64_t dq = fresh(d_q) + (q & 1) * STAGE_U, dk = dq + QK_U;
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma<false>(tmem + TP_G, dq + kslice(ks), dk + kslice(ks), id_g, ks != 0 ? 1u : 0u);
        umma_commit(bars + PB_GFULL);
      }
      __syncwarp();
    };
    WalkSeg sg{};
    int qb = 0;
    // Yo and S of chunk k: the workers have written its scaled values and the states it receives
    auto issue_state = [&](int k) {
      const int q = qb + k;
      if (!await(PB_VSREADY, q & 1)) return;
      const bool has_state = k > 0 || sg.cin != 0;
      const uint64_t dq = fresh(d_q) + (q & 1) * STAGE_U, dkt = fresh(d_kt) + (q & 1) * STAGE_U, dh = fresh(d_h), dvs = dh + 2 * HEAD_U;
      if (elect_one()) {
        if (has_state) {
          if (g.hs_out != nullptr) {   // the states this chunk receives, straight from their operand tiles
            const int c = ANTI ? nc - 1 - (sg.p0 + k) : sg.p0 + k;
            const size_t bh = static_cast<size_t>(sg.seq) * 2;
            tma_store_2d(&map_hs, sH, 0, static_cast<int>((bh * nc + c) * WN));
            tma_store_2d(&map_hs, sH + W_TILE_V, 0, static_cast<int>(((bh + 1) * nc + c) * WN));
            bulk_commit();
          }
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma<false>(tmem + TP_YO, dq + kslice(ks), dh + ks * ROWS_U, id_yo, ks != 0 ? 1u : 0u);
        }
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma<false>(tmem + TP_S, dkt + ks * ROWS_U, dvs + ks * ROWS_U, id_s, ks != 0 ? 1u : 0u);
        // the workers rewrite the state tiles once S(k) is complete: the stores must have read them by then
        if (g.hs_out != nullptr && has_state) bulk_wait_read<0>();
        umma_commit(bars + PB_SFULL);
      }
      __syncwarp();
    };
    for (int si = 0; ok && walk_segment(cta, ncta, nseq, nc, si, sg); ++si) {
#pragma unroll 1
      for (int k = -1; ok && k < sg.n; ++k) {   // k = -1 only starts chunk 0
        const int q = qb + k;
        if (k >= 0 && (!await(PB_PREADY, q & 1) || !await(PB_VFULL, q & 1))) break;
        if (k >= 0 && elect_one()) {
          const uint64_t dv = fresh(d_v);
#pragma unroll
          for (int hh = 0; hh < 2; ++hh)
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)   // 16 steps: 16 score columns, then 8 columns of head 0's P and 8 of head 1's
              umma_f16_ta(tmem + TP_YD + hh * 64, tmem + TP_G + ks * 16 + hh * 8, dv + hh * HEAD_U + ks * ROWS_U, id_yd, ks != 0 ? 1u : 0u);
          umma_commit(bars + PB_YFULL);
        }
        __syncwarp();
        if (k + 1 < sg.n) {
          issue_g(q + 1);
          if (ok) issue_state(k + 1);
        }
      }
      qb += sg.n;
    }
    mp_launch_dependents();
    if (g.hs_out != nullptr) bulk_wait_all<0>();
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // ------------------------------ workers -----------------------------------
    const int quarter = warp & 3;              // TMEM lane quarter this warp may read
    const int wg = (warp - 4) >> 2;            // score columns: 32-column piece `wg` for both heads
    const int ch = wg >> 1, half = wg & 1;     // everything else: 32 columns (`half`) of head `ch` of the pair
    const int r = quarter * 32 + lane;         // row of every 128-row tile
    const uint32_t tl = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    unsigned char* hrow = sH + ch * W_TILE_V + r * 128;
    // this thread's 64 bytes of a [128][32] tile of z or of the output, 64-byte swizzle (two 16-byte pieces a row apart share a bank line)
    const uint32_t half_row = (ch * 2 + half) * WP2_HALF + r * 64, half_sw = (r >> 1) & 3;
    WalkSeg sg;
    int qb = 0;
    bool alive = true;
    for (int si = 0; alive && walk_segment(cta, ncta, nseq, nc, si, sg); ++si) {
      const int n = sg.n;
      const int h = 2 * (sg.seq % hp) + ch, b = sg.seq / hp;
      const uint32_t bh = static_cast<uint32_t>(b) * g.H + h, LP = static_cast<uint32_t>(nc) * WQ;   // B H LP fits 31 bits: see mp_ssd_walk
      // this thread's step in the first chunk of the walk, in the arrays per step of its head and of the other one
      const uint32_t step0 = bh * LP + r, other0 = (ch == 0 ? bh + 1 : bh - 1) * LP + r;
      const uint32_t tstate = tl + TP_H + ch * 64 + half * 32;
      const int c_first = ANTI ? nc - 1 - sg.p0 : sg.p0;
      // the 32 columns of the state a chunk receives: fp32 in TMEM, and an r16 copy for its q H
      auto store_state = [&](const float* hv) {
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) *reinterpret_cast<uint4*>(hrow + (((half * 4 + q4) ^ (r & 7)) << 4)) = walk_pack8(hv + q4 * 8);
        tmem_st_32x32(tstate, reinterpret_cast<const uint32_t*>(hv));
        tmem_st_wait();
      };
      if (sg.cin) {
        // the states the first part of these sequences ended with: written by all worker warps of the CTA that walked it
        if (lane == 0) {
          const uint64_t t0 = mp_globaltimer_ns();
          const uint64_t limit = mp_wait_limit_ns(g.status);
          while (true) {
            int seen;
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(g.carry_flag + sg.seq) : "memory");
            if (seen >= 16) break;
            if (*abort != 0) break;
            if (mp_globaltimer_ns() - t0 > limit) {
              *abort = 1;
              if (g.status != nullptr) atomicExch(g.status, MP_STATUS_WAIT_TIMEOUT);
              break;
            }
            __nanosleep(200);
          }
        }
        __syncwarp();
        if (*abort != 0) { alive = false; break; }
        const float4* src = reinterpret_cast<const float4*>(g.carry + (static_cast<size_t>(bh) * WN + r) * WP + half * 32);
        float hv[32];
#pragma unroll
        for (int q4 = 0; q4 < 8; ++q4) {
          const float4 v4 = __ldcg(src + q4);
          hv[q4 * 4] = v4.x; hv[q4 * 4 + 1] = v4.y; hv[q4 * 4 + 2] = v4.z; hv[q4 * 4 + 3] = v4.w;
        }
        store_state(hv);   // (the tiles are free: their last readers were complete before the previous segment's last S was)
      } else {
        if (g.hs_out != nullptr) {   // the first chunk of a sequence's walk receives nothing
          uint4* dst = reinterpret_cast<uint4*>(g.hs_out + ((static_cast<size_t>(bh) * nc + c_first) * WN + r) * WP + half * 32);
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) dst[q4] = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      // scalars of the chunk in hand (cur) and of the one after it (nxt), which are requested a whole chunk before they are used
      float cum_cur = 0.f, dt_cur = 0.f, last_cur = 0.f;
      float cum_nxt, dt_nxt, colf_nxt, oth_nxt, last_nxt;
      auto fetch = [&](int k) {
        const uint32_t i = static_cast<uint32_t>(ANTI ? c_first - k : c_first + k) * WQ;
        cum_nxt = g.cum[step0 + i]; dt_nxt = g.dtt[step0 + i]; colf_nxt = g.colf[step0 + i]; oth_nxt = g.cum[other0 + i];
        last_nxt = g.cum[step0 - r + i + WQ - 1];
      };
      fetch(0);

#pragma unroll 1
      for (int k = -1; k < n; ++k) {   // finishes chunk k, prepares chunk k+1; k = -1 only prepares
        const bool more = k + 1 < n;
        const int c = ANTI ? c_first - k : c_first + k;
        const int q = qb + k;
        const uint32_t par = static_cast<uint32_t>(q) & 1u, parn = static_cast<uint32_t>(q + 1) & 1u;
        if (k >= 0) {
          const bool has_state = k > 0 || sg.cin != 0;
          cum_cur = cum_nxt; dt_cur = dt_nxt; last_cur = last_nxt;
          if (more) fetch(k + 1);
          // ---- out = r o (Yd + f o Yo) of chunk k -------------------------------------------
          if (!walk_wait(bars + PB_YFULL, par, g.status, abort)) { alive = false; break; }
          tcgen05_fence_after_sync();
          const float fo = has_state ? (ANTI ? w_exp(last_cur - cum_cur) : w_exp(cum_cur)) : 0.f;
          const float ro = ANTI ? dt_cur : 1.f;
          unsigned char* stage = smem + (q & 1) * WP2_QK;   // q and k of chunk k, read by now: the output goes where q was, z is where k was
          if (DOT && !walk_wait(bars + PB_ZFULL, par, g.status, abort)) { alive = false; break; }
          float dot = 0.f;
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            uint32_t yd[16], yo[16];
            tmem_ld_32x16(tl + TP_YD + ch * 64 + half * 32 + p * 16, yd);
            if (has_state) tmem_ld_32x16(tl + TP_YO + ch * 64 + half * 32 + p * 16, yo);
            tmem_ld_wait();
            if (!has_state) {
#pragma unroll
              for (int e = 0; e < 16; ++e) yo[e] = 0u;
            }
#pragma unroll
            for (int q4 = 0; q4 < 2; ++q4) {
              float o[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) o[e] = ro * (__uint_as_float(yd[q4 * 8 + e]) + fo * __uint_as_float(yo[q4 * 8 + e]));
              const uint32_t slot = half_row + ((((p * 2 + q4) ^ half_sw)) << 4);
              if (DOT) {
                const uint4 zq = *reinterpret_cast<const uint4*>(stage + W_TILE_QK + slot);
                const __half2* z2 = reinterpret_cast<const __half2*>(&zq);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 zf = __half22float2(z2[e]);
                  dot += zf.x * o[2 * e] + zf.y * o[2 * e + 1];
                }
              }
              if (OUT) *reinterpret_cast<uint4*>(stage + slot) = walk_pack8(o);
            }
          }
          if (DOT) {
            g.dot_out[half * (static_cast<size_t>(g.B) * g.H * LP) + step0 + static_cast<uint32_t>(c) * WQ] = dot;
          }
          if (OUT) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              tma_store_3d(&map_out, stage + (ch * 2 + half) * WP2_HALF + quarter * 32 * 64, h * WP + half * 32, c * WQ + quarter * 32, b);
              bulk_commit();
            }
          }
        }
        // the stage of chunk k goes back once this warp's output has left it
        auto release = [&]() {
          __syncwarp();
          if (lane == 0) {
            if (OUT) bulk_wait_read<0>();
            mbar_arrive(bars + PB_EMPTY0 + (q & 1));
          }
        };
        if (!more) release();
        if (more) {
          // ---- scalars of chunk k+1 into shared memory (every warp is past its P(k): Yd(k) was complete) -------------
          if (half == 0) {
            s_colf[ch * WQ + r] = colf_nxt;
            if ((r & 7) == (ANTI ? 0 : 7)) s_ref[ch * 16 + (r >> 3)] = cum_nxt;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(bars + PB_SCAL);
          // ---- w o v of chunk k+1: operand of its state update ------------------------------------------------------
          if (!walk_wait(bars + PB_VFULL, parn, g.status, abort)) { alive = false; break; }
          {
            const __half2 wt2 = __float2half2_rn(ANTI ? w_exp(cum_nxt) : w_exp(last_nxt - cum_nxt) * dt_nxt);
            const unsigned char* src = sV + ch * W_TILE_V + r * 128;
            unsigned char* dst = sVs + ch * W_TILE_V + r * 128;
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              const int off = ((half * 4 + q4) ^ (r & 7)) << 4;
              uint4 v = *reinterpret_cast<const uint4*>(src + off);
              __half2* h2 = reinterpret_cast<__half2*>(&v);
#pragma unroll
              for (int e = 0; e < 4; ++e) h2[e] = __hmul2(h2[e], wt2);
              *reinterpret_cast<uint4*>(dst + off) = v;
            }
          }
          warp_arrive(bars + PB_VSREADY, lane);
          if (k >= 0) release();
          // ---- P = G o F of chunk k+1, both heads, in place of the scores -------------------------------------------
          if (!walk_wait(bars + PB_SCAL, parn, g.status, abort)) { alive = false; break; }
          if (!walk_wait(bars + PB_GFULL, parn, g.status, abort)) { alive = false; break; }
          tcgen05_fence_after_sync();
          // This warp's 32 steps, one head after the other; F: see ssd_walk_kernel.
          const uint32_t gcol = tl + TP_G + wg * 32;
          if (ANTI ? (wg < quarter) : (wg > quarter)) {   // warp-uniform: the whole piece is masked
            uint32_t zero[32];
#pragma unroll
            for (int e = 0; e < 32; ++e) zero[e] = 0u;
            tmem_st_32x32(gcol, zero);
          } else {
            const bool diag = wg == quarter;
#pragma unroll 1
            for (int blk = 0; blk < 2; ++blk) {
              uint32_t v[16], po[16];
              tmem_ld_32x16(gcol + blk * 16, v);
              const int jb0 = wg * 32 + blk * 16;
              const float2 ref0 = *reinterpret_cast<const float2*>(s_ref + (jb0 >> 3)), ref1 = *reinterpret_cast<const float2*>(s_ref + 16 + (jb0 >> 3));
              tmem_ld_wait();
              const float cum0 = ch == 0 ? cum_nxt : oth_nxt, cum1 = ch == 0 ? oth_nxt : cum_nxt;
              const float rarg[4] = {ANTI ? ref0.x - cum0 : cum0 - ref0.x, ANTI ? ref0.y - cum0 : cum0 - ref0.y,   // <= 0 off the diagonal
                                     ANTI ? ref1.x - cum1 : cum1 - ref1.x, ANTI ? ref1.y - cum1 : cum1 - ref1.y};
              const float rmax = fmaxf(fmaxf(rarg[0], rarg[1]), fmaxf(rarg[2], rarg[3]));
              if (!__any_sync(0xffffffffu, rmax > 80.f)) {
#pragma unroll
                for (int hs = 0; hs < 4; ++hs) {   // head of the pair, 8 steps; no branch in here: the loads and exponentials of all four overlap
                  const int hh = hs >> 1, sp = hs & 1;
                  const float rowf = w_exp(rarg[hs]);
                  const float4 c0 = *reinterpret_cast<const float4*>(s_colf + hh * WQ + jb0 + sp * 8);
                  const float4 c1 = *reinterpret_cast<const float4*>(s_colf + hh * WQ + jb0 + sp * 8 + 4);
                  const float f[8] = {c0.x * rowf, c0.y * rowf, c0.z * rowf, c0.w * rowf, c1.x * rowf, c1.y * rowf, c1.z * rowf, c1.w * rowf};
#pragma unroll
                  for (int e = 0; e < 4; ++e) {
                    const __half2 hv = __floats2half2_rn(__uint_as_float(v[sp * 8 + 2 * e]) * f[2 * e], __uint_as_float(v[sp * 8 + 2 * e + 1]) * f[2 * e + 1]);
                    po[hs * 4 + e] = *reinterpret_cast<const uint32_t*>(&hv);
                  }
                }
              } else {   // a row factor that does not fit: the step factors from global memory
#pragma unroll
                for (int hh = 0; hh < 2; ++hh) {
                  const float cum_r = hh == 0 ? cum0 : cum1;
                  const uint32_t o0 = (hh == ch ? step0 : other0) - r + static_cast<uint32_t>(ANTI ? c_first - k - 1 : c_first + k + 1) * WQ + jb0;
#pragma unroll
                  for (int e = 0; e < 8; ++e) {
                    float f[2];
#pragma unroll
                    for (int t = 0; t < 2; ++t)
                      f[t] = ANTI ? w_exp(fminf(g.cum[o0 + 2 * e + t] - cum_r, 0.f)) : w_exp(fminf(cum_r - g.cum[o0 + 2 * e + t], 0.f)) * g.dtt[o0 + 2 * e + t];
                    const __half2 hv = __floats2half2_rn(__uint_as_float(v[2 * e]) * f[0], __uint_as_float(v[2 * e + 1]) * f[1]);
                    po[hh * 8 + e] = *reinterpret_cast<const uint32_t*>(&hv);
                    asm volatile("" ::: "memory");   // one element's loads at a time: this path is rare and must not cost registers
                  }
                }
              }
              if (diag) {   // word e of a head holds steps 2e and 2e + 1 of the block
                int lr = lane - blk * 16;
                asm volatile("" : "+r"(lr));   // the masks are made here: hoisted out of the walk's loop they take sixteen registers
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  const uint32_t keep = ANTI ? (2 * e >= lr ? 0xffffffffu : (2 * e + 1 >= lr ? 0xffff0000u : 0u))
                                             : (2 * e + 1 <= lr ? 0xffffffffu : (2 * e <= lr ? 0xffffu : 0u));
                  po[e] &= keep;
                  po[8 + e] &= keep;
                }
              }
              tmem_st_32x16(gcol + blk * 16, po);
            }
          }
          tmem_st_wait();
          // ---- the state chunk k+2 receives: H' = D H + S of chunk k+1; Yd(k+1) goes where S was -------------------------------
          if (!walk_wait(bars + PB_SFULL, parn, g.status, abort)) { alive = false; break; }
          tcgen05_fence_after_sync();
          if (k + 2 < n || sg.cout) {
            float hv[32];
            tmem_ld_32x32(tl + TP_S + ch * 64 + half * 32, reinterpret_cast<uint32_t*>(hv));
            if (k >= 0 || sg.cin) {
              const float D = w_exp(last_nxt);
#pragma unroll
              for (int p = 0; p < 4; ++p) {
                uint32_t h8[8];
                tmem_ld_32x8(tstate + p * 8, h8);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) hv[p * 8 + e] = fmaf(D, __uint_as_float(h8[e]), hv[p * 8 + e]);
              }
            } else {
              tmem_ld_wait();
            }
            if (k + 2 < n) {
              store_state(hv);
            } else {   // the first part of the sequences ends here: their states go to the CTA that walks the rest
              float4* dst = reinterpret_cast<float4*>(g.carry + (static_cast<size_t>(bh) * WN + r) * WP + half * 32);
#pragma unroll
              for (int q4 = 0; q4 < 8; ++q4) __stcg(dst + q4, make_float4(hv[q4 * 4], hv[q4 * 4 + 1], hv[q4 * 4 + 2], hv[q4 * 4 + 3]));
              __threadfence();
              __syncwarp();
              if (lane == 0) atomicAdd(g.carry_flag + sg.seq, 1);
            }
          }
          warp_arrive(bars + PB_PREADY, lane);
        }
      }
      qb += n;
    }
    if (OUT && lane == 0) bulk_wait_all<0>();
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, TC_COLS);
}

// ---------------------------------------------------------------------------
// Gradients of B and C (summed over the heads of a group).  One CTA per (batch, 128-step chunk, group)
// walks the group's heads; per head h
//     Sc  = gy_h x_h^T                       128 x 128, K = 64      -> TMEM
//     acc += Sc o L_h                        in registers (L_h = causal mask * exp(cum_i - cum_j) * dt_j)
//     gC += (e_h o gy_h) Hc_h^T,  gB += (w_h o x_h) Ha_h^T          128 x 128, K = 64, accumulated over the heads in TMEM
// (Hc_h / Ha_h = the state the chunk receives from its predecessors / successors, left by the two walks;
//  e_i = exp(cum_i), w_j = exp(cum_last - cum_j) dt_j; the row factors are multiplied into the operand
//  tiles in place once the score MMA has read them).  After the last head the summed scores go to shared memory once
// and serve both products, as a K-major operand for gC += acc B and as an MN-major one for gB += acc^T C.
// No per-head score tile and no per-head partial output ever reaches global memory.
// ---------------------------------------------------------------------------
constexpr int GG_TILE = WQ * 128;                 // [128 rows][128 B]
constexpr int GG_STAGE = 4 * GG_TILE;             // gy, x, Hc, Ha
constexpr int GG_OFF_ACC = 2 * GG_STAGE;          // summed scores, [2 k-blocks][128 rows][128 B]
constexpr int GG_OFF_TAIL = GG_OFF_ACC + 2 * GG_TILE;
constexpr int GG_SMEM_BYTES = GG_OFF_TAIL + 4096 + 1024;
constexpr uint32_t GT_SC = 0, GT_C = 256, GT_B = 384;   // score buffers at 0 / 128
enum { GB_FULL0 = 0, GB_FULL1, GB_EMPTY0, GB_EMPTY1, GB_SC0, GB_SC1, GB_SCALED, GB_SCAL, GB_GG, GB_BCFULL, GB_ACC, GB_OUT, GB_COUNT };

struct GroupArgs {
  int B, L, H, G, nc;
  const float* cum; const float* dtt; const float* colf;   // [B, H, L], causal column factors
  uint32_t* status;
};

__global__ void __launch_bounds__(W_THREADS, 1) ssd_group_grads_kernel(const __grid_constant__ CUtensorMap map_gy,
                                                                      const __grid_constant__ CUtensorMap map_x,
                                                                      const __grid_constant__ CUtensorMap map_hc,
                                                                      const __grid_constant__ CUtensorMap map_ha,
                                                                      const __grid_constant__ CUtensorMap map_b,
                                                                      const __grid_constant__ CUtensorMap map_c,
                                                                      const __grid_constant__ CUtensorMap map_gb,
                                                                      const __grid_constant__ CUtensorMap map_gc, const GroupArgs g) {
  extern __shared__ unsigned char walk_smem_raw[];
  unsigned char* smem = mp_smem_align1024(walk_smem_raw);
  unsigned char* sGG = smem + GG_OFF_ACC;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + GG_OFF_TAIL);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + GG_OFF_TAIL + 112);
  volatile int* abort = reinterpret_cast<volatile int*>(smem + GG_OFF_TAIL + 116);
  float* s_cum = reinterpret_cast<float*>(smem + GG_OFF_TAIL + 128);   // [2][128]
  float* s_colf = s_cum + 2 * WQ;                                      // [2][128]
  float* s_dt = s_colf + 2 * WQ;                                       // [2][128]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int hpg = g.H / g.G;
  const int grp = blockIdx.x % g.G;
  const int c = (blockIdx.x / g.G) % g.nc;
  const int b = blockIdx.x / (g.G * g.nc);
  const int row0 = c * WQ;
  const int nh = hpg;

  if (threadIdx.x == 0) {
    mbar_init(bars + GB_FULL0, 1); mbar_init(bars + GB_FULL1, 1);
    mbar_init(bars + GB_EMPTY0, 1); mbar_init(bars + GB_EMPTY1, 1);
    mbar_init(bars + GB_SC0, 1); mbar_init(bars + GB_SC1, 1);
    mbar_init(bars + GB_SCALED, 8); mbar_init(bars + GB_SCAL, 8); mbar_init(bars + GB_GG, 8);
    mbar_init(bars + GB_BCFULL, 1); mbar_init(bars + GB_ACC, 1); mbar_init(bars + GB_OUT, 8);
    *abort = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, TC_COLS);
  tcgen05_fence_before_sync();
  __syncthreads();
  tcgen05_fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  mp_grid_wait();

  if (warp == 0) {
    // ------------------------------ TMA: loads, then the output stores -------------
    if (lane == 0) {
      bool ok = true;
      for (int hi = 0; hi < nh; ++hi) {
        const int h = grp * hpg + hi, s = hi & 1;
        if (!walk_wait(bars + GB_EMPTY0 + s, ((hi >> 1) & 1) ^ 1u, g.status, abort)) { ok = false; break; }
        unsigned char* st = smem + s * GG_STAGE;
        const int srow = ((b * g.H + h) * g.nc + c) * WN;
        mbar_arrive_expect_tx(bars + GB_FULL0 + s, GG_STAGE);
        tma_load_3d(st, &map_gy, h * WP, row0, b, bars + GB_FULL0 + s);
        tma_load_3d(st + GG_TILE, &map_x, h * WP, row0, b, bars + GB_FULL0 + s);
        tma_load_2d(st + 2 * GG_TILE, &map_hc, 0, srow, bars + GB_FULL0 + s);
        tma_load_2d(st + 3 * GG_TILE, &map_ha, 0, srow, bars + GB_FULL0 + s);
      }
      // B and C of the chunk take the place of the two stages once their last MMAs have completed
      for (int s = 0; ok && s < 2; ++s) {
        const int uses = (nh + 1 - s) / 2;       // heads that went through stage s
        if (uses > 0 && !walk_wait(bars + GB_EMPTY0 + s, (uses - 1) & 1, g.status, abort)) { ok = false; break; }
      }
      if (ok) {
        mbar_arrive_expect_tx(bars + GB_BCFULL, 4 * GG_TILE);
        tma_load_3d(smem, &map_b, grp * WN, row0, b, bars + GB_BCFULL);
        tma_load_3d(smem + GG_TILE, &map_b, grp * WN + 64, row0, b, bars + GB_BCFULL);
        tma_load_3d(smem + GG_STAGE, &map_c, grp * WN, row0, b, bars + GB_BCFULL);
        tma_load_3d(smem + GG_STAGE + GG_TILE, &map_c, grp * WN + 64, row0, b, bars + GB_BCFULL);
        if (walk_wait(bars + GB_OUT, 0, g.status, abort)) {
          // staged outputs: gC behind the B tiles of stage 0, gB behind the C tiles of stage 1
          tma_store_3d(&map_gc, smem + 2 * GG_TILE, grp * WN, row0, b);
          tma_store_3d(&map_gc, smem + 3 * GG_TILE, grp * WN + 64, row0, b);
          tma_store_3d(&map_gb, smem + GG_STAGE + 2 * GG_TILE, grp * WN, row0, b);
          tma_store_3d(&map_gb, smem + GG_STAGE + 3 * GG_TILE, grp * WN + 64, row0, b);
          bulk_commit();
          bulk_wait_all<0>();
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (the warp as a whole, see elect_one) ----
    const uint32_t id_kk = umma_instr_desc(UMMA_FMT_F16, 0u, 0u, 128, 128);   // K-major x K-major
    const uint32_t id_kn = umma_instr_desc(UMMA_FMT_F16, 0u, 1u, 128, 128);   // K-major A x MN-major B
    const uint32_t id_nn = umma_instr_desc(UMMA_FMT_F16, 1u, 1u, 128, 128);   // MN-major A x MN-major B
    // K-major descriptors of the tiles of stage 0 (gy, x, Hc, Ha); stage 1 and the k-slices differ in the address field
    const uint32_t s0 = mp_smem_u32(smem);
    const uint64_t d_t = umma_smem_desc(s0, 16, 1024);
    constexpr uint32_t STAGE_U = GG_STAGE >> 4, TILE_U = GG_TILE >> 4, ROWS_U = 2048 >> 4;
    bool ok = true;
    auto await = [&](int bar, uint32_t parity) {
      ok = walk_wait(bars + bar, parity, g.status, abort);
      ok = __all_sync(0xffffffffu, ok) != 0;
      return ok;
    };
    auto issue_score = [&](int hi) {
      tcgen05_fence_after_sync();
      const uint64_t dt = d_t + (hi & 1) * STAGE_U;
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma<false>(tmem + GT_SC + (hi & 1) * 128, dt + 2 * ks, dt + TILE_U + 2 * ks, id_kk, ks != 0 ? 1u : 0u);
        umma_commit(bars + GB_SC0 + (hi & 1));
      }
      __syncwarp();
    };
    if (await(GB_FULL0, 0)) issue_score(0);
    for (int hi = 0; ok && hi < nh; ++hi) {
      const int s = hi & 1;
      if (hi + 1 < nh) {   // the next head's scores run while the workers transform this head's
        if (!await(GB_FULL0 + ((hi + 1) & 1), ((hi + 1) >> 1) & 1)) break;
        issue_score(hi + 1);
      }
      if (!await(GB_SCALED, hi & 1)) break;
      tcgen05_fence_after_sync();
      const uint64_t dt = d_t + s * STAGE_U;
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma<false>(tmem + GT_C, dt + 2 * ks, dt + 2 * TILE_U + 2 * ks, id_kk, (hi | ks) != 0 ? 1u : 0u);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) umma<false>(tmem + GT_B, dt + TILE_U + 2 * ks, dt + 3 * TILE_U + 2 * ks, id_kk, (hi | ks) != 0 ? 1u : 0u);
        umma_commit(bars + GB_EMPTY0 + s);
      }
      __syncwarp();
    }
    // summed scores x B and (summed scores)^T x C
    if (ok && await(GB_GG, 0) && await(GB_BCFULL, 0)) {
      tcgen05_fence_after_sync();
      const uint64_t d_sg = umma_smem_desc(mp_smem_u32(sGG), 16, 1024), d_sgt = umma_smem_desc(mp_smem_u32(sGG), GG_TILE, 1024);
      const uint64_t d_b = umma_smem_desc(s0, GG_TILE, 1024), d_c = umma_smem_desc(s0 + GG_STAGE, GG_TILE, 1024);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)     // K = step j: A K-major over the two 64-column blocks, B rows j (MN-major, two 64-column blocks)
          umma<false>(tmem + GT_C, d_sg + (ks >> 2) * TILE_U + (ks & 3) * 2, d_b + ks * ROWS_U, id_kn, 1u);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)     // K = step i: A = transposed view of the same tile (MN-major), C rows i
          umma<false>(tmem + GT_B, d_sgt + ks * ROWS_U, d_c + ks * ROWS_U, id_nn, 1u);
        umma_commit(bars + GB_ACC);
      }
      __syncwarp();
    }
    mp_launch_dependents();
  } else {
    // ------------------------------ workers -----------------------------------
    const int quarter = warp & 3;
    const int ch = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const uint32_t tl = tmem + (static_cast<uint32_t>(quarter * 32) << 16);
    float acc[64];
#pragma unroll
    for (int e = 0; e < 64; ++e) acc[e] = 0.f;
    auto scal_ptr = [&](const float* base, int hi) { return base + (static_cast<size_t>(b) * g.H + grp * hpg + hi) * (static_cast<size_t>(g.nc) * WQ) + c * WQ + r; };
    float cum_n = *scal_ptr(g.cum, 0), dt_n = *scal_ptr(g.dtt, 0), colf_n = *scal_ptr(g.colf, 0);
    float cum_p = 0.f, dt_p = 0.f, colf_p = 0.f;
    if (nh > 1) { cum_p = *scal_ptr(g.cum, 1); dt_p = *scal_ptr(g.dtt, 1); colf_p = *scal_ptr(g.colf, 1); }
    bool ok = true;
    for (int hi = 0; hi < nh; ++hi) {
      const int s = hi & 1;
      const float cum_r = cum_n, dt_r = dt_n;
      float* cumb = s_cum + s * WQ;
      float* colfb = s_colf + s * WQ;
      float* dtb = s_dt + s * WQ;
      // every warp arrives: the phase also tells the writers of the other buffer that all warps are done with it
      if (ch == 0) { cumb[r] = cum_n; colfb[r] = colf_n; dtb[r] = dt_n; }
      __syncwarp();
      if (lane == 0) mbar_arrive(bars + GB_SCAL);
      cum_n = cum_p; dt_n = dt_p; colf_n = colf_p;
      if (hi + 2 < nh) { cum_p = *scal_ptr(g.cum, hi + 2); dt_p = *scal_ptr(g.dtt, hi + 2); colf_p = *scal_ptr(g.colf, hi + 2); }
      if (!walk_wait(bars + GB_SCAL, hi & 1, g.status, abort)) { ok = false; break; }
      const float cum_last = cumb[WQ - 1];
      // ---- acc += Sc o L ------------------------------------------------------------
      if (!walk_wait(bars + GB_SC0 + s, (hi >> 1) & 1, g.status, abort)) { ok = false; break; }
      tcgen05_fence_after_sync();
#pragma unroll
      for (int pp = 0; pp < 2; ++pp) {
        const int pc = ch * 2 + pp;
        const int j0 = pc * 32;
        if (pc > quarter) continue;                 // above the diagonal for every row of the warp
        uint32_t v[32];
        tmem_ld_32x32(tl + GT_SC + s * 128 + j0, v);
        const bool diag = pc == quarter;
        tmem_ld_wait();
        // Factors relative to the last column of each 8-column sub-piece (see the walk kernel); without a branch per sub-piece the
        // exponentials and shared-memory loads of all four overlap.
        const int last_col = diag ? lane : 31;
        float rarg[4];
#pragma unroll
        for (int sp = 0; sp < 4; ++sp) rarg[sp] = cum_r - cumb[j0 + sp * 8 + 7];
        if (!__any_sync(0xffffffffu, fmaxf(fmaxf(rarg[0], rarg[1]), fmaxf(rarg[2], rarg[3])) > 80.f)) {
#pragma unroll
          for (int sp = 0; sp < 4; ++sp) {
            const float rowf = w_exp(rarg[sp]);
            const float4 c0 = *reinterpret_cast<const float4*>(colfb + j0 + sp * 8);
            const float4 c1 = *reinterpret_cast<const float4*>(colfb + j0 + sp * 8 + 4);
            const float f[8] = {c0.x * rowf, c0.y * rowf, c0.z * rowf, c0.w * rowf, c1.x * rowf, c1.y * rowf, c1.z * rowf, c1.w * rowf};
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (sp * 8 + e <= last_col) acc[pp * 32 + sp * 8 + e] += __uint_as_float(v[sp * 8 + e]) * f[e];
          }
        } else {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (e <= last_col) acc[pp * 32 + e] += __uint_as_float(v[e]) * (w_exp(fminf(cum_r - cumb[j0 + e], 0.f)) * dtb[j0 + e]);
        }
      }
      // ---- row factors into the operand tiles, in place (the score MMA has read them) ----
      {
        const __half2 e2 = __float2half2_rn(w_exp(cum_r));
        const __half2 w2 = __float2half2_rn(w_exp(cum_last - cum_r) * dt_r);
        unsigned char* gyrow = smem + s * GG_STAGE + r * 128;
        unsigned char* xrow = gyrow + GG_TILE;
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const int off = ((ch * 4 + q4) ^ (r & 7)) << 4;
          uint4 a = *reinterpret_cast<const uint4*>(gyrow + off);
          uint4 x4 = *reinterpret_cast<const uint4*>(xrow + off);
          __half2* ha = reinterpret_cast<__half2*>(&a);
          __half2* hx = reinterpret_cast<__half2*>(&x4);
#pragma unroll
          for (int e = 0; e < 4; ++e) { ha[e] = __hmul2(ha[e], e2); hx[e] = __hmul2(hx[e], w2); }
          *reinterpret_cast<uint4*>(gyrow + off) = a;
          *reinterpret_cast<uint4*>(xrow + off) = x4;
        }
      }
      warp_arrive(bars + GB_SCALED, lane);
    }
    if (ok) {
      // ---- summed scores -> r16 operand tile ------------------------------------------
      unsigned char* prow = sGG + ch * GG_TILE + r * 128;
#pragma unroll
      for (int q8 = 0; q8 < 8; ++q8) {
        uint4 pk;
        uint32_t* ow = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const __half2 hv = __floats2half2_rn(acc[q8 * 8 + 2 * e], acc[q8 * 8 + 2 * e + 1]);
          ow[e] = *reinterpret_cast<const uint32_t*>(&hv);
        }
        *reinterpret_cast<uint4*>(prow + ((q8 ^ (r & 7)) << 4)) = pk;
      }
      warp_arrive(bars + GB_GG, lane);
      // ---- outputs ---------------------------------------------------------------------
      if (walk_wait(bars + GB_ACC, 0, g.status, abort)) {
        tcgen05_fence_after_sync();
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {   // 0: gC (staged behind B in stage 0), 1: gB (behind C in stage 1)
          unsigned char* stg = smem + which * GG_STAGE + 2 * GG_TILE + ch * GG_TILE + r * 128;
#pragma unroll
          for (int pp = 0; pp < 2; ++pp) {
            uint32_t v[32];
            tmem_ld_32x32(tl + (which ? GT_B : GT_C) + ch * 64 + pp * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              uint4 pk;
              uint32_t* ow = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const __half2 hv = __floats2half2_rn(__uint_as_float(v[q4 * 8 + 2 * e]), __uint_as_float(v[q4 * 8 + 2 * e + 1]));
                ow[e] = *reinterpret_cast<const uint32_t*>(&hv);
              }
              *reinterpret_cast<uint4*>(stg + (((pp * 4 + q4) ^ (r & 7)) << 4)) = pk;
            }
          }
        }
        warp_arrive(bars + GB_OUT, lane);
      }
    }
  }
  tcgen05_fence_before_sync();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, TC_COLS);
}

// dt*A prefix sums inside every 128-step chunk, dt, and the column factors of both walk directions, all in
// [B, H, L] order.  One CTA per (b, chunk, eight heads), one warp per head, four
// neighbouring steps per lane; dt comes in as rows of eight heads (one sector each) through shared memory, where one head per CTA
// read a sector for every value.
// Column factor of step t relative to the far end of its 8-step piece: causal exp(cum[t | 7] - cum[t]) dt[t], anti-causal
// exp(cum[t] - cum[t & ~7]); both are at most one (dt).
// RAW: the step sizes arrive as the projection's raw r16 output (row pitch `raw_pitch`) and the decay rates as A_log:
//   dt = softplus(raw + bias[h]), A = -exp(A_log[h])  (the arithmetic of launch_softplus_bias / launch_neg_exp),
// both also written out (dt_out [B, L, H], A_out [H]) for the reverse pass.
constexpr int WS_HEADS = 8;                    // heads per CTA of the two scalar kernels
constexpr int WS_THREADS = 32 * WS_HEADS;
template <bool RAW>
__global__ void __launch_bounds__(WS_THREADS) ssd_walk_cumsum_kernel(const float* __restrict__ dt, const float* __restrict__ A,
                                                                     float* __restrict__ cum, float* __restrict__ dtt,
                                                                     float* __restrict__ colf_c, float* __restrict__ colf_a, int L, int H, int hblocks,
                                                                     int* __restrict__ carry_flags, int n_flags, const __half* __restrict__ raw,
                                                                     size_t raw_pitch, const float* __restrict__ bias, float* __restrict__ dt_out,
                                                                     float* __restrict__ A_out) {
  mp_grid_dependency();
  __shared__ float s_dt[WQ][WS_HEADS + 1];
  if (blockIdx.x == 0)   // the walks that follow in stream order hand states from CTA to CTA through these counters
    for (int i = threadIdx.x; i < n_flags; i += WS_THREADS) carry_flags[i] = 0;
  const int nc = L / WQ;
  const int h0 = static_cast<int>(blockIdx.x % hblocks) * WS_HEADS, bc = blockIdx.x / hblocks, c = bc % nc, b = bc / nc;
#pragma unroll
  for (int k = 0; k < WQ * WS_HEADS / WS_THREADS; ++k) {
    const int idx = k * WS_THREADS + threadIdx.x, t = idx / WS_HEADS, h = h0 + idx % WS_HEADS;
    float d = 0.f;
    if (h < H) {
      const size_t row = static_cast<size_t>(b) * L + c * WQ + t;
      if (RAW) {
        const float pre = __half2float(raw[row * raw_pitch + h]) + bias[h];
        d = pre > 20.f ? pre : log1pf(__expf(pre));
        dt_out[row * H + h] = d;
      } else {
        d = dt[row * H + h];
      }
    }
    s_dt[t][idx % WS_HEADS] = d;
  }
  __syncthreads();
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, h = h0 + w;
  if (h >= H) return;
  const float a = RAW ? -__expf(A[h]) : A[h];
  if (RAW && bc == 0 && lane == 0) A_out[h] = a;
  float d[4], v[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    d[e] = s_dt[lane * 4 + e][w];
    v[e] = __fmul_rn(d[e], a);
  }
  // Inclusive sums of 32 steps (eight lanes) by doubling offsets, then the totals of the 32-step groups before: the order in which one
  // thread per step would add them.
  const int l8 = lane & 7;
  {
    const float p3 = __shfl_up_sync(0xffffffffu, v[3], 1);
    const float w0 = l8 >= 1 ? v[0] + p3 : v[0], w1 = v[1] + v[0], w2 = v[2] + v[1], w3 = v[3] + v[2];
    v[0] = w0; v[1] = w1; v[2] = w2; v[3] = w3;
  }
  {
    const float p2 = __shfl_up_sync(0xffffffffu, v[2], 1), p3 = __shfl_up_sync(0xffffffffu, v[3], 1);
    const float w2 = v[2] + v[0], w3 = v[3] + v[1];
    if (l8 >= 1) { v[0] += p2; v[1] += p3; }
    v[2] = w2; v[3] = w3;
  }
#pragma unroll
  for (int off = 1; off < 8; off <<= 1)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float up = __shfl_up_sync(0xffffffffu, v[e], off);
      if (l8 >= off) v[e] += up;
    }
  float base = 0.f;
#pragma unroll
  for (int g = 0; g < 3; ++g) {
    const float tot = __shfl_sync(0xffffffffu, v[3], g * 8 + 7);
    if (g < (lane >> 3)) base += tot;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] += base;
  const float c_hi = __shfl_sync(0xffffffffu, v[3], lane | 1), c_lo = __shfl_sync(0xffffffffu, v[0], lane & ~1);
  const size_t o = (static_cast<size_t>(b) * H + h) * (static_cast<size_t>(nc) * WQ) + c * WQ + lane * 4;
  *reinterpret_cast<float4*>(cum + o) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(dtt + o) = make_float4(d[0], d[1], d[2], d[3]);
  *reinterpret_cast<float4*>(colf_c + o) = make_float4(w_exp(c_hi - v[0]) * d[0], w_exp(c_hi - v[1]) * d[1], w_exp(c_hi - v[2]) * d[2], w_exp(c_hi - v[3]) * d[3]);
  if (colf_a != nullptr) *reinterpret_cast<float4*>(colf_a + o) = make_float4(w_exp(v[0] - c_lo), w_exp(v[1] - c_lo), w_exp(v[2] - c_lo), w_exp(v[3] - c_lo));
}

// ---------------------------------------------------------------------------
// gdt, gA from the walks' row dots u = <gy, y>, v = <gx, x>.  With g_a_t the gradient of the loss with respect to dt_t A_h:
//   g_a_t = g_a_{t+1} + u_t - v_t,  gdt_t = v_t / dt_t + A_h g_a_t,  gA_h = sum_t dt_t g_a_t.
// u_t - v_t cancels and carries the rounding noise of two different operator instances, so a suffix sum over the whole
// sequence random-walks (measured: gA off by 5 % at 8192 steps).  The sum is therefore pinned at every chunk boundary to a value
// without such noise, summed only inside a chunk, and the residual between a chunk's two pins is spread linearly over its steps.
//   pin(c) = g_a just behind chunk c = < what chunk c receives from its successors, what chunk c+1 receives from its predecessors >
// (ssd_boundary_dot_kernel, beside the group-gradient kernel).  Collecting it from the two kernels that hold the states was 60 us
// faster at [8, 8192, 32, 64] but takes the product at another place, and the last bits of gdt with it.
// Every chunk is then on its own: one CTA per (b, chunk, eight heads), one warp per head, four neighbouring steps per lane, and
// gdt (and graw) leave as rows of eight heads.
// With `raw` (the projection's raw step sizes, r16, pitched) the reverse of dt = softplus(raw + bias[h]) is applied on the
// way out: graw = gdt * sigmoid(raw + bias) (r16, pitched); its sums go to gb_part (the arithmetic of launch_softplus_bias_reverse).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float walk_sigmoid(float x) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
  return r;
}
struct ScalarArgs {
  const float* u; const float* v;   // [2][B, H, L]: one array per half of the columns
  const float* dtt;                 // [B, H, L]
  const float* A;
  const float* pin;                 // [B, H, nc]: g_a just behind the chunk
  float* gdt;                       // [B, L, H]
  float* ga_part; float* gb_part;   // [B * nc][H]
  const __half* raw; size_t raw_pitch; const float* bias; __half* graw; size_t graw_pitch;
  int B, L, H, nc, hblocks;
};
template <bool RAW>
__global__ void __launch_bounds__(WS_THREADS) ssd_walk_scalars_kernel(const ScalarArgs g) {
  mp_grid_dependency();
  __shared__ float s_gd[WQ][WS_HEADS + 1];
  const int h0 = static_cast<int>(blockIdx.x % g.hblocks) * WS_HEADS, bc = blockIdx.x / g.hblocks, c = bc % g.nc, b = bc / g.nc;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, h = h0 + w;
  if (h < g.H) {
    const size_t bh = static_cast<size_t>(b) * g.H + h, LP = static_cast<size_t>(g.nc) * WQ, half = static_cast<size_t>(g.B) * g.H * LP;
    const size_t o = bh * LP + c * WQ + lane * 4;
    const float4 u0 = *reinterpret_cast<const float4*>(g.u + o), u1 = *reinterpret_cast<const float4*>(g.u + half + o);
    const float4 v0 = *reinterpret_cast<const float4*>(g.v + o), v1 = *reinterpret_cast<const float4*>(g.v + half + o);
    const float4 d4 = *reinterpret_cast<const float4*>(g.dtt + o);
    const float right = g.pin[bh * g.nc + c], left = c > 0 ? g.pin[bh * g.nc + c - 1] : 0.f;   // g_a behind the chunk and at its first step
    const float vt[4] = {v0.x + v1.x, v0.y + v1.y, v0.z + v1.z, v0.w + v1.w}, dt[4] = {d4.x, d4.y, d4.z, d4.w};
    // suffix sums of u - v: 32 steps (eight lanes) by doubling offsets, then the totals of the 32-step groups behind them
    float x[4] = {u0.x + u1.x - vt[0], u0.y + u1.y - vt[1], u0.z + u1.z - vt[2], u0.w + u1.w - vt[3]};
    const int l8 = 7 - (lane & 7);
    {
      const float n0 = __shfl_down_sync(0xffffffffu, x[0], 1);
      const float w3 = l8 >= 1 ? x[3] + n0 : x[3], w2 = x[2] + x[3], w1 = x[1] + x[2], w0 = x[0] + x[1];
      x[0] = w0; x[1] = w1; x[2] = w2; x[3] = w3;
    }
    {
      const float n0 = __shfl_down_sync(0xffffffffu, x[0], 1), n1 = __shfl_down_sync(0xffffffffu, x[1], 1);
      const float w1 = x[1] + x[3], w0 = x[0] + x[2];
      if (l8 >= 1) { x[3] += n1; x[2] += n0; }
      x[0] = w0; x[1] = w1;
    }
#pragma unroll
    for (int off = 1; off < 8; off <<= 1)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float dn = __shfl_down_sync(0xffffffffu, x[e], off);
        if (l8 >= off) x[e] += dn;
      }
    float behind = 0.f;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const float tot = __shfl_sync(0xffffffffu, x[0], 24 - 8 * q);
      if (q < ((31 - lane) >> 3)) behind += tot;
    }
    float within[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) within[e] = x[e] + behind;
    const float total = __shfl_sync(0xffffffffu, within[0], 0);
    const float resid = c > 0 ? left - (right + total) : 0.f;   // what the sum misses of the pin at the chunk's first step
    const float a_h = g.A[h];
    float ga_acc = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int t = lane * 4 + e;
      const float ga = right + within[e] + resid * (static_cast<float>(WQ - t) / static_cast<float>(WQ));
      ga_acc += dt[e] * ga;
      s_gd[t][w] = vt[e] / dt[e] + a_h * ga;
    }
    ga_acc = warp_reduce<SumOp>(ga_acc);
    if (lane == 0) g.ga_part[static_cast<size_t>(bc) * g.H + h] = ga_acc;
  }
  __syncthreads();
  float gb = 0.f;
#pragma unroll
  for (int k = 0; k < WQ * WS_HEADS / WS_THREADS; ++k) {
    const int idx = k * WS_THREADS + threadIdx.x, t = idx / WS_HEADS, hh = h0 + idx % WS_HEADS;
    if (hh < g.H) {
      const size_t row = static_cast<size_t>(b) * g.L + c * WQ + t;
      const float gd = s_gd[t][idx % WS_HEADS];
      g.gdt[row * g.H + hh] = gd;
      if (RAW) {
        const float gr = gd * walk_sigmoid(__half2float(g.raw[row * g.raw_pitch + hh]) + g.bias[hh]);
        g.graw[row * g.graw_pitch + hh] = __float2half_rn(gr);
        gb += gr;
      }
    }
  }
  if (RAW) {   // a thread has one head in all its steps: threads of equal idx % 8 meet
    __shared__ float s_gb[WS_HEADS][WS_HEADS];
#pragma unroll
    for (int off = 16; off >= WS_HEADS; off >>= 1) gb += __shfl_xor_sync(0xffffffffu, gb, off);
    if (lane < WS_HEADS) s_gb[w][lane] = gb;
    __syncthreads();
    if (threadIdx.x < WS_HEADS && h0 + static_cast<int>(threadIdx.x) < g.H) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < WS_HEADS; ++q) t += s_gb[q][threadIdx.x];
      g.gb_part[static_cast<size_t>(bc) * g.H + h0 + threadIdx.x] = t;
    }
  }
}

// One CTA per head: gA[h] = the sum of its parts; with A_log's gradient wanted (A = -exp(A_log), so dA / dA_log = A)
// gA_log[h] += gA[h] * A[h]; with the step bias's gradient wanted gbias[h] += the sum of its parts.
__global__ void __launch_bounds__(128) ssd_walk_sum_parts_kernel(const float* __restrict__ ga_part, const float* __restrict__ gb_part, int parts, int H,
                                                                 const float* __restrict__ A, float* __restrict__ gA, float* __restrict__ gA_log,
                                                                 float* __restrict__ gbias) {
  mp_grid_dependency();
  __shared__ float red[64];
  const int h = blockIdx.x;
  float sa = 0.f, sb = 0.f;
  for (int i = threadIdx.x; i < parts; i += 128) {
    sa += ga_part[static_cast<size_t>(i) * H + h];
    if (gbias != nullptr) sb += gb_part[static_cast<size_t>(i) * H + h];
  }
  sa = cta_reduce<SumOp, 128>(sa, red, 0.f);
  sb = cta_reduce<SumOp, 128>(sb, red, 0.f);
  if (threadIdx.x == 0) {
    gA[h] = sa;
    if (gA_log != nullptr) gA_log[h] += sa * A[h];
    if (gbias != nullptr) atomicAdd(gbias + h, sb);   // scans on two streams may share a bias
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn walk_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    MP_CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    if (p == nullptr || q != cudaDriverEntryPointSuccess) MP_FATAL("cuTensorMapEncodeTiled is not available");
    fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// r16 matrix [rows, cols] (row-major), box {64 columns, 128 rows}, 128-byte swizzle
CUtensorMap walk_map(const void* base, size_t rows, size_t cols) {
  CUtensorMap m;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * sizeof(__half)};
  const cuuint32_t box[2] = {64, 128};
  const cuuint32_t es[2] = {1, 1};
  MP_CU_CHECK(walk_encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, es,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
  return m;
}

// r16 tensor [batch, rows, cols] (row-major), box {64 columns, 128 rows, 1}, 128-byte swizzle (64-byte with 32 columns): rows past the end of a batch
// entry read as zeros and are not written.
CUtensorMap walk_map3(const void* base, size_t batch, size_t rows, size_t cols, uint32_t box_cols = 64, uint32_t box_rows = 128) {
  CUtensorMap m;
  const cuuint64_t dims[3] = {cols, rows, batch};
  const cuuint64_t strides[2] = {cols * sizeof(__half), rows * cols * sizeof(__half)};
  const cuuint32_t box[3] = {box_cols, box_rows, 1};
  const cuuint32_t es[3] = {1, 1, 1};
  MP_CU_CHECK(walk_encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, es,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
  return m;
}

}  // namespace

// Host-side view of the chunk walk's work partition (the function the kernels use, compiled for the host): segment
// `idx` of CTA `cta` out of `ncta` for `nseq` sequences of `nc` chunks -> out = {sequence, first position, chunks,
// carried-in state, carried-out state}; returns 0 past the CTA's last segment.  For tests; needs no GPU.
extern "C" int mpSsdWalkPartition(int cta, int ncta, int nseq, int nc, int idx, int* out) {
  WalkSeg sg;
  if (ncta <= 0 || ncta > nseq || nc <= 0 || cta < 0 || cta >= ncta || idx < 0) return 0;
  if (!walk_segment(cta, ncta, nseq, nc, idx, sg)) return 0;
  out[0] = sg.seq; out[1] = sg.p0; out[2] = sg.n; out[3] = sg.cin; out[4] = sg.cout;
  return 1;
}

// ---------------------------------------------------------------------------
// Interface to the launchers in ssd.cu.
// ---------------------------------------------------------------------------
bool mp_ssd_walk_supported(int L, int H, int P, int N, int G) {
  return P == WP && N == WN && L % WQ == 0 && L > 0 && G > 0 && H % G == 0 && getenv("MP_SSD_NO_WALK") == nullptr;
}

static int walk_head_blocks(int H) { return (H + WS_HEADS - 1) / WS_HEADS; }

void mp_ssd_walk_cumsum(const float* dt, const float* A, float* cum, float* dtt, float* colf_c, float* colf_a, int B, int L, int H,
                        int* carry_flags, int n_flags, cudaStream_t st) {
  const int hb = walk_head_blocks(H);
  MpLaunch(B * (L / WQ) * hb, WS_THREADS, 0, st)(ssd_walk_cumsum_kernel<false>, dt, A, cum, dtt, colf_c, colf_a, L, H, hb, carry_flags, n_flags,
                                                            nullptr, 0, nullptr, nullptr, nullptr);
  MP_LAUNCH_CHECK();
}

// The same from the raw projection output and A_log (see the kernel); dt_out and A_out are what the reverse pass takes.
void mp_ssd_walk_cumsum_raw(const __half* raw, size_t raw_pitch, const float* bias, const float* A_log, float* dt_out, float* A_out, float* cum,
                            float* dtt, float* colf_c, int B, int L, int H, int* carry_flags, int n_flags, cudaStream_t st) {
  const int hb = walk_head_blocks(H);
  MpLaunch(B * (L / WQ) * hb, WS_THREADS, 0, st)(ssd_walk_cumsum_kernel<true>, nullptr, A_log, cum, dtt, colf_c, nullptr, L, H, hb, carry_flags,
                                                            n_flags, raw, raw_pitch, bias, dt_out, A_out);
  MP_LAUNCH_CHECK();
}

// gdt, gA (and graw, gbias, gA_log, with raw) from the row dots and the pins; ga_part, gb_part: [B * nc][H].
void mp_ssd_walk_scalars(const float* u, const float* v, const float* dtt, const float* A, const float* pin, float* gdt, float* gA, float* ga_part,
                         float* gb_part, const __half* raw, size_t raw_pitch, const float* bias, __half* graw, size_t graw_pitch, float* gbias,
                         float* gA_log, int B, int L, int H, cudaStream_t st) {
  ScalarArgs g;
  g.u = u; g.v = v; g.dtt = dtt; g.A = A; g.pin = pin; g.gdt = gdt; g.ga_part = ga_part; g.gb_part = gb_part;
  g.raw = raw; g.raw_pitch = raw_pitch; g.bias = bias; g.graw = graw; g.graw_pitch = graw_pitch;
  g.B = B; g.L = L; g.H = H; g.nc = L / WQ; g.hblocks = walk_head_blocks(H);
  const int grid = B * g.nc * g.hblocks;
  if (raw != nullptr) MpLaunch(grid, WS_THREADS, 0, st)(ssd_walk_scalars_kernel<true>, g);
  else MpLaunch(grid, WS_THREADS, 0, st)(ssd_walk_scalars_kernel<false>, g);
  MP_LAUNCH_CHECK();
  MpLaunch(H, 128, 0, st)(ssd_walk_sum_parts_kernel, ga_part, gb_part, B * g.nc, H, A, gA, gA_log, raw != nullptr ? gbias : nullptr);
  MP_LAUNCH_CHECK();
}

// One walk.  q, k: [B*L, G*128]; v, z, out: [B*L, H*64]; cum, dtt, colf (of the walk's direction): [B, H, L] from mp_ssd_walk_cumsum.
void mp_ssd_walk(int anti, const __half* q, const __half* k, const __half* v, const float* cum, const float* dtt, const float* colf, __half* out,
                 const __half* z,
                 float* dot_out, __half* hs_out, float* carry, int* carry_flag, int max_ctas, int B, int L, int H, int G, uint32_t* status,
                 cudaStream_t st) {
  WalkArgs g;
  g.B = B; g.L = L; g.H = H; g.G = G; g.nc = L / WQ;
  g.cum = cum; g.dtt = dtt; g.colf = colf; g.out = out; g.z = z; g.dot_out = dot_out; g.hs_out = hs_out; g.status = status;
  g.carry = carry; g.carry_flag = carry_flag;
  // One CTA per SM slot it may use, every CTA the same number of chunks; never more CTAs than sequences, so that a CTA's
  // range is at least one sequence long (see walk_segment).  MP_SSD_WALK_PER_SEQUENCE: one CTA per sequence, no hand-off.
  // Two heads at a time where their group has an even number of heads and there are enough sequences: a chunk of a pair takes 1.4
  // times as long as a chunk of one head (4.3 against 3.05 us in the forward), which pays unless CTAs are left without a sequence; at
  // 192 sequences on 148 CTAs, a ratio of 1.297, both take 80 us.  The pair kernel counts steps in 32 bits.
  // MP_SSD_WALK_NO_PAIRS: one head at a time, for an A/B.
  const bool bounded = max_ctas > 0 && getenv("MP_SSD_WALK_PER_SEQUENCE") == nullptr;
  auto load = [&](int seqs) { return bounded && seqs > max_ctas ? static_cast<double>(seqs) / max_ctas : 1.0; };   // sequences per CTA
  const bool pairs = (H / G) % 2 == 0 && static_cast<size_t>(B) * H * g.nc * WQ < (size_t{1} << 31) && 1.4 * load(B * H / 2) < load(B * H) &&
                     getenv("MP_SSD_WALK_NO_PAIRS") == nullptr;
  int grid = pairs ? B * H / 2 : B * H;
  if (bounded && max_ctas < grid) grid = max_ctas;
  const CUtensorMap mq = walk_map3(q, B, L, static_cast<size_t>(G) * WN), mk = walk_map3(k, B, L, static_cast<size_t>(G) * WN);
  const CUtensorMap mv = walk_map3(v, B, L, static_cast<size_t>(H) * WP);
  const CUtensorMap mh = hs_out != nullptr ? walk_map(hs_out, static_cast<size_t>(B) * H * g.nc * WN, WP) : mv;
  auto launch = [&](auto kernel, auto pair_kernel) {
    if (pairs) {
      const CUtensorMap mz = z != nullptr ? walk_map3(z, B, L, static_cast<size_t>(H) * WP, 32, 128) : mv;
      const CUtensorMap mo = out != nullptr ? walk_map3(out, B, L, static_cast<size_t>(H) * WP, 32, 32) : mv;
      MP_CUDA_CHECK(cudaFuncSetAttribute(pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WP2_SMEM_BYTES));
      MpLaunch(grid, WP2_THREADS, WP2_SMEM_BYTES, st)(pair_kernel, mq, mk, mv, mh, mz, mo, g);
    } else {
      MP_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, W_SMEM_BYTES));
      MpLaunch(grid, W_THREADS, W_SMEM_BYTES, st)(kernel, mq, mk, mv, mh, g);
    }
  };
  const bool dot = z != nullptr && dot_out != nullptr;
  if (!dot) { g.z = nullptr; g.dot_out = nullptr; }
  if (anti && !dot) MP_FATAL("ssd walk: the anti-causal form comes with its row dots");
  auto form = [&](auto A, auto D) {
    constexpr int a = decltype(A)::value;
    constexpr bool d = decltype(D)::value;
    launch(ssd_walk_kernel<a, d>, ssd_walk_pair_kernel<a, d>);
  };
  using std::integral_constant;
  if (anti) form(integral_constant<int, 1>{}, std::true_type{});
  else if (dot) form(integral_constant<int, 0>{}, std::true_type{});
  else form(integral_constant<int, 0>{}, std::false_type{});
  MP_LAUNCH_CHECK();
}

// gB, gC [B*L, G*128] from gy, x [B*L, H*64], Bm, Cm [B*L, G*128] and the states left by the two walks
// (hs_causal, hs_anti: [B, H, nc][128][64]).
void mp_ssd_group_grads(const __half* gy, const __half* x, const __half* Bm, const __half* Cm, const __half* hs_causal, const __half* hs_anti,
                        const float* cum, const float* dtt, const float* colf_c, __half* gB, __half* gC, int B, int L,
                        int H, int G, uint32_t* status, cudaStream_t st) {
  GroupArgs g;
  g.B = B; g.L = L; g.H = H; g.G = G; g.nc = L / WQ;
  g.cum = cum; g.dtt = dtt; g.colf = colf_c; g.status = status;
  const size_t srows = static_cast<size_t>(B) * H * g.nc * WN;
  const CUtensorMap mgy = walk_map3(gy, B, L, static_cast<size_t>(H) * WP), mx = walk_map3(x, B, L, static_cast<size_t>(H) * WP);
  const CUtensorMap mhc = walk_map(hs_causal, srows, WP), mha = walk_map(hs_anti, srows, WP);
  const CUtensorMap mb = walk_map3(Bm, B, L, static_cast<size_t>(G) * WN), mc = walk_map3(Cm, B, L, static_cast<size_t>(G) * WN);
  const CUtensorMap mgb = walk_map3(gB, B, L, static_cast<size_t>(G) * WN), mgc = walk_map3(gC, B, L, static_cast<size_t>(G) * WN);
  MP_CUDA_CHECK(cudaFuncSetAttribute(ssd_group_grads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, GG_SMEM_BYTES));
  MpLaunch(B * g.nc * G, W_THREADS, GG_SMEM_BYTES, st)(ssd_group_grads_kernel, mgy, mx, mhc, mha, mb, mc, mgb, mgc, g);
  MP_LAUNCH_CHECK();
}
