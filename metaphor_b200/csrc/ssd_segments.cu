// Mamba-2 SSD scan of r16 tensors with fp32 arithmetic throughout, over segments of 64 steps that run side by side (head size 64,
// state 128, any number of steps).  It serves the calls that whole tensor-core chunks do not cover: lengths that are no multiple of
// the chunk, and other chunk lengths; pointers need no more than the alignment of their elements.  Its results are those of the
// recurrence (ssd_generic.cu) to the accuracy of fp32 sums: weights, scores and states are never rounded to r16, and A's gradient is a sum of the
// products that make it up, not a difference of row dots, so that it keeps its digits where almost nothing is carried from step to
// step ([2, 200, 16] with step sizes around 2: the r16 chunk walk is off by 0.6 of gA and 0.03 of gdt, this by 1.4e-7 and 1.3e-7).
//
// With cum the inclusive prefix sums of dt A inside a segment (differences of them taken in r64), E their last value, H the state a
// segment receives from its predecessors and Y the adjoint state it receives from its successors:
//   M_ij = exp(cum_i - cum_j) (i >= j),  G = C B^T,  X = gy x^T,  e_j = exp(E - cum_j)
//   y_i  = sum_j M G dt_j x_j + exp(cum_i) H^T C_i
//   gx_j = dt_j (sum_i M G gy_i + e_j Y^T B_j)
//   gC_i = sum_j M X dt_j B_j + exp(cum_i) H gy_i            gB_j = dt_j (sum_i M X C_i + e_j Y x_j)
//   s_j  = sum_i M G X + e_j <B_j, Y x_j>
//   ga_t = sum_{i >= t > j} M G X dt_j + sum_{i >= t} exp(cum_i) <C_i, H gy_i> + sum_{j < t} dt_j e_j <B_j, Y x_j> + exp(E) <Y, H>
//   gdt_t = s_t + A ga_t,   gA = sum_t dt_t ga_t
// Launches: states made inside every segment, both directions (segment_states); carried from segment to segment, element by element
// (segment_carry); outputs (segment_forward / segment_reverse); for the reverse two folds.
//
// What bounds it is the FP pipe with its shared-memory operands: 1.5 M (forward) and 3.7 M (reverse) multiply-adds per head and segment,
// states included; at a third of the pipe's peak, since the reverse's tiles leave room for one CTA of eight warps per SM.
// Forward / reverse in us, the recurrence -> segments (the chunk walk on padded chunks, with its r16 losses):
//   [2, 1000, 24] 1 806 / 41 544 -> 97 / 259 (29 / 82),   [8, 8191, 32] 41 650 / 800 600 -> 3 945 / 8 951 (279 / 923),
//   [2, 32, 24] 62 / 1 260 -> 9.5 / 24 (11 / 60),   [1, 100, 2] 182 / 3 957 -> 22 / 38 (11 / 33).
// Below 32 steps the recurrence stays (60 / 1 214 us at [2, 31, 24]): its forward needs no scratch, and callers may rely on that.
#include "mp_common.cuh"

namespace {

constexpr int SG_Q = 64;              // steps per segment
constexpr int SG_N = 128, SG_P = 64;  // state size, head size
constexpr int SG_THREADS = 256;
constexpr int SG_NPITCH = SG_N + 4, SG_PPITCH = SG_P + 4;   // floats per row of a shared tile: rows 16 bytes apart in the banks
constexpr int SG_STATE = SG_N * SG_P;

struct SegArgs {
  const __half* x; const float* dt; const float* A; const __half* Bm; const __half* Cm; const __half* gy;
  __half* y;                 // forward
  __half* gx; float* gdt;    // reverse
  float* states;             // [B H][nseg][128][64]: causal states; the adjoint ones follow in the reverse
  float* decay;              // [B H][nseg]: exp(E)
  float* ga_part;            // [B H][nseg]
  float* gb_part;            // [splits][B L G][128] sums over the heads of a split, gB then gC
  int B, L, H, G, nseg, splits;
  bool vec;                  // every r16 pointer is 16-byte aligned
};

// Scalars of a segment, by one warp: cum[64] (r64) and dt[64]; steps past the sequence do not decay and have dt = 0.
__device__ __forceinline__ void segment_scalars(const SegArgs& g, int b, int h, int t0, double* cum, float* dt, int lane) {
  const double a = static_cast<double>(g.A[h]);
  const int t = t0 + 2 * lane;
  const float* src = g.dt + (static_cast<size_t>(b) * g.L + t) * g.H + h;
  const float d0 = t < g.L ? src[0] : 0.f, d1 = t + 1 < g.L ? src[g.H] : 0.f;
  const double v0 = d0 * a, v1 = d1 * a;
  double s = v0 + v1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double up = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += up;
  }
  cum[2 * lane] = s - v1;
  cum[2 * lane + 1] = s;
  dt[2 * lane] = d0;
  dt[2 * lane + 1] = d1;
}
__device__ __forceinline__ float segment_exp(double v) { return expf(static_cast<float>(v)); }

// [64 steps][COLS] of r16 -> fp32 tile; `scale`: a factor per step or null.  Steps past the sequence become zeros.
template <int COLS, int PITCH>
__device__ __forceinline__ void segment_tile(float* dst, const __half* src, size_t pitch, int rows, bool vec, const float* scale) {
#pragma unroll
  for (int k = 0; k < SG_Q * COLS / 8 / SG_THREADS; ++k) {
    const int idx = k * SG_THREADS + threadIdx.x, r = idx / (COLS / 8), c = idx % (COLS / 8) * 8;
    float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (r < rows) {
      const __half* p = src + r * pitch + c;
      if (vec) {
        unpack<__half>(ld_pack(p, 0), f);
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __half2float(p[e]);
      }
      if (scale != nullptr) {
        const float s = scale[r];
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= s;
      }
    }
    float4* o = reinterpret_cast<float4*>(dst + r * PITCH + c);
    o[0] = make_float4(f[0], f[1], f[2], f[3]);
    o[1] = make_float4(f[4], f[5], f[6], f[7]);
  }
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float at(const float4& v, int e) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; }   // e is a constant

// A state [128][64] in shared memory: rows of 64 floats, the sixteen 16-byte pieces of a row exchanged by bits 2 .. 5 of the row, so that
// neighbouring groups of four rows can be read at one piece without bank conflicts.
__device__ __forceinline__ int state_at(int n, int p4) { return n * SG_P + ((p4 ^ ((n >> 2) & 15)) << 2); }

// Four neighbouring r16 outputs.
__device__ __forceinline__ void segment_store(__half* dst, const float* v, bool vec) {
  if (vec) {
    const __half2 lo = __floats2half2_rn(v[0], v[1]), hi = __floats2half2_rn(v[2], v[3]);
    uint2 u;
    u.x = *reinterpret_cast<const uint32_t*>(&lo);
    u.y = *reinterpret_cast<const uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(dst) = u;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) dst[e] = __float2half_rn(v[e]);
  }
}

// What a segment adds to the state behind it (blockIdx.y = 0) and to the adjoint state before it (1).
// Threads: eight state rows x four head columns each.
__global__ void __launch_bounds__(SG_THREADS) segment_states_kernel(const SegArgs g) {
  mp_grid_dependency();
  extern __shared__ __align__(16) float seg_smem[];
  float* sK = seg_smem;                         // [64][132] B or C
  float* sV = sK + SG_Q * SG_NPITCH;            // [64][68] x or gy, scaled
  double* cum = reinterpret_cast<double*>(sV + SG_Q * SG_PPITCH);
  float* dt = reinterpret_cast<float*>(cum + SG_Q);
  float* w = dt + SG_Q;
  const bool anti = blockIdx.y != 0;
  const int seq = blockIdx.x / g.nseg, seg = blockIdx.x % g.nseg, b = seq / g.H, h = seq % g.H, grp = h / (g.H / g.G);
  const int t0 = seg * SG_Q, rows = min(SG_Q, g.L - t0);
  if (threadIdx.x < 32) {
    segment_scalars(g, b, h, t0, cum, dt, threadIdx.x);
    __syncwarp();
    const double last = cum[SG_Q - 1];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = 2 * threadIdx.x + e;
      w[t] = anti ? segment_exp(cum[t]) : dt[t] * segment_exp(last - cum[t]);
    }
    if (threadIdx.x == 0 && !anti) g.decay[blockIdx.x] = segment_exp(last);
  }
  if (anti ? seg == 0 : seg == g.nseg - 1) return;   // nothing lies beyond
  __syncthreads();
  const size_t row = static_cast<size_t>(b) * g.L + t0;
  segment_tile<SG_N, SG_NPITCH>(sK, (anti ? g.Cm : g.Bm) + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec, nullptr);
  segment_tile<SG_P, SG_PPITCH>(sV, (anti ? g.gy : g.x) + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows, g.vec, w);
  __syncthreads();
  const int n0 = threadIdx.x / 16 * 8, p0 = threadIdx.x % 16 * 4;
  float acc[8][4] = {};
#pragma unroll 4
  for (int k = 0; k < SG_Q; ++k) {
    const float4 a0 = ld4(sK + k * SG_NPITCH + n0), a1 = ld4(sK + k * SG_NPITCH + n0 + 4), v = ld4(sV + k * SG_PPITCH + p0);
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(r < 4 ? at(a0, r) : at(a1, r - 4), at(v, c), acc[r][c]);
  }
  float* out = g.states + (static_cast<size_t>(anti) * g.B * g.H * g.nseg + blockIdx.x) * SG_STATE;
#pragma unroll
  for (int r = 0; r < 8; ++r) *reinterpret_cast<float4*>(out + (n0 + r) * SG_P + p0) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
}

// In place: what every segment adds becomes what every segment receives.  One thread per four elements of a sequence's state.
__global__ void __launch_bounds__(SG_THREADS) segment_carry_kernel(const SegArgs g) {
  mp_grid_dependency();
  const bool anti = blockIdx.y != 0;
  constexpr int PER = SG_STATE / 4 / SG_THREADS;   // CTAs per sequence
  const int seq = blockIdx.x / PER, e = (blockIdx.x % PER) * SG_THREADS + threadIdx.x;
  float4* st = reinterpret_cast<float4*>(g.states + (static_cast<size_t>(anti) * g.B * g.H + seq) * g.nseg * SG_STATE) + e;
  const float* decay = g.decay + static_cast<size_t>(seq) * g.nseg;
  constexpr size_t STEP = SG_STATE / 4;
  float4 carry = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s0 = 0; s0 < g.nseg; s0 += 4) {
    float4 add[4];
    float d[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {      // (the last segment in walk order has nothing to add)
      const int s = anti ? g.nseg - 1 - s0 - u : s0 + u;
      const bool live = s0 + u < g.nseg - 1;
      add[u] = live ? st[s * STEP] : make_float4(0.f, 0.f, 0.f, 0.f);
      d[u] = live ? decay[s] : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (s0 + u >= g.nseg) break;
      const int s = anti ? g.nseg - 1 - s0 - u : s0 + u;
      st[s * STEP] = carry;
      carry = make_float4(fmaf(d[u], carry.x, add[u].x), fmaf(d[u], carry.y, add[u].y), fmaf(d[u], carry.z, add[u].z), fmaf(d[u], carry.w, add[u].w));
    }
  }
}

// State of a segment from global to shared memory (see state_at).
__device__ __forceinline__ void segment_load_state(float* dst, const float* src) {
#pragma unroll
  for (int k = 0; k < SG_STATE / 4 / SG_THREADS; ++k) {
    const int idx = k * SG_THREADS + threadIdx.x, n = idx / (SG_P / 4), p4 = idx % (SG_P / 4);
    *reinterpret_cast<float4*>(dst + state_at(n, p4)) = *reinterpret_cast<const float4*>(src + idx * 4);
  }
}

// Scores a_i b_j^T of the 16 x 16 blocks on and below the diagonal: thread (ty, tx) has i = ty + 16 u, j = tx + 16 v.
template <int K, int PITCH>
__device__ __forceinline__ void segment_scores(const float* a, const float* b, int ty, int tx, float (&acc)[4][4]) {
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = 0.f;
  // sixteen products at a time: the sums of the long chain would carry most of gdt's error (2.5e-7 of its norm with one chain)
#pragma unroll 1
  for (int k0 = 0; k0 < K; k0 += 16) {
    float part[4][4] = {};
#pragma unroll
    for (int k = k0; k < k0 + 16; k += 4) {
      float4 av[4], bv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) { av[u] = ld4(a + (ty + 16 * u) * PITCH + k); bv[u] = ld4(b + (tx + 16 * u) * PITCH + k); }
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v <= u; ++v)
#pragma unroll
          for (int e = 0; e < 4; ++e) part[u][v] = fmaf(at(av[u], e), at(bv[v], e), part[u][v]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v <= u; ++v) acc[u][v] += part[u][v];
  }
}

// y of one (sequence, segment).  Thread (ty, tx): four rows 16 apart or next to each other, four columns.
__global__ void __launch_bounds__(SG_THREADS, 2) segment_forward_kernel(const SegArgs g) {
  mp_grid_dependency();
  extern __shared__ __align__(16) float seg_smem[];
  float* sC = seg_smem;                          // [64][132]
  float* sB = sC + SG_Q * SG_NPITCH;             // [64][132], then the state [128][64]
  float* sX = sB + SG_Q * SG_NPITCH;             // [64][68]
  float* sW = sX + SG_Q * SG_PPITCH;             // [64][68]
  double* cum = reinterpret_cast<double*>(sW + SG_Q * SG_PPITCH);
  float* dt = reinterpret_cast<float*>(cum + SG_Q);
  const int seq = blockIdx.x / g.nseg, seg = blockIdx.x % g.nseg, b = seq / g.H, h = seq % g.H, grp = h / (g.H / g.G);
  const int t0 = seg * SG_Q, rows = min(SG_Q, g.L - t0);
  const size_t row = static_cast<size_t>(b) * g.L + t0;
  if (threadIdx.x < 32) segment_scalars(g, b, h, t0, cum, dt, threadIdx.x);
  segment_tile<SG_N, SG_NPITCH>(sC, g.Cm + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec, nullptr);
  segment_tile<SG_N, SG_NPITCH>(sB, g.Bm + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec, nullptr);
  segment_tile<SG_P, SG_PPITCH>(sX, g.x + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows, g.vec, nullptr);
  __syncthreads();
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  {
    float s[4][4];
    segment_scores<SG_N, SG_NPITCH>(sC, sB, ty, tx, s);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v <= u; ++v) {
        const int i = ty + 16 * u, j = tx + 16 * v;
        sW[i * SG_PPITCH + j] = s[u][v] * segment_exp(cum[i] - cum[j]) * dt[j];   // (read for j <= i)
      }
  }
  __syncthreads();
  if (seg > 0) segment_load_state(sB, g.states + static_cast<size_t>(blockIdx.x) * SG_STATE);
  const int p0 = tx * 4;
  float acc[4][4] = {};
#pragma unroll
  for (int jb = 0; jb < 4; ++jb) {
#pragma unroll 2
    for (int j = jb * 16; j < jb * 16 + 16; j += 4) {
      float4 v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = ld4(sX + (j + e) * SG_PPITCH + p0);
#pragma unroll
      for (int u = jb; u < 4; ++u) {
        const float4 w = ld4(sW + (ty + 16 * u) * SG_PPITCH + j);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (u == jb && j + e > ty + 16 * u) continue;   // left out, not multiplied by zero: a later step may be infinite
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[u][c] = fmaf(at(w, e), at(v[e], c), acc[u][c]);
        }
      }
    }
  }
  if (seg > 0) {
    __syncthreads();
    float st[4][4] = {};
#pragma unroll 2
    for (int n = 0; n < SG_N; n += 4) {
      float4 v[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = ld4(sB + state_at(n + e, tx));
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 w = ld4(sC + (ty + 16 * u) * SG_NPITCH + n);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int c = 0; c < 4; ++c) st[u][c] = fmaf(at(w, e), at(v[e], c), st[u][c]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float f = segment_exp(cum[ty + 16 * u]);
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[u][c] = fmaf(f, st[u][c], acc[u][c]);
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int i = ty + 16 * u;
    if (i < rows) segment_store(g.y + ((row + i) * g.H + h) * SG_P + p0, acc[u], g.vec);
  }
}

// Gradients of one (batch entry, segment, group, share of the group's heads); gB and gC of the share stay in registers.
// Thread (ty, tx): scores as in segment_scores; everything else rows 4 ty .. 4 ty + 3, head columns 4 tx .. 4 tx + 3, state columns
// 4 tx .. 4 tx + 3 and those 64 further.
__global__ void __launch_bounds__(SG_THREADS, 1) segment_reverse_kernel(const SegArgs g) {
  mp_grid_dependency();
  extern __shared__ __align__(16) float seg_smem[];
  float* sB = seg_smem;                          // [64][132]
  float* sC = sB + SG_Q * SG_NPITCH;             // [64][132]
  float* sG = sC + SG_Q * SG_NPITCH;             // [64][68] G
  float* sMG = sG + SG_Q * SG_PPITCH;            // [64][68] M G
  float* sMX = sMG + SG_Q * SG_PPITCH;           // [64][68] M X
  float* sX = sMX + SG_Q * SG_PPITCH;            // [64][68]
  float* sGy = sX + SG_Q * SG_PPITCH;            // [64][68]
  float* sS = sGy + SG_Q * SG_PPITCH;            // [128][64] state: Y, then H
  double* cum = reinterpret_cast<double*>(sS + SG_STATE);
  float* dt = reinterpret_cast<float*>(cum + SG_Q);
  float* su = dt + SG_Q;                         // [64] exp(cum_i) <C_i, H gy_i>
  float* sv = su + SG_Q;                         // [64] e_j <B_j, Y x_j>
  float* part = sv + SG_Q;                       // [2][8 warps][64]: parts of s and ga from inside the segment
  float* red = part + 2 * 8 * SG_Q;              // [8]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  const int hpg = g.H / g.G;
  const int split = blockIdx.x % g.splits;
  int rest = blockIdx.x / g.splits;
  const int grp = rest % g.G;
  rest /= g.G;
  const int seg = rest % g.nseg, b = rest / g.nseg;
  const int t0 = seg * SG_Q, rows = min(SG_Q, g.L - t0);
  const bool before = seg > 0, behind = seg < g.nseg - 1;
  const size_t row = static_cast<size_t>(b) * g.L + t0;
  const int r0 = ty * 4, c0 = tx * 4, rb = ty / 4 * 16;   // rb: first row of the 16-row block (the same for a whole warp)
  segment_tile<SG_N, SG_NPITCH>(sB, g.Bm + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec, nullptr);
  segment_tile<SG_N, SG_NPITCH>(sC, g.Cm + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec, nullptr);
  __syncthreads();
  {
    float s[4][4];
    segment_scores<SG_N, SG_NPITCH>(sC, sB, ty, tx, s);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v <= u; ++v) sG[(ty + 16 * u) * SG_PPITCH + tx + 16 * v] = s[u][v];
  }
  float gB[4][8] = {}, gC[4][8] = {};
  const int h_first = grp * hpg + static_cast<int>(static_cast<long long>(hpg) * split / g.splits);
  const int h_end = grp * hpg + static_cast<int>(static_cast<long long>(hpg) * (split + 1) / g.splits);
#pragma unroll 1
  for (int h = h_first; h < h_end; ++h) {
    const size_t unit = (static_cast<size_t>(b) * g.H + h) * g.nseg + seg;
    const float* hstate = g.states + unit * SG_STATE;
    const float* ystate = g.states + (static_cast<size_t>(g.B) * g.H * g.nseg + unit) * SG_STATE;
    __syncthreads();   // the previous head's tiles and scalars have been read (and sG is complete)
    if (warp == 0) segment_scalars(g, b, h, t0, cum, dt, lane);
    segment_tile<SG_P, SG_PPITCH>(sX, g.x + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows, g.vec, nullptr);
    segment_tile<SG_P, SG_PPITCH>(sGy, g.gy + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows, g.vec, nullptr);
    if (behind) segment_load_state(sS, ystate);
    __syncthreads();
    {
      float s[4][4];
      segment_scores<SG_P, SG_PPITCH>(sGy, sX, ty, tx, s);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v <= u; ++v) {
          const int i = ty + 16 * u, j = tx + 16 * v, o = i * SG_PPITCH + j;
          const float m = segment_exp(cum[i] - cum[j]);   // (read for j <= i)
          sMX[o] = m * s[u][v];
          sMG[o] = m * sG[o];
        }
    }
    __syncthreads();
    const double last = cum[SG_Q - 1];
    {   // s and ga from inside the segment: a warp takes eight rows, a lane two columns
      const float d0 = dt[2 * lane], d1 = dt[2 * lane + 1];
      float s0 = 0.f, s1 = 0.f, g0 = 0.f, g1 = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int i = warp * 8 + k, o = i * SG_PPITCH + 2 * lane;
        const float w0 = 2 * lane <= i ? sMX[o] * sG[o] : 0.f, w1 = 2 * lane + 1 <= i ? sMX[o + 1] * sG[o + 1] : 0.f;
        s0 += w0;
        s1 += w1;
        const float q0 = d0 * w0, mine = q0 + d1 * w1;
        float sum = mine;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const float up = __shfl_up_sync(0xffffffffu, sum, off);
          if (lane >= off) sum += up;
        }
        float ex = __shfl_up_sync(0xffffffffu, sum, 1);   // the columns left of this lane's
        if (lane == 0) ex = 0.f;
        if (2 * lane <= i) g0 += ex;
        if (2 * lane + 1 <= i) g1 += ex + q0;
      }
      part[warp * SG_Q + 2 * lane] = s0;
      part[warp * SG_Q + 2 * lane + 1] = s1;
      part[(8 + warp) * SG_Q + 2 * lane] = g0;
      part[(8 + warp) * SG_Q + 2 * lane + 1] = g1;
    }
    float e[4], dr[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) { e[r] = segment_exp(last - cum[r0 + r]); dr[r] = dt[r0 + r]; }
    {   // ---- gx ----
      float acc[4][4] = {};
      auto step = [&](int i, bool diag) {   // diag: steps before the row are left out, not multiplied by zero
        const float4 w = ld4(sMG + i * SG_PPITCH + r0), v = ld4(sGy + i * SG_PPITCH + c0);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (diag && i < r0 + r) continue;
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(at(w, r), at(v, c), acc[r][c]);
        }
      };
#pragma unroll 4
      for (int i = rb; i < rb + 16; ++i) step(i, true);
#pragma unroll 4
      for (int i = rb + 16; i < SG_Q; ++i) step(i, false);
      if (behind) {
        float st[4][4] = {};
#pragma unroll 2
        for (int n = 0; n < SG_N; n += 4) {
          float4 v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = ld4(sS + state_at(n + k, tx));
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float4 w = ld4(sB + (r0 + r) * SG_NPITCH + n);
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
              for (int c = 0; c < 4; ++c) st[r][c] = fmaf(at(w, k), at(v[k], c), st[r][c]);
          }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(e[r], st[r][c], acc[r][c]);
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] *= dr[r];
        if (r0 + r < rows) segment_store(g.gx + ((row + r0 + r) * g.H + h) * SG_P + c0, acc[r], g.vec);
      }
    }
    // state v of rows of `t` (x or gy): [4 rows][8 state columns]
    auto state_rows = [&](const float* t, float (&o)[4][8]) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) o[r][c] = 0.f;
#pragma unroll 1
      for (int p4 = 0; p4 < SG_P / 4; ++p4) {
        float4 w[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) w[r] = ld4(t + (r0 + r) * SG_PPITCH + p4 * 4);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const float4 v = ld4(sS + state_at(c0 + (c & 3) + (c >> 2) * 64, p4));
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int k = 0; k < 4; ++k) o[r][c] = fmaf(at(w[r], k), at(v, k), o[r][c]);
        }
      }
    };
    // <rows of `t` (B or C), o> over the sixteen threads of a row
    auto row_dots = [&](const float* t, const float (&o)[4][8], float* out) {
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4 w0 = ld4(t + (r0 + r) * SG_NPITCH + c0), w1 = ld4(t + (r0 + r) * SG_NPITCH + 64 + c0);
        float d = 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) d += at(w0, c) * o[r][c] + at(w1, c) * o[r][4 + c];
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
        if (tx == 0) out[r0 + r] = d;
      }
    };
    float o[4][8];
    {   // ---- gB ----
      if (behind) {
        state_rows(sX, o);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 8; ++c) o[r][c] *= e[r];
        row_dots(sB, o, sv);
      } else {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 8; ++c) o[r][c] = 0.f;
        if (tx == 0)
#pragma unroll
          for (int r = 0; r < 4; ++r) sv[r0 + r] = 0.f;
      }
      auto step = [&](int i, bool diag) {
        const float4 w = ld4(sMX + i * SG_PPITCH + r0), v0 = ld4(sC + i * SG_NPITCH + c0), v1 = ld4(sC + i * SG_NPITCH + 64 + c0);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (diag && i < r0 + r) continue;
#pragma unroll
          for (int c = 0; c < 8; ++c) o[r][c] = fmaf(at(w, r), c < 4 ? at(v0, c) : at(v1, c - 4), o[r][c]);
        }
      };
#pragma unroll 2
      for (int i = rb; i < rb + 16; ++i) step(i, true);
#pragma unroll 2
      for (int i = rb + 16; i < SG_Q; ++i) step(i, false);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) gB[r][c] = fmaf(dr[r], o[r][c], gB[r][c]);
    }
    __syncthreads();   // Y has been read
    float pin = 0.f;
    if (before) {
#pragma unroll
      for (int k = 0; k < SG_STATE / 4 / SG_THREADS; ++k) {
        const int idx = k * SG_THREADS + threadIdx.x, n = idx / (SG_P / 4), p4 = idx % (SG_P / 4);
        const float4 v = *reinterpret_cast<const float4*>(hstate + idx * 4);
        if (behind) {
          const float4 w = *reinterpret_cast<const float4*>(ystate + idx * 4);
          pin += v.x * w.x + v.y * w.y + v.z * w.z + v.w * w.w;
        }
        *reinterpret_cast<float4*>(sS + state_at(n, p4)) = v;
      }
      pin = warp_reduce<SumOp>(pin);
    }
    if (lane == 0) red[warp] = pin;
    __syncthreads();
    {   // ---- gC ----
      if (before) {
        state_rows(sGy, o);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float f = segment_exp(cum[r0 + r]);
#pragma unroll
          for (int c = 0; c < 8; ++c) o[r][c] *= f;
        }
        row_dots(sC, o, su);
      } else {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 8; ++c) o[r][c] = 0.f;
        if (tx == 0)
#pragma unroll
          for (int r = 0; r < 4; ++r) su[r0 + r] = 0.f;
      }
      auto steps = [&](int j, bool diag) {
        const float4 d4 = ld4(dt + j);
        float4 w[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          w[r] = ld4(sMX + (r0 + r) * SG_PPITCH + j);
          w[r].x *= d4.x; w[r].y *= d4.y; w[r].z *= d4.z; w[r].w *= d4.w;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float4 v0 = ld4(sB + (j + k) * SG_NPITCH + c0), v1 = ld4(sB + (j + k) * SG_NPITCH + 64 + c0);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            if (diag && j + k > r0 + r) continue;
#pragma unroll
            for (int c = 0; c < 8; ++c) o[r][c] = fmaf(at(w[r], k), c < 4 ? at(v0, c) : at(v1, c - 4), o[r][c]);
          }
        }
      };
#pragma unroll 1
      for (int j = 0; j < rb; j += 4) steps(j, false);
#pragma unroll 1
      for (int j = rb; j < rb + 16; j += 4) steps(j, true);
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 8; ++c) gC[r][c] += o[r][c];
    }
    __syncthreads();   // su, sv, red
    if (warp == 0) {   // ---- gdt, gA ----
      const int t = 2 * lane;
      float s0 = sv[t], s1 = sv[t + 1], ga0 = 0.f, ga1 = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        s0 += part[w * SG_Q + t];
        s1 += part[w * SG_Q + t + 1];
        ga0 += part[(8 + w) * SG_Q + t];
        ga1 += part[(8 + w) * SG_Q + t + 1];
      }
      const float u0 = su[t], u1 = su[t + 1], d0 = dt[t], d1 = dt[t + 1], v0 = d0 * sv[t], v1 = d1 * sv[t + 1];
      float suf = u0 + u1, pre = v0 + v1;   // sums over this lane's steps and those behind / before them
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const float dn = __shfl_down_sync(0xffffffffu, suf, off), up = __shfl_up_sync(0xffffffffu, pre, off);
        if (lane + off < 32) suf += dn;
        if (lane >= off) pre += up;
      }
      float suf1 = __shfl_down_sync(0xffffffffu, suf, 1), pre0 = __shfl_up_sync(0xffffffffu, pre, 1);
      if (lane == 31) suf1 = 0.f;
      if (lane == 0) pre0 = 0.f;
      float through = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) through += red[w];
      through *= segment_exp(last);
      ga0 += suf + pre0 + through;
      ga1 += u1 + suf1 + pre0 + v0 + through;
      const float a = g.A[h];
      float* gdt = g.gdt + (row + t) * g.H + h;
      if (t < rows) gdt[0] = fmaf(a, ga0, s0);
      if (t + 1 < rows) gdt[g.H] = fmaf(a, ga1, s1);
      const float sum = warp_reduce<SumOp>(d0 * ga0 + d1 * ga1);
      if (lane == 0) g.ga_part[unit] = sum;
    }
  }
  const size_t bc = static_cast<size_t>(g.B) * g.L * g.G * SG_N;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    if (r0 + r >= rows) continue;
    float* o = g.gb_part + static_cast<size_t>(split) * 2 * bc + ((row + r0 + r) * g.G + grp) * SG_N + c0;
    *reinterpret_cast<float4*>(o) = make_float4(gB[r][0], gB[r][1], gB[r][2], gB[r][3]);
    *reinterpret_cast<float4*>(o + 64) = make_float4(gB[r][4], gB[r][5], gB[r][6], gB[r][7]);
    *reinterpret_cast<float4*>(o + bc) = make_float4(gC[r][0], gC[r][1], gC[r][2], gC[r][3]);
    *reinterpret_cast<float4*>(o + bc + 64) = make_float4(gC[r][4], gC[r][5], gC[r][6], gC[r][7]);
  }
}

// gB (blockIdx.y = 0) and gC (1): the sums of the head shares, rounded; four neighbouring values per thread.
__global__ void __launch_bounds__(SG_THREADS) segment_fold_kernel(const float* __restrict__ part, __half* gB, __half* gC, size_t bc, int splits, bool vec) {
  mp_grid_dependency();
  const size_t i = (blockIdx.x * static_cast<size_t>(SG_THREADS) + threadIdx.x) * 4;
  if (i >= bc) return;
  const float* p = part + blockIdx.y * bc + i;
  float4 s = ld4(p);
  for (int k = 1; k < splits; ++k) {
    const float4 v = ld4(p + static_cast<size_t>(k) * 2 * bc);
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  const float f[4] = {s.x, s.y, s.z, s.w};
  segment_store((blockIdx.y ? gC : gB) + i, f, vec);
}

// gA[h]: one warp per head.
__global__ void __launch_bounds__(32) segment_sum_kernel(const float* __restrict__ part, float* gA, int B, int H, int nseg) {
  mp_grid_dependency();
  const int h = blockIdx.x;
  float s = 0.f;
  for (int i = threadIdx.x; i < B * nseg; i += 32) s += part[(static_cast<size_t>(i / nseg) * H + h) * nseg + i % nseg];
  s = warp_reduce<SumOp>(s);
  if (threadIdx.x == 0) gA[h] = s;
}

constexpr size_t SG_SCALARS = SG_Q * (sizeof(double) + sizeof(float));
constexpr size_t SG_SMEM_STATES = (SG_Q * (SG_NPITCH + SG_PPITCH) + SG_Q) * sizeof(float) + SG_SCALARS;
constexpr size_t SG_SMEM_FORWARD = SG_Q * 2 * (SG_NPITCH + SG_PPITCH) * sizeof(float) + SG_SCALARS;
constexpr size_t SG_SMEM_REVERSE = (SG_Q * (2 * SG_NPITCH + 5 * SG_PPITCH) + SG_STATE + (2 + 16) * SG_Q + 8) * sizeof(float) + SG_SCALARS;
static_assert(SG_STATE <= SG_Q * SG_NPITCH, "the state takes the place of B");

// Heads of a group per CTA of the reverse: shares until there are four CTAs per SM to hand out.
int segment_splits(int B, int L, int H, int G) {
  const long units = static_cast<long>(B) * ((L + SG_Q - 1) / SG_Q) * G;
  const long want = (4 * 148 + units - 1) / units, hpg = H / G;
  return static_cast<int>(want < 1 ? 1 : (want < hpg ? want : hpg));
}

struct SegScratch { float* states; float* decay; float* ga_part; float* gb_part; size_t total; };
SegScratch segment_carve(void* base, int B, int L, int H, int G, bool reverse) {
  SegScratch s;
  const size_t start = (256 - (reinterpret_cast<uintptr_t>(base) & 255)) & 255;   // the caller's pointer may have any alignment
  size_t off = 0;
  auto take = [&](size_t floats) {
    float* p = base != nullptr ? reinterpret_cast<float*>(static_cast<unsigned char*>(base) + start + off) : nullptr;
    off += (floats * sizeof(float) + 255) & ~size_t(255);
    return p;
  };
  const size_t units = static_cast<size_t>(B) * H * ((static_cast<size_t>(L) + SG_Q - 1) / SG_Q);
  s.states = take(units * SG_STATE * (reverse ? 2 : 1));
  s.decay = take(units);
  s.ga_part = take(reverse ? units : 0);
  s.gb_part = take(reverse ? static_cast<size_t>(segment_splits(B, L, H, G)) * 2 * B * L * G * SG_N : 0);
  s.total = off + 256;
  return s;
}

SegArgs segment_args(const void* x, const void* dt, const void* A, const void* Bm, const void* Cm, const SegScratch& w, int B, int L, int H, int G) {
  SegArgs g{};
  g.x = static_cast<const __half*>(x); g.dt = static_cast<const float*>(dt); g.A = static_cast<const float*>(A);
  g.Bm = static_cast<const __half*>(Bm); g.Cm = static_cast<const __half*>(Cm);
  g.states = w.states; g.decay = w.decay; g.ga_part = w.ga_part; g.gb_part = w.gb_part;
  g.B = B; g.L = L; g.H = H; g.G = G; g.nseg = (L + SG_Q - 1) / SG_Q;
  g.vec = mp_aligned16(x) && mp_aligned16(Bm) && mp_aligned16(Cm);
  return g;
}

// The states every segment receives, in one direction or both.
void segment_state_launches(const SegArgs& g, int directions, cudaStream_t st) {
  MP_CUDA_CHECK(cudaFuncSetAttribute(segment_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SG_SMEM_STATES)));
  MpLaunch(dim3(g.B * g.H * g.nseg, directions), SG_THREADS, SG_SMEM_STATES, st)(segment_states_kernel, g);
  MP_LAUNCH_CHECK();
  if (g.nseg > 1) {
    MpLaunch(dim3(g.B * g.H * (SG_STATE / 4 / SG_THREADS), directions), SG_THREADS, 0, st)(segment_carry_kernel, g);
    MP_LAUNCH_CHECK();
  }
}

}  // namespace

// ---------------------------------------------------------------------------
// Interface to the launchers in ssd.cu.
// ---------------------------------------------------------------------------
bool mp_ssd_segments_supported(int L, int H, int P, int N, int G) { return P == SG_P && N == SG_N && L >= 32 && G > 0 && H % G == 0; }

size_t mp_ssd_segments_scratch(int B, int L, int H, int G, bool reverse) { return segment_carve(nullptr, B, L, H, G, reverse).total; }

void mp_ssd_segments_forward(const void* x, const void* dt, const void* A, const void* Bm, const void* Cm, void* y, void* scratch, int B, int L,
                             int H, int G, cudaStream_t st) {
  SegArgs g = segment_args(x, dt, A, Bm, Cm, segment_carve(scratch, B, L, H, G, false), B, L, H, G);
  g.y = static_cast<__half*>(y);
  g.vec = g.vec && mp_aligned16(y);
  if (g.nseg > 1) segment_state_launches(g, 1, st);
  MP_CUDA_CHECK(cudaFuncSetAttribute(segment_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SG_SMEM_FORWARD)));
  MpLaunch(B * H * g.nseg, SG_THREADS, SG_SMEM_FORWARD, st)(segment_forward_kernel, g);
  MP_LAUNCH_CHECK();
}

void mp_ssd_segments_reverse(const void* x, const void* dt, const void* A, const void* Bm, const void* Cm, const void* gy, void* gx, void* gdt,
                             void* gA, void* gB, void* gC, void* scratch, int B, int L, int H, int G, cudaStream_t st) {
  SegArgs g = segment_args(x, dt, A, Bm, Cm, segment_carve(scratch, B, L, H, G, true), B, L, H, G);
  g.gy = static_cast<const __half*>(gy); g.gx = static_cast<__half*>(gx); g.gdt = static_cast<float*>(gdt);
  g.splits = segment_splits(B, L, H, G);
  const bool fold_vec = mp_aligned16(gB) && mp_aligned16(gC);
  g.vec = g.vec && mp_aligned16(gy) && mp_aligned16(gx);
  if (g.nseg > 1) segment_state_launches(g, 2, st);
  MP_CUDA_CHECK(cudaFuncSetAttribute(segment_reverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SG_SMEM_REVERSE)));
  MpLaunch(B * g.nseg * G * g.splits, SG_THREADS, SG_SMEM_REVERSE, st)(segment_reverse_kernel, g);
  MP_LAUNCH_CHECK();
  const size_t bc = static_cast<size_t>(B) * L * G * SG_N;
  MpLaunch(dim3(static_cast<unsigned>((bc / 4 + SG_THREADS - 1) / SG_THREADS), 2), SG_THREADS, 0, st)(segment_fold_kernel, g.gb_part, static_cast<__half*>(gB),
                                                                                                   static_cast<__half*>(gC), bc, g.splits, fold_vec);
  MpLaunch(H, 32, 0, st)(segment_sum_kernel, g.ga_part, static_cast<float*>(gA), B, H, g.nseg);
  MP_LAUNCH_CHECK();
}
