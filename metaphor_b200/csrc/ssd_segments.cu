// Mamba-2 SSD scan of r16 tensors to the accuracy of fp32 arithmetic, over segments of 64 steps that run side by side (head size 64,
// state 128, any number of steps).  It serves the calls that whole tensor-core chunks do not cover: lengths that are no multiple of
// the chunk, and other chunk lengths; pointers need no more than the alignment of their elements.  Its results are those of the
// recurrence (ssd_generic.cu) to the accuracy of fp32 sums: weights, scores and states are fp32 values (in a product two terms, 23 bits, with
// their own exponents), and A's gradient is a sum of the products that make it up, not a difference of row dots, so that it keeps its digits
// where almost nothing is carried from step to step ([2, 200, 16] with step sizes around 2: the r16 chunk walk is off by 0.6 of gA and 0.03 of
// gdt, this by 2.3e-7 and 1.2e-7).
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
// Launches: states made inside every segment, both directions (segment_states); carried from segment to segment, block by block
// (segment_carry); outputs (segment_forward / segment_reverse); for the reverse two folds.
//
// Every product has one operand that is r16 in memory (x, B, C, gy), which tf32 holds whole: 11 bits and a wider exponent.  The other, in fp32
// (weights times scores, scaled values, states), is split where it is read into two tf32 terms, 11 bits rounded and the rest, with nothing shared
// between values.  A product is then two tensor-core MMAs; the scores, r16 by r16, are one r16 MMA.  mma.sync and not tcgen05, because the sums
// stay in registers and are taken out of the accumulator, which truncates, after every 16 products and added up rounded.
// A CTA with an infinity or a NaN among its results does its share again on the FP pipe (*_plain below): where an r16 tile holds one, the
// lower term of a value that needs none would meet it with a zero, and so would a step that the mask leaves out.
//
// Forward / reverse in us, recurrence -> fp32 on the FP pipe (24 TFLOP/s of its 72) -> here:
//   [2, 1000, 24] 1 806 / 41 544 -> 96 / 260 -> 50 / 128,   [8, 8191, 32] 41 650 / 800 600 -> 3 950 / 8 972 -> 1 853 / 4 901,
//   [1, 8191, 2] 57 / 107 -> 40 / 89 (FP pipe -> here),     [1, 100, 2] 182 / 3 957 -> 21 / 38 -> 15 / 26.
// The 2-norm of the errors against r64: y, gx, gB, gC are r16 roundings on all three; gdt 1.2e-7 - 1.8e-7 here, 1.3e-7 - 2.5e-7 on the FP pipe.
// Two r16 terms under a power of two per row or 16 x 16 block are half the MMAs and nothing to widen or split when read (44 / 93 us for the first
// shape), but values 2^33 below the largest of a block then made results wrong by up to a fifth of themselves where the large one met a zero.
// What bounds the reverse: its sixteen warps issue in 56 % of the cycles, tensor pipe 37 %, ALU (addresses, splits) 44 %; the states and the carry
// move 128 KB of global memory a head and segment.
// Below 32 steps the recurrence stays (60 / 1 214 us at [2, 31, 24]): its forward needs no scratch, and callers may rely on that.
#include "mp_async.cuh"

namespace {

constexpr int SG_Q = 64;              // steps per segment
constexpr int SG_N = 128, SG_P = 64;  // state size, head size
constexpr int SG_STATE_BYTES = SG_N * SG_P * 4;

struct SegArgs {
  const __half* x; const float* dt; const float* A; const __half* Bm; const __half* Cm; const __half* gy;
  __half* y;                 // forward
  __half* gx; float* gdt;    // reverse
  float* states;             // [B H][nseg][64 p][128 n] states received; the adjoint ones follow in the reverse
  float* decay;              // [B H][nseg]: exp(E)
  float* ga_part;            // [B H][nseg]
  float* gb_part;            // [splits][B L G][128] sums over the heads of a split, gB then gC
  int B, L, H, G, nseg, splits;
  bool vec;                  // every r16 pointer is 16-byte aligned
};

// Scalars of a segment, by one warp: a lane's two inclusive sums of dt A and the last one; steps past the sequence do not decay (dt = 0).
struct SegScan { double c0, c1, last; };
__device__ __forceinline__ SegScan segment_scan(double a, float d0, float d1, int lane) {
  const double v0 = d0 * a, v1 = d1 * a;
  double s = v0 + v1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double up = __shfl_up_sync(0xffffffffu, s, o);
    if (lane >= o) s += up;
  }
  return {s - v1, s, __shfl_sync(0xffffffffu, s, 31)};
}
__device__ __forceinline__ void segment_scalars(const SegArgs& g, int b, int h, int t0, double* cum, float* dt, int lane) {
  const int t = t0 + 2 * lane;
  const float* src = g.dt + (static_cast<size_t>(b) * g.L + t) * g.H + h;
  const float d0 = t < g.L ? src[0] : 0.f, d1 = t + 1 < g.L ? src[g.H] : 0.f;
  const SegScan s = segment_scan(static_cast<double>(g.A[h]), d0, d1, lane);
  cum[2 * lane] = s.c0;
  cum[2 * lane + 1] = s.c1;
  dt[2 * lane] = d0;
  dt[2 * lane + 1] = d1;
}
__device__ __forceinline__ float segment_exp(double v) { return expf(static_cast<float>(v)); }

// ---------------------------------------------------------------------------
// r16 tiles in shared memory: rows of PITCH bytes, their 16-byte chunks exchanged by the row, so that the eight rows of an ldmatrix
// lie in different banks.
// ---------------------------------------------------------------------------
template <int PITCH>
__device__ __forceinline__ uint32_t tile_at(uint32_t base, int r, int c) {
  return base + r * PITCH + ((c ^ (PITCH == 64 ? (r >> 1) & 3 : r & 7)) << 4);
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void st_shared16(uint32_t dst, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// 64 steps of CHUNKS 16-byte chunks; steps past the sequence become zeros.
template <int CHUNKS, int THREADS>
__device__ __forceinline__ void tile_load(uint32_t dst, const __half* src, size_t pitch, int rows, bool vec) {
#pragma unroll
  for (int k = 0; k < SG_Q * CHUNKS / THREADS; ++k) {
    const int idx = k * THREADS + threadIdx.x, r = idx / CHUNKS, c = idx % CHUNKS;
    const uint32_t at = tile_at<CHUNKS * 16>(dst, r, c);
    const __half* p = src + r * pitch + c * 8;
    if (r >= rows) {
      st_shared16(at, make_uint4(0, 0, 0, 0));
    } else if (vec) {
      cp_async16(at, p);
    } else {
      const unsigned short* u = reinterpret_cast<const unsigned short*>(p);
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = u[2 * e] | static_cast<uint32_t>(u[2 * e + 1]) << 16;
      st_shared16(at, make_uint4(w[0], w[1], w[2], w[3]));
    }
  }
}
__device__ __forceinline__ uint32_t r16_finite(uint32_t v) {   // infinities and NaN replaced by zero
  if ((v & 0x7c00u) == 0x7c00u) v &= 0xffff0000u;
  if ((v & 0x7c000000u) == 0x7c000000u) v &= 0x0000ffffu;
  return v;
}

// fp32 tiles in shared memory: rows of PITCH bytes, their 16-byte chunks exchanged by the row, so that two chunks of four neighbouring rows, of
// four even and of four odd ones lie in different banks.
template <int PITCH>
__device__ __forceinline__ uint32_t wide_at(uint32_t base, int r, int c) { return base + r * PITCH + ((c ^ (((r ^ (r >> 2)) & 3) << 1)) << 4); }
__device__ __forceinline__ float2 ld_shared8(uint32_t src) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(src) : "memory");
  return v;
}
__device__ __forceinline__ float ld_shared4(uint32_t src) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(src) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_shared16f(uint32_t src) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(src) : "memory");
  return v;
}

// A state: rows p of 512 bytes.
template <int THREADS>
__device__ __forceinline__ void state_load(uint32_t dst, const float* src) {
#pragma unroll
  for (int k = 0; k < SG_STATE_BYTES / 16 / THREADS; ++k) {
    const int idx = k * THREADS + threadIdx.x;
    cp_async16(wide_at<512>(dst, idx >> 5, idx & 31), src + idx * 4);
  }
}

// ---------------------------------------------------------------------------
// Fragments.  A lane holds rows g and g + 8 of a 16-row operand or result, columns 2 q, 2 q + 1 of every eight (g = lane / 4, q = lane % 4).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma0(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {   // nothing accumulated before
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// The same in tf32 over eight columns: a lane holds columns q and q + 4, which are used for columns 2 q and 2 q + 1 of an r16 operand.
__device__ __forceinline__ void mma8(float (&d)[4], float a0, float a1, float a2, float a3, float b0, float b1) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(__float_as_uint(a0)), "r"(__float_as_uint(a1)), "r"(__float_as_uint(a2)), "r"(__float_as_uint(a3)), "r"(__float_as_uint(b0)),
                 "r"(__float_as_uint(b1)));
}
__device__ __forceinline__ void mma80(float (&d)[4], float a0, float a1, float a2, float a3, float b0, float b1) {   // nothing accumulated before
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(__float_as_uint(a0)), "r"(__float_as_uint(a1)), "r"(__float_as_uint(a2)), "r"(__float_as_uint(a3)), "r"(__float_as_uint(b0)),
                 "r"(__float_as_uint(b1)), "f"(0.f));
}
// d += a b over 16 columns (mma160: d = a b), operands as values in the order of an r16 operand's registers.
__device__ __forceinline__ void mma160(float (&d)[4], const float (&a)[8], const float* b) {
  mma80(d, a[0], a[2], a[1], a[3], b[0], b[1]);
  mma8(d, a[4], a[6], a[5], a[7], b[2], b[3]);
}
__device__ __forceinline__ void mma16(float (&d)[4], const float (&a)[8], const float* b) {
  mma8(d, a[0], a[2], a[1], a[3], b[0], b[1]);
  mma8(d, a[4], a[6], a[5], a[7], b[2], b[3]);
}
__device__ __forceinline__ void widen(float* v, const uint32_t* r, int n) {   // n is a constant
#pragma unroll
  for (int e = 0; e < n; ++e) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(r + e));
    v[2 * e] = f.x;
    v[2 * e + 1] = f.y;
  }
}
// Operand of 16 rows from r0 on, 16 columns from chunk c0 on (two chunks), of a tile [rows][columns]; _t: of a tile [columns][rows], rows
// of chunks r0, r0 + 1, columns from c0 on.
template <int PITCH>
__device__ __forceinline__ void load_a(uint32_t (&a)[4], uint32_t tile, int r0, int c0, int lane) { ldsm(a, tile_at<PITCH>(tile, r0 + (lane & 15), c0 + (lane >> 4))); }
template <int PITCH>
__device__ __forceinline__ void load_a_t(uint32_t (&a)[4], uint32_t tile, int c0, int r0, int lane) {
  ldsm_t(a, tile_at<PITCH>(tile, c0 + (lane & 7) + ((lane >> 4) << 3), r0 + ((lane >> 3) & 1)));
}
// Two neighbouring column operands (eight columns each): columns are rows n0 .. n0 + 15 of the tile, the sum runs over chunks c0, c0 + 1.
template <int PITCH>
__device__ __forceinline__ void load_b(uint32_t (&b)[4], uint32_t tile, int n0, int c0, int lane) {
  ldsm(b, tile_at<PITCH>(tile, n0 + (lane & 7) + ((lane >> 4) << 3), c0 + ((lane >> 3) & 1)));
}
// The same where the sum runs over rows k0 .. k0 + 15 of the tile and the columns are those of chunks c0, c0 + 1.
template <int PITCH>
__device__ __forceinline__ void load_b_t(uint32_t (&b)[4], uint32_t tile, int k0, int c0, int lane) { ldsm_t(b, tile_at<PITCH>(tile, k0 + (lane & 15), c0 + (lane >> 4))); }

// A value as two terms that tf32 holds: 11 bits rounded, and the rest, of which the MMA reads 11 bits.  What is not finite, or rounds up to that,
// makes a NaN of the result.
__device__ __forceinline__ void split(float v, float& hi, float& lo) {
  hi = __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xffffe000u);
  lo = v - hi;
}
// The same where an infinity has to stay one: 11 bits cut off, the rest rounded; none where there is none.
__device__ __forceinline__ void split_keeping(float v, float& hi, float& lo) {
  hi = __uint_as_float(__float_as_uint(v) & 0xffffe000u);
  const float rest = v - hi;
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(rest));
  lo = rest == rest ? __uint_as_float(r) : 0.f;
}

// ---------------------------------------------------------------------------
// What a segment adds to the state behind it (blockIdx.y = 0) and to the adjoint state before it (1).  A warp has 16 of the 64 rows p.
// ---------------------------------------------------------------------------
constexpr int SS_THREADS = 128;
constexpr size_t SS_SMEM = SG_Q * SG_P * 2 + SG_Q * SG_N * 2 + SG_Q * sizeof(float);

__global__ void __launch_bounds__(SS_THREADS) segment_states_kernel(const SegArgs g) {
  mp_grid_dependency();
  extern __shared__ __align__(128) unsigned char seg_smem[];
  const bool anti = blockIdx.y != 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3;
  const int seq = blockIdx.x / g.nseg, seg = blockIdx.x % g.nseg, b = seq / g.H, h = seq % g.H, grp = h / (g.H / g.G);
  const int t0 = seg * SG_Q, rows = min(SG_Q, g.L - t0);
  const uint32_t sv = mp_smem_u32(seg_smem), sk = sv + SG_Q * SG_P * 2;
  float* wt = reinterpret_cast<float*>(seg_smem + SG_Q * SG_P * 2 + SG_Q * SG_N * 2);
  const bool needed = anti ? seg > 0 : seg < g.nseg - 1;   // something lies beyond
  if (needed) {
    const size_t row = static_cast<size_t>(b) * g.L + t0;
    tile_load<SG_P / 8, SS_THREADS>(sv, (anti ? g.gy : g.x) + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows, g.vec);
    tile_load<SG_N / 8, SS_THREADS>(sk, (anti ? g.Cm : g.Bm) + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec);
    cp_async_commit();
  }
  if (warp == 0) {
    const int t = t0 + 2 * lane;
    const float* src = g.dt + (static_cast<size_t>(b) * g.L + t) * g.H + h;
    const float d0 = t < g.L ? src[0] : 0.f, d1 = t + 1 < g.L ? src[g.H] : 0.f;
    const SegScan sc = segment_scan(static_cast<double>(g.A[h]), d0, d1, lane);
    wt[2 * lane] = anti ? segment_exp(sc.c0) : d0 * segment_exp(sc.last - sc.c0);
    wt[2 * lane + 1] = anti ? segment_exp(sc.c1) : d1 * segment_exp(sc.last - sc.c1);
    if (lane == 0 && !anti) g.decay[blockIdx.x] = segment_exp(sc.last);
  }
  if (!needed) return;
  cp_async_wait<0>();
  __syncthreads();
  // rows p of the scaled values, over the 64 steps
  float hi[4][8], lo[4][8];
#pragma unroll
  for (int kt = 0; kt < 4; ++kt) {
    uint32_t r[4];
    load_a_t<SG_P * 2>(r, sv, kt * 16, warp * 2, lane);
    float v[8];
    widen(v, r, 4);
    const float2 wa = *reinterpret_cast<const float2*>(wt + kt * 16 + 2 * q), wb = *reinterpret_cast<const float2*>(wt + kt * 16 + 8 + 2 * q);
#pragma unroll
    for (int e = 0; e < 8; ++e) split_keeping(v[e] * (e < 4 ? (e & 1 ? wa.y : wa.x) : (e & 1 ? wb.y : wb.x)), hi[kt][e], lo[kt][e]);
  }
  float* out = g.states + (static_cast<size_t>(anti) * g.B * g.H * g.nseg + blockIdx.x) * (SG_N * SG_P) + (warp * 16 + (lane >> 2)) * SG_N + 2 * q;
#pragma unroll 2
  for (int nb = 0; nb < SG_N / 16; ++nb) {
    // `finite`: the r16 operand of the lower terms, whose zeros must not meet an infinity
    auto sums = [&](float (&s)[2][4], bool finite) {
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        uint32_t bb[4];
        load_b_t<SG_N * 2>(bb, sk, kt * 16, nb * 2, lane);
        float b[8];
        widen(b, bb, 4);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float c[4];
          if (finite) {
            const uint32_t bf[2] = {r16_finite(bb[2 * u]), r16_finite(bb[2 * u + 1])};
            float f[4];
            widen(f, bf, 2);
            mma160(c, lo[kt], f);
          } else {
            mma160(c, lo[kt], b + 4 * u);
          }
          mma16(c, hi[kt], b + 4 * u);
#pragma unroll
          for (int e = 0; e < 4; ++e) s[u][e] = kt == 0 ? c[e] : s[u][e] + c[e];
        }
      }
    };
    float s[2][4];
    sums(s, false);
    float check = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) check = fmaf(s[0][e], 0.f, fmaf(s[1][e], 0.f, check));
    if (__any_sync(0xffffffffu, check != 0.f)) sums(s, true);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      *reinterpret_cast<float2*>(out + nb * 16 + u * 8) = make_float2(s[u][0], s[u][1]);
      *reinterpret_cast<float2*>(out + 8 * SG_N + nb * 16 + u * 8) = make_float2(s[u][2], s[u][3]);
    }
  }
}

// In place: what every segment adds becomes what every segment receives.  A thread has four values of a sequence's states; it reads four
// segments ahead, and what it overwrites (the segment behind the one whose sum it has) it has read before.
constexpr int SC_THREADS = 128;
__global__ void __launch_bounds__(SC_THREADS) segment_carry_kernel(const SegArgs g) {
  mp_grid_dependency();
  constexpr int PER = SG_N * SG_P / 4 / SC_THREADS;   // CTAs per sequence
  const bool anti = blockIdx.y != 0;
  const int seq = blockIdx.x / PER;
  float4* base = reinterpret_cast<float4*>(g.states + (static_cast<size_t>(anti) * g.B * g.H + seq) * g.nseg * (SG_N * SG_P)) +
                 (blockIdx.x % PER) * SC_THREADS + threadIdx.x;
  const float* decay = g.decay + static_cast<size_t>(seq) * g.nseg;
  const int steps = g.nseg - 1;
  auto segment = [&](int k) { return anti ? g.nseg - 1 - k : k; };
  float4 next[4];
  float dnext[4];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int k = min(k0 + u, steps - 1);
      next[u] = base[static_cast<size_t>(segment(k)) * (SG_N * SG_P / 4)];
      dnext[u] = decay[segment(k)];
    }
  };
  fetch(0);
  float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  for (int k0 = 0; k0 < steps; k0 += 4) {
    float4 add[4];
    float d[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) { add[u] = next[u]; d[u] = dnext[u]; }
    if (k0 + 4 < steps) fetch(k0 + 4);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (k0 + u >= steps) break;
      c.x = fmaf(d[u], c.x, add[u].x);
      c.y = fmaf(d[u], c.y, add[u].y);
      c.z = fmaf(d[u], c.z, add[u].z);
      c.w = fmaf(d[u], c.w, add[u].w);
      base[static_cast<size_t>(segment(k0 + u) + (anti ? -1 : 1)) * (SG_N * SG_P / 4)] = c;
    }
  }
}

constexpr int SG_THREADS = 256;

// A CTA's share: one segment of one batch entry, one group, some of the group's heads.
struct SegShare { int b, seg, grp, split, h_first, h_end; };
__device__ __forceinline__ SegShare segment_share(const SegArgs& g) {
  SegShare s;
  const int hpg = g.H / g.G;
  s.split = blockIdx.x % g.splits;
  int rest = blockIdx.x / g.splits;
  s.grp = rest % g.G;
  rest /= g.G;
  s.seg = rest % g.nseg;
  s.b = rest / g.nseg;
  s.h_first = s.grp * hpg + static_cast<int>(static_cast<long long>(hpg) * s.split / g.splits);
  s.h_end = s.grp * hpg + static_cast<int>(static_cast<long long>(hpg) * (s.split + 1) / g.splits);
  return s;
}

// What the kernels need of one head's steps in the segment.
struct SegSteps { double cum[SG_Q]; float dt[SG_Q], grow[SG_Q], left[SG_Q]; };   // grow = exp(cum), left = exp(E - cum)
__device__ __forceinline__ void segment_steps(const SegArgs& g, int b, int h, int t0, SegSteps& s, int lane) {
  segment_scalars(g, b, h, t0, s.cum, s.dt, lane);
  __syncwarp();
  const double last = s.cum[SG_Q - 1];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const double c = s.cum[2 * lane + e];
    s.grow[2 * lane + e] = segment_exp(c);
    s.left[2 * lane + e] = segment_exp(last - c);
  }
}

// ---------------------------------------------------------------------------
// Scores.  The ten 16 x 16 blocks on and below the diagonal of a 64 x 64 matrix are dealt out to the warps; a block's scores of C and B stay
// with its warp over the heads.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool block_of(int k, int& ib, int& jb) {
  ib = k < 1 ? 0 : k < 3 ? 1 : k < 6 ? 2 : 3;
  jb = k - ib * (ib + 1) / 2;
  return k < 10;
}
// Rows 16 ib of tile a times rows 16 jb of tile b, over K; 16 products at a time are taken out of the accumulator.
template <int K>
__device__ __forceinline__ void block_scores(float (&s)[2][4], uint32_t a, uint32_t b, int ib, int jb, int lane) {
#pragma unroll
  for (int e = 0; e < 4; ++e) s[0][e] = s[1][e] = 0.f;
#pragma unroll
  for (int k = 0; k < K / 16; ++k) {
    uint32_t av[4], bv[4];
    load_a<K * 2>(av, a, ib * 16, 2 * k, lane);
    load_b<K * 2>(bv, b, jb * 16, 2 * k, lane);
    float c0[4], c1[4];
    mma0(c0, av, bv[0], bv[1]);
    mma0(c1, av, bv[2], bv[3]);
#pragma unroll
    for (int e = 0; e < 4; ++e) { s[0][e] += c0[e]; s[1][e] += c1[e]; }
  }
}
// M of a block: exp(cum_i - cum_j), zero above the diagonal.
__device__ __forceinline__ void block_decays(float (&m)[2][4], const double* cum, int ib, int jb, int g, int q) {
  const double c0 = cum[ib * 16 + g], c1 = cum[ib * 16 + g + 8];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int j = u * 8 + 2 * q;   // in the block
    const double2 cj = *reinterpret_cast<const double2*>(cum + jb * 16 + j);
    m[u][0] = segment_exp(c0 - cj.x);
    m[u][1] = segment_exp(c0 - cj.y);
    m[u][2] = segment_exp(c1 - cj.x);
    m[u][3] = segment_exp(c1 - cj.y);
    if (ib == jb) {
      if (j > g) m[u][0] = 0.f;
      if (j + 1 > g) m[u][1] = 0.f;
      if (j > g + 8) m[u][2] = 0.f;
      if (j + 1 > g + 8) m[u][3] = 0.f;
    }
  }
}
// A block of a tile [64][64] in fp32.
__device__ __forceinline__ void block_store(const float (&v)[2][4], uint32_t tile, int ib, int jb, int lane) {
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int r = 0; r < 2; ++r)
      asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(wide_at<SG_Q * 4>(tile, ib * 16 + (lane >> 2) + 8 * r, jb * 4 + u * 2 + ((lane & 3) >> 1)) +
                                                           8 * (lane & 1)),
                   "f"(v[u][2 * r]), "f"(v[u][2 * r + 1]) : "memory");
}

// ---------------------------------------------------------------------------
// Products.  A warp has a few columns of the result and all 64 rows (NR = 4 blocks of 16), or two of the four blocks (NR = 2: `part` 0 has the
// first and the last, 1 the others, which is as many blocks of scores), so that what it reads of a state, and of the tiles that the scores are
// multiplied by, serves all of them.
// ---------------------------------------------------------------------------
template <int NR>
__device__ __forceinline__ int row_block(int i, int part) { return NR == 4 ? i : part ? 1 + i : 3 * i; }

// Rows of a tile [64][128] (over n) times a state: columns p = 8 c .. 8 c + 7.
template <int NR>
__device__ __forceinline__ void times_state_p(float (&o)[NR][4], uint32_t rows, uint32_t state, int c, int part, int lane) {
  const int q = lane & 3;
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
#pragma unroll 2
  for (int k = 0; k < 8; ++k) {
    float hi[4], lo[4];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float2 v = ld_shared8(wide_at<512>(state, c * 8 + (lane >> 2), k * 4 + 2 * h + (q >> 1)) + 8 * (q & 1));
      split(v.x, hi[2 * h], lo[2 * h]);
      split(v.y, hi[2 * h + 1], lo[2 * h + 1]);
    }
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      uint32_t r[4];
      load_a<SG_N * 2>(r, rows, row_block<NR>(i, part) * 16, 2 * k, lane);
      float a[8], s[4];
      widen(a, r, 4);
      mma160(s, a, lo);
      mma16(s, a, hi);
#pragma unroll
      for (int e = 0; e < 4; ++e) o[i][e] += s[e];
    }
  }
}
// Rows of a tile [64][64] (over p) times a state: columns n = 16 nb .. 16 nb + 15.
template <int NR>
__device__ __forceinline__ void times_state_n(float (&o)[NR][2][4], uint32_t rows, uint32_t state, int nb, int part, int lane) {
  const int q = lane & 3, n = lane >> 2;
#pragma unroll
  for (int i = 0; i < NR; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][0][e] = o[i][1][e] = 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float hi[2][4], lo[2][4];
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        split(ld_shared4(wide_at<512>(state, k * 16 + 2 * q + (e & 1) + 8 * (e >> 1), nb * 4 + u * 2 + (n >> 2)) + 4 * (n & 3)), hi[u][e], lo[u][e]);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      uint32_t r[4];
      load_a<SG_P * 2>(r, rows, row_block<NR>(i, part) * 16, 2 * k, lane);
      float a[8];
      widen(a, r, 4);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float s[4];
        mma160(s, a, lo[u]);
        mma16(s, a, hi[u]);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][u][e] += s[e];
      }
    }
  }
}
// The operand for eight columns (chunk c) and all 64 steps of a tile [64][64].
__device__ __forceinline__ void load_steps(uint32_t (&b)[4][2], uint32_t tile, int c, int lane) {
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    uint32_t v[4];
    ldsm_t(v, tile_at<SG_P * 2>(tile, k * 32 + lane, c));
    b[2 * k][0] = v[0]; b[2 * k][1] = v[1]; b[2 * k + 1][0] = v[2]; b[2 * k + 1][1] = v[3];
  }
}
// o += scores (LOWER: rows i, over j up to the row's block; otherwise rows j, over i from the row's block on) times COLS tiles of eight columns.
template <int NR, bool LOWER, int COLS>
__device__ __forceinline__ void times_scores(float (&o)[NR][COLS][4], uint32_t scores, const uint32_t (&b)[4][2 * COLS], int part, int lane) {
  const int q = lane & 3, r = lane >> 2;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float bv[4 * COLS];
    widen(bv, b[k], 2 * COLS);
#pragma unroll
    for (int i = 0; i < NR; ++i) {
      const int rb = row_block<NR>(i, part);
      if (LOWER ? k > rb : k < rb) continue;
      float hi[8], lo[8];   // rows r, r + 8 of the block, steps 2 q, 2 q + 1, then those eight further
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float2 v;
        if (LOWER) {
          v = ld_shared8(wide_at<SG_Q * 4>(scores, rb * 16 + r + 8 * (e & 1), k * 4 + 2 * (e >> 1) + (q >> 1)) + 8 * (q & 1));
        } else {
          v.x = ld_shared4(wide_at<SG_Q * 4>(scores, k * 16 + 2 * q + 8 * (e >> 1), rb * 4 + 2 * (e & 1) + (r >> 2)) + 4 * (r & 3));
          v.y = ld_shared4(wide_at<SG_Q * 4>(scores, k * 16 + 2 * q + 1 + 8 * (e >> 1), rb * 4 + 2 * (e & 1) + (r >> 2)) + 4 * (r & 3));
        }
        split(v.x, hi[2 * e], lo[2 * e]);
        split(v.y, hi[2 * e + 1], lo[2 * e + 1]);
      }
#pragma unroll
      for (int u = 0; u < COLS; ++u) {
        float s[4];
        mma160(s, lo, bv + 4 * u);
        mma16(s, hi, bv + 4 * u);
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][u][e] += s[e];
      }
    }
  }
}
// Two neighbouring r16 results.
__device__ __forceinline__ void store_pair(__half* dst, float v0, float v1, bool vec) {
  const __half2 h = __floats2half2_rn(v0, v1);
  if (vec) {
    *reinterpret_cast<__half2*>(dst) = h;
  } else {
    dst[0] = __low2half(h);
    dst[1] = __high2half(h);
  }
}

// ---------------------------------------------------------------------------
// The same outputs on the FP pipe, for a CTA that met an infinity or a NaN: fp32 tiles, and steps that the mask leaves out are not read.
// ---------------------------------------------------------------------------
constexpr int SG_NPITCH = SG_N + 4, SG_PPITCH = SG_P + 4;   // floats per row of a shared tile: rows 16 bytes apart in the banks

// [64 steps][COLS] of r16 -> fp32 tile.  Steps past the sequence become zeros.
template <int COLS, int PITCH, int THREADS>
__device__ __forceinline__ void plain_tile(float* dst, const __half* src, size_t pitch, int rows) {
#pragma unroll 1
  for (int idx = threadIdx.x; idx < SG_Q * COLS; idx += THREADS) {
    const int r = idx / COLS, c = idx % COLS;
    dst[r * PITCH + c] = r < rows ? __half2float(src[r * pitch + c]) : 0.f;
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

template <int THREADS>
__device__ __forceinline__ void plain_state(float* dst, const float* state) {
#pragma unroll 1
  for (int idx = threadIdx.x; idx < SG_N * SG_P; idx += THREADS) {
    const int p = idx / SG_N, n = idx % SG_N;
    dst[state_at(n, p >> 2) + (p & 3)] = state[idx];
  }
}

// Scores a_i b_j^T of the 16 x 16 blocks on and below the diagonal: thread (ty, tx) has i = ty + 16 u, j = tx + 16 v.
template <int K, int PITCH>
__device__ __forceinline__ void segment_scores(const float* a, const float* b, int ty, int tx, float (&acc)[4][4]) {
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = 0.f;
  // sixteen products at a time, as the tensor cores have them
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

// y of heads h_first .. h_end - 1 in one segment.  Thread (ty, tx): four rows 16 apart, four columns.
__device__ __noinline__ void segment_forward_plain(const SegArgs& g, float* smem, int b, int seg, int grp, int h_first, int h_end) {
  float* sC = smem;                              // [64][132]
  float* sB = sC + SG_Q * SG_NPITCH;             // [64][132], then the state [128][64]
  float* sX = sB + SG_Q * SG_NPITCH;             // [64][68]
  float* sW = sX + SG_Q * SG_PPITCH;             // [64][68]
  double* cum = reinterpret_cast<double*>(sW + SG_Q * SG_PPITCH);
  float* dt = reinterpret_cast<float*>(cum + SG_Q);
  const int t0 = seg * SG_Q, rows = min(SG_Q, g.L - t0);
  const size_t row = static_cast<size_t>(b) * g.L + t0;
#pragma unroll 1
  for (int h = h_first; h < h_end; ++h) {
    __syncthreads();
    if (threadIdx.x < 32) segment_scalars(g, b, h, t0, cum, dt, threadIdx.x);
    plain_tile<SG_N, SG_NPITCH, SG_THREADS>(sC, g.Cm + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows);
    plain_tile<SG_N, SG_NPITCH, SG_THREADS>(sB, g.Bm + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows);
    plain_tile<SG_P, SG_PPITCH, SG_THREADS>(sX, g.x + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows);
    __syncthreads();
    const int ty = threadIdx.x / 16, tx = threadIdx.x % 16, p0 = tx * 4;
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
    if (seg > 0) {
      const size_t unit = (static_cast<size_t>(b) * g.H + h) * g.nseg + seg;
      plain_state<SG_THREADS>(sB, g.states + unit * (SG_N * SG_P));
      __syncthreads();
    }
    {
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
  }
}


// ---------------------------------------------------------------------------
// y of one (batch entry, segment, group, share of the group's heads).  A warp has eight of the 64 columns; the next head's tiles arrive
// while one is worked on.
// ---------------------------------------------------------------------------
constexpr int SF_X = SG_Q * SG_P * 2;
constexpr size_t SF_TILES = SG_Q * SG_N * 2 + 2 * SF_X + SG_STATE_BYTES + SG_Q * SG_Q * 4;   // C, x twice, state, weights
constexpr size_t SF_SMEM = SF_TILES + 2 * sizeof(SegSteps);

__global__ void __launch_bounds__(SG_THREADS, 2) segment_forward_kernel(const SegArgs g) {
  mp_grid_dependency();
  extern __shared__ __align__(128) unsigned char seg_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r0 = lane >> 2;
  const SegShare sh = segment_share(g);
  const int t0 = sh.seg * SG_Q, rows = min(SG_Q, g.L - t0);
  const size_t row = static_cast<size_t>(sh.b) * g.L + t0;
  const bool before = sh.seg > 0;
  const uint32_t sC = mp_smem_u32(seg_smem), sX = sC + SG_Q * SG_N * 2, sH = sX + 2 * SF_X, sW = sH + SG_STATE_BYTES;
  SegSteps* steps = reinterpret_cast<SegSteps*>(seg_smem + SF_TILES);
  auto load_x = [&](int h) {
    tile_load<SG_P / 8, SG_THREADS>(sX + ((h - sh.h_first) & 1) * SF_X, g.x + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows, g.vec);
  };
  auto load_state = [&](int h) {
    if (before) state_load<SG_THREADS>(sH, g.states + ((static_cast<size_t>(sh.b) * g.H + h) * g.nseg + sh.seg) * (SG_N * SG_P));
  };
  tile_load<SG_N / 8, SG_THREADS>(sC, g.Cm + (row * g.G + sh.grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec);
  tile_load<SG_N / 8, SG_THREADS>(sH, g.Bm + (row * g.G + sh.grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec);   // B, for the scores
  load_x(sh.h_first);
  cp_async_commit();
  if (warp == 7) segment_steps(g, sh.b, sh.h_first, t0, steps[0], lane);
  cp_async_wait<0>();
  __syncthreads();
  float G[2][2][4];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    int ib, jb;
    if ((s == 0 || warp >> 1 == 2) && block_of(warp + 4 * s, ib, jb)) block_scores<SG_N>(G[s], sC, sH, ib, jb, lane);
  }
  __syncthreads();   // the state takes the place of B
  load_state(sh.h_first);
  cp_async_commit();
  float check = 0.f;   // becomes NaN with the first result that is none, or infinite
#pragma unroll 1
  for (int h = sh.h_first; h < sh.h_end; ++h) {
    const int par = (h - sh.h_first) & 1;
    cp_async_wait<0>();
    __syncthreads();   // this head's tiles are there, the last one's have been read
    if (h + 1 < sh.h_end) {
      load_x(h + 1);
      if (warp == 7) segment_steps(g, sh.b, h + 1, t0, steps[par ^ 1], lane);
    }
    const SegSteps& st = steps[par];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      int ib, jb;
      if (s == 1 && warp >> 1 != 2) continue;   // the last two blocks are the second ones of warps 4 and 5
      block_of(warp + 4 * s, ib, jb);
      float m[2][4];
      block_decays(m, st.cum, ib, jb, r0, q);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 dj = *reinterpret_cast<const float2*>(st.dt + jb * 16 + u * 8 + 2 * q);
#pragma unroll
        for (int e = 0; e < 4; ++e) m[u][e] = G[s][u][e] * m[u][e] * (e & 1 ? dj.y : dj.x);
      }
      block_store(m, sW, ib, jb, lane);
    }
    float o[4][1][4];
    if (before) {
      float v[4][4];
      times_state_p<4>(v, sC, sH, warp, 0, lane);
#pragma unroll
      for (int rb = 0; rb < 4; ++rb) {
        const float f0 = st.grow[rb * 16 + r0], f1 = st.grow[rb * 16 + r0 + 8];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[rb][0][e] = v[rb][e] * (e < 2 ? f0 : f1);
      }
    } else {
#pragma unroll
      for (int rb = 0; rb < 4; ++rb)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[rb][0][e] = 0.f;
    }
    __syncthreads();   // the weights are complete, the state has been read
    if (h + 1 < sh.h_end) load_state(h + 1);
    cp_async_commit();
    uint32_t b[4][2];
    load_steps(b, sX + par * SF_X, warp, lane);
    times_scores<4, true, 1>(o, sW, b, 0, lane);
    __half* y = g.y + ((row + r0) * g.H + h) * SG_P + warp * 8 + 2 * q;
#pragma unroll
    for (int rb = 0; rb < 4; ++rb)
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int i = rb * 16 + r * 8;
        check = fmaf(o[rb][0][2 * r], 0.f, fmaf(o[rb][0][2 * r + 1], 0.f, check));
        if (r0 + i < rows) store_pair(y + static_cast<size_t>(i) * g.H * SG_P, o[rb][0][2 * r], o[rb][0][2 * r + 1], g.vec);
      }
  }
  if (__syncthreads_or(check != 0.f)) segment_forward_plain(g, reinterpret_cast<float*>(seg_smem), sh.b, sh.seg, sh.grp, sh.h_first, sh.h_end);
}

// ---------------------------------------------------------------------------
// Gradients of one (batch entry, segment, group, share of the group's heads).  Of the sixteen warps two share 16 of the 128 columns of gB and
// gC, which stay in their registers over the heads, and eight of the 64 columns of gx.
// ---------------------------------------------------------------------------
constexpr int SR_THREADS = 512, SR_WARPS = SR_THREADS / 32;
constexpr int SR_X = SG_Q * SG_P * 2;
constexpr int SR_STAGE = 2 * SR_X + SG_STATE_BYTES;   // x, gy, H: two of them; Y is read first and loaded again in the middle
struct SegScalars {   // of one head; two of them, and three SegSteps (the next head's are made while the last one's are read)
  float s[4][SG_Q];       // [row block] sums over the block's rows of M G X
  float ga[4][SG_Q];      // [column block] sums over the block's columns of M G X dt, for the row blocks below it
  float tri[SG_Q];        // ga from inside the diagonal blocks
  float su[8][SG_Q];      // [16 columns] exp(cum_i) <C_i, H gy_i>
  float sv[8][SG_Q];      // [16 columns] e_j <B_j, Y x_j>
  float pin[SR_WARPS];    // [warp] parts of <Y, H>
};
constexpr size_t SR_TILES = 2 * SG_Q * SG_N * 2 + 2 * SR_STAGE + SG_STATE_BYTES + 2 * SG_Q * SG_Q * 4;
constexpr size_t SR_SMEM = SR_TILES + 3 * sizeof(SegSteps) + 2 * sizeof(SegScalars);

// gdt and a part of gA of one head, by one warp; a lane has two steps, eight lanes a block of 16.
__device__ __forceinline__ void segment_gradients(const SegArgs& g, const SegScalars& w, const SegSteps& st, int h, size_t row, int rows, size_t unit, int lane) {
  const int t = 2 * lane, blk = lane >> 3;
  const float2 d = *reinterpret_cast<const float2*>(st.dt + t);
  float s0 = 0.f, s1 = 0.f;               // s of these steps (columns)
  float below0 = 0.f, below1 = 0.f;       // the same from the row blocks below the diagonal one
  float left0 = 0.f, left1 = 0.f;         // sums of these steps' rows over the column blocks left of the diagonal one
  float across = 0.f;                     // blocks below and left of the diagonal one, whole
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 c = *reinterpret_cast<const float2*>(w.s[k] + t), r = *reinterpret_cast<const float2*>(w.ga[k] + t);
    if (k > blk) { below0 += c.x; below1 += c.y; }
    if (k == blk) { s0 = c.x; s1 = c.y; }
    if (k < blk) { left0 += r.x; left1 += r.y; }
    const float all = warp_reduce_width<SumOp, 8>(k < blk ? r.x + r.y : 0.f);   // block (blk, k)
#pragma unroll
    for (int i = k + 2; i < 4; ++i) {
      const float v = __shfl_sync(0xffffffffu, all, i * 8);
      if (k < blk && blk < i) across += v;
    }
  }
  s0 += below0;
  s1 += below1;
  float u0 = 0.f, u1 = 0.f, v0 = 0.f, v1 = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float2 u = *reinterpret_cast<const float2*>(w.su[k] + t), v = *reinterpret_cast<const float2*>(w.sv[k] + t);
    u0 += u.x; u1 += u.y; v0 += v.x; v1 += v.y;
  }
  s0 += v0;
  s1 += v1;
  v0 *= d.x;
  v1 *= d.y;
  const float q0 = d.x * below0, q1 = d.y * below1;
  float suf = u0 + u1, pre = v0 + v1;                       // over the segment: this lane's steps and those behind / before them
  float suf_b = left0 + left1, pre_b = q0 + q1;             // over the block
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const float dn = __shfl_down_sync(0xffffffffu, suf, off), up = __shfl_up_sync(0xffffffffu, pre, off);
    if (lane + off < 32) suf += dn;
    if (lane >= off) pre += up;
    if (off < 8) {
      const float dn_b = __shfl_down_sync(0xffffffffu, suf_b, off, 8), up_b = __shfl_up_sync(0xffffffffu, pre_b, off, 8);
      if ((lane & 7) + off < 8) suf_b += dn_b;
      if ((lane & 7) >= off) pre_b += up_b;
    }
  }
  float suf1 = __shfl_down_sync(0xffffffffu, suf, 1), pre0 = __shfl_up_sync(0xffffffffu, pre, 1);
  float suf1_b = __shfl_down_sync(0xffffffffu, suf_b, 1, 8), pre0_b = __shfl_up_sync(0xffffffffu, pre_b, 1, 8);
  if (lane == 31) suf1 = 0.f;
  if (lane == 0) pre0 = 0.f;
  if ((lane & 7) == 7) suf1_b = 0.f;
  if ((lane & 7) == 0) pre0_b = 0.f;
  float through = 0.f;
#pragma unroll
  for (int k = 0; k < SR_WARPS; ++k) through += w.pin[k];
  through *= segment_exp(st.cum[SG_Q - 1]);
  const float2 tri = *reinterpret_cast<const float2*>(w.tri + t);
  const float ga0 = tri.x + suf_b + pre0_b + across + (suf + pre0 + through);
  const float ga1 = tri.y + left1 + suf1_b + (pre0_b + q0) + across + (u1 + suf1 + pre0 + v0 + through);
  const float a = g.A[h];
  float* gdt = g.gdt + (row + t) * g.H + h;
  if (t < rows) gdt[0] = fmaf(a, ga0, s0);
  if (t + 1 < rows) gdt[g.H] = fmaf(a, ga1, s1);
  const float sum = warp_reduce<SumOp>(d.x * ga0 + d.y * ga1);
  if (lane == 0) g.ga_part[unit] = sum;
}

// The sums of M G X that s and ga are made of, from one block of it (w).
__device__ __forceinline__ void block_sums(const float (&w)[2][4], const float* dt, SegScalars& sc, int ib, int jb, int lane) {
  const int q = lane & 3, r = lane >> 2;
  // over the block's rows: four columns a lane, one of them left to each half of the lanes with this q twice, then added up
  float c[2][2], c2[2];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int e = 0; e < 2; ++e) c[u][e] = w[u][e] + w[u][2 + e];
  const bool b16 = lane & 16, b8 = lane & 8;
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float other = __shfl_xor_sync(0xffffffffu, b16 ? c[0][e] : c[1][e], 16);
    c2[e] = (b16 ? c[1][e] : c[0][e]) + other;
  }
  const float other = __shfl_xor_sync(0xffffffffu, b8 ? c2[0] : c2[1], 8);
  float c1 = (b8 ? c2[1] : c2[0]) + other;
  c1 += __shfl_xor_sync(0xffffffffu, c1, 4);
  if ((lane & 4) == 0) sc.s[ib][jb * 16 + (b16 ? 8 : 0) + 2 * q + (b8 ? 1 : 0)] = c1;
  float p[2][4];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const float2 dj = *reinterpret_cast<const float2*>(dt + jb * 16 + u * 8 + 2 * q);
#pragma unroll
    for (int e = 0; e < 4; ++e) p[u][e] = w[u][e] * (e & 1 ? dj.y : dj.x);
  }
  if (ib != jb) {   // over the block's columns
    float s0 = (p[0][0] + p[0][1]) + (p[1][0] + p[1][1]), s1 = (p[0][2] + p[0][3]) + (p[1][2] + p[1][3]);
#pragma unroll
    for (int off = 1; off < 4; off <<= 1) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, off);
      s1 += __shfl_xor_sync(0xffffffffu, s1, off);
    }
    if (q == 0) { sc.ga[jb][ib * 16 + r] = s0; sc.ga[jb][ib * 16 + r + 8] = s1; }
    return;
  }
  // the diagonal block: sum_{i >= t > j}, in a row the sum over the columns before t, then over the rows
  float t4[2][2] = {};
#pragma unroll
  for (int k = 0; k < 2; ++k) {   // row r, row r + 8
    float base = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float q0 = p[u][2 * k], q1 = p[u][2 * k + 1];
      float sum = q0 + q1;
#pragma unroll
      for (int off = 1; off < 4; off <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, sum, off, 4);
        if (q >= off) sum += up;
      }
      float ex = __shfl_up_sync(0xffffffffu, sum, 1, 4);
      const float all = __shfl_sync(0xffffffffu, sum, 3, 4);
      if (q == 0) ex = 0.f;
      ex += base;
      const int j = u * 8 + 2 * q, i = r + 8 * k;
      if (j <= i) t4[u][0] += ex;
      if (j + 1 <= i) t4[u][1] += ex + q0;
      base += all;
    }
  }
  float t2[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float o = __shfl_xor_sync(0xffffffffu, b16 ? t4[0][e] : t4[1][e], 16);
    t2[e] = (b16 ? t4[1][e] : t4[0][e]) + o;
  }
  const float o = __shfl_xor_sync(0xffffffffu, b8 ? t2[0] : t2[1], 8);
  float t1 = (b8 ? t2[1] : t2[0]) + o;
  t1 += __shfl_xor_sync(0xffffffffu, t1, 4);
  if ((lane & 4) == 0) sc.tri[jb * 16 + (b16 ? 8 : 0) + 2 * q + (b8 ? 1 : 0)] = t1;
}

// Rows' dot products over a warp's 16 columns: those of `v` with the tile's, and v[row] *= f[row] before.
__device__ __forceinline__ void row_dots(float (&v)[2][2][4], const float* f, uint32_t tile, int nb, float* out, int part, int lane) {
  const int q = lane & 3, r = lane >> 2;
#pragma unroll
  for (int rb = 0; rb < 2; ++rb) {
    const int i = row_block<2>(rb, part) * 16 + r;
    const float f0 = f[i], f1 = f[i + 8];
    float d0 = 0.f, d1 = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      uint32_t t0, t1;
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(t0) : "r"(tile_at<SG_N * 2>(tile, i, nb * 2 + u) + 4 * q) : "memory");
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(t1) : "r"(tile_at<SG_N * 2>(tile, i + 8, nb * 2 + u) + 4 * q) : "memory");
      const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&t0)), b = __half22float2(*reinterpret_cast<const __half2*>(&t1));
      v[rb][u][0] *= f0; v[rb][u][1] *= f0; v[rb][u][2] *= f1; v[rb][u][3] *= f1;
      d0 += a.x * v[rb][u][0] + a.y * v[rb][u][1];
      d1 += b.x * v[rb][u][2] + b.y * v[rb][u][3];
    }
#pragma unroll
    for (int off = 1; off < 4; off <<= 1) {
      d0 += __shfl_xor_sync(0xffffffffu, d0, off);
      d1 += __shfl_xor_sync(0xffffffffu, d1, off);
    }
    if (q == 0) { out[i] = d0; out[i + 8] = d1; }
  }
}

// Gradients of heads h_first .. h_end - 1 of a group in one segment; gB and gC of the heads stay in registers.
// The first 256 threads of the CTA; thread (ty, tx): scores as in segment_scores; everything else rows 4 ty .. 4 ty + 3, head columns 4 tx .. 4 tx + 3, state columns
// 4 tx .. 4 tx + 3 and those 64 further.
__device__ __noinline__ void segment_reverse_plain(const SegArgs& g, float* smem, int b, int seg, int grp, int split, int h_first, int h_end) {
  float* sB = smem;                              // [64][132]
  float* sC = sB + SG_Q * SG_NPITCH;             // [64][132]
  float* sG = sC + SG_Q * SG_NPITCH;             // [64][68] G
  float* sMG = sG + SG_Q * SG_PPITCH;            // [64][68] M G
  float* sMX = sMG + SG_Q * SG_PPITCH;           // [64][68] M X
  float* sX = sMX + SG_Q * SG_PPITCH;            // [64][68]
  float* sGy = sX + SG_Q * SG_PPITCH;            // [64][68]
  float* sS = sGy + SG_Q * SG_PPITCH;            // [128][64] state: Y, then H
  double* cum = reinterpret_cast<double*>(sS + SG_N * SG_P);
  float* dt = reinterpret_cast<float*>(cum + SG_Q);
  float* su = dt + SG_Q;                         // [64] exp(cum_i) <C_i, H gy_i>
  float* sv = su + SG_Q;                         // [64] e_j <B_j, Y x_j>
  float* part = sv + SG_Q;                       // [2][8 warps][64]: parts of s and ga from inside the segment
  float* red = part + 2 * 8 * SG_Q;              // [8]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  const int t0 = seg * SG_Q, rows = min(SG_Q, g.L - t0);
  const bool before = seg > 0, behind = seg < g.nseg - 1;
  const size_t row = static_cast<size_t>(b) * g.L + t0;
  const int r0 = ty * 4, c0 = tx * 4, rb = ty / 4 * 16;   // rb: first row of the 16-row block (the same for a whole warp)
  plain_tile<SG_N, SG_NPITCH, SG_THREADS>(sB, g.Bm + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows);
  plain_tile<SG_N, SG_NPITCH, SG_THREADS>(sC, g.Cm + (row * g.G + grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows);
  named_bar_sync(1, SG_THREADS);
  {
    float s[4][4];
    segment_scores<SG_N, SG_NPITCH>(sC, sB, ty, tx, s);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v <= u; ++v) sG[(ty + 16 * u) * SG_PPITCH + tx + 16 * v] = s[u][v];
  }
  float gB[4][8] = {}, gC[4][8] = {};
#pragma unroll 1
  for (int h = h_first; h < h_end; ++h) {
    const size_t unit = (static_cast<size_t>(b) * g.H + h) * g.nseg + seg;
    const size_t yunit = static_cast<size_t>(g.B) * g.H * g.nseg + unit;
    const float *hstate = g.states + unit * (SG_N * SG_P), *ystate = g.states + yunit * (SG_N * SG_P);
    named_bar_sync(1, SG_THREADS);   // the previous head's tiles and scalars have been read (and sG is complete)
    if (warp == 0) segment_scalars(g, b, h, t0, cum, dt, lane);
    plain_tile<SG_P, SG_PPITCH, SG_THREADS>(sX, g.x + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows);
    plain_tile<SG_P, SG_PPITCH, SG_THREADS>(sGy, g.gy + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows);
    if (behind) plain_state<SG_THREADS>(sS, ystate);
    named_bar_sync(1, SG_THREADS);
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
    named_bar_sync(1, SG_THREADS);
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
    named_bar_sync(1, SG_THREADS);   // Y has been read
    float pin = 0.f;
    if (before) {
#pragma unroll 1
      for (int idx = threadIdx.x; idx < SG_N * SG_P; idx += SG_THREADS) {
        const int p = idx / SG_N, n = idx % SG_N;
        const float v = hstate[idx];
        if (behind) pin += v * ystate[idx];
        sS[state_at(n, p >> 2) + (p & 3)] = v;
      }
      pin = warp_reduce<SumOp>(pin);
    }
    if (lane == 0) red[warp] = pin;
    named_bar_sync(1, SG_THREADS);
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
    named_bar_sync(1, SG_THREADS);   // su, sv, red
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

__global__ void __launch_bounds__(SR_THREADS, 1) segment_reverse_kernel(const SegArgs g) {
  mp_grid_dependency();
  extern __shared__ __align__(128) unsigned char seg_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3, r0 = lane >> 2;
  const int cols = warp & 7, part = warp >> 3;
  const SegShare sh = segment_share(g);
  const int t0 = sh.seg * SG_Q, rows = min(SG_Q, g.L - t0);
  const bool before = sh.seg > 0, behind = sh.seg < g.nseg - 1;
  const size_t row = static_cast<size_t>(sh.b) * g.L + t0;
  const uint32_t smem = mp_smem_u32(seg_smem), sB = smem, sC = sB + SG_Q * SG_N * 2, stages = sC + SG_Q * SG_N * 2, sY = stages + 2 * SR_STAGE;
  const uint32_t sW = sY + SG_STATE_BYTES, sM = sW + SG_Q * SG_Q * 4;   // M X dt, M G
  SegSteps* steps = reinterpret_cast<SegSteps*>(seg_smem + SR_TILES);
  SegScalars* scalars = reinterpret_cast<SegScalars*>(steps + 3);
  auto unit_of = [&](int h) { return (static_cast<size_t>(sh.b) * g.H + h) * g.nseg + sh.seg; };
  auto load_stage = [&](int h) {
    const uint32_t st = stages + ((h - sh.h_first) & 1) * SR_STAGE;
    tile_load<SG_P / 8, SR_THREADS>(st, g.x + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows, g.vec);
    tile_load<SG_P / 8, SR_THREADS>(st + SR_X, g.gy + (row * g.H + h) * SG_P, static_cast<size_t>(g.H) * SG_P, rows, g.vec);
    if (before) state_load<SR_THREADS>(st + 2 * SR_X, g.states + unit_of(h) * (SG_N * SG_P));
  };
  auto load_adjoint = [&](int h) {
    const size_t unit = static_cast<size_t>(g.B) * g.H * g.nseg + unit_of(h);
    if (behind) state_load<SR_THREADS>(sY, g.states + unit * (SG_N * SG_P));
  };
  tile_load<SG_N / 8, SR_THREADS>(sB, g.Bm + (row * g.G + sh.grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec);
  tile_load<SG_N / 8, SR_THREADS>(sC, g.Cm + (row * g.G + sh.grp) * SG_N, static_cast<size_t>(g.G) * SG_N, rows, g.vec);
  cp_async_commit();
  load_stage(sh.h_first);
  load_adjoint(sh.h_first);
  cp_async_commit();
  if (warp == 15) segment_steps(g, sh.b, sh.h_first, t0, steps[0], lane);
  cp_async_wait<1>();
  __syncthreads();
  float G[2][4];   // C B^T of the warp's block
  int ib, jb;
  const bool scores = block_of(warp, ib, jb);
  if (scores) block_scores<SG_N>(G, sC, sB, ib, jb, lane);
  float gB[2][2][4] = {}, gC[2][2][4] = {};
  float check = 0.f;   // becomes NaN with the first result that is none, or infinite
#pragma unroll 1
  for (int h = sh.h_first; h < sh.h_end; ++h) {
    const int n = h - sh.h_first;
    const uint32_t sx = stages + (n & 1) * SR_STAGE, sgy = sx + SR_X, sH = sgy + SR_X;
    cp_async_wait<0>();
    __syncthreads();   // this head's tiles are there, the other stage, the weights and the last head's scalars are complete and read
    if (h + 1 < sh.h_end) {
      load_stage(h + 1);
      if (warp == 15) segment_steps(g, sh.b, h + 1, t0, steps[(n + 1) % 3], lane);
    }
    cp_async_commit();
    if (warp == 14 && n > 0) segment_gradients(g, scalars[(n - 1) & 1], steps[(n - 1) % 3], h - 1, row, rows, unit_of(h - 1), lane);
    SegScalars& sc = scalars[n & 1];
    const SegSteps& st = steps[n % 3];
    // ---- scores: M X dt and M G, the sums of M G X ----
    if (scores) {
      float x[2][4], m[2][4], w[2][4];
      block_scores<SG_P>(x, sgy, sx, ib, jb, lane);
      block_decays(m, st.cum, ib, jb, r0, q);
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          x[u][e] *= m[u][e];
          w[u][e] = x[u][e] * G[u][e];
          m[u][e] *= G[u][e];
        }
      if (ib == jb)   // beyond the diagonal a score may be infinite
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (u * 8 + 2 * q + (e & 1) > r0 + (e >> 1) * 8) x[u][e] = w[u][e] = m[u][e] = 0.f;
      block_sums(w, st.dt, sc, ib, jb, lane);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 dj = *reinterpret_cast<const float2*>(st.dt + jb * 16 + u * 8 + 2 * q);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[u][e] *= e & 1 ? dj.y : dj.x;
      }
      block_store(x, sW, ib, jb, lane);
      block_store(m, sM, ib, jb, lane);
    }
    {   // ---- <Y, H> ----
      float pin = 0.f;
      if (before && behind) {
#pragma unroll
        for (int k = 0; k < SG_STATE_BYTES / 16 / SR_THREADS; ++k) {
          const int idx = k * SR_THREADS + threadIdx.x;
          const float4 a = ld_shared16f(wide_at<512>(sY, idx >> 5, idx & 31)), b = ld_shared16f(wide_at<512>(sH, idx >> 5, idx & 31));
          pin += (a.x * b.x + a.y * b.y) + (a.z * b.z + a.w * b.w);
        }
        pin = warp_reduce<SumOp>(pin);
      }
      if (lane == 0) sc.pin[warp] = pin;
    }
    // ---- the adjoint state's part of gB and gx ----
    float o[2][1][4];
    if (behind) {
      float v[2][2][4], p[2][4];
      times_state_n<2>(v, sx, sY, cols, part, lane);
      row_dots(v, st.left, sB, cols, sc.sv[cols], part, lane);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = row_block<2>(i, part) * 16 + r0;
        const float d0 = st.dt[r], d1 = st.dt[r + 8];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e) gB[i][u][e] = fmaf(e < 2 ? d0 : d1, v[i][u][e], gB[i][u][e]);
      }
      times_state_p<2>(p, sB, sY, cols, part, lane);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = row_block<2>(i, part) * 16 + r0;
        const float e0 = st.left[r], e1 = st.left[r + 8];
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][0][e] = p[i][e] * (e < 2 ? e0 : e1);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][0][e] = 0.f;
      if (part == 0 && lane < 16) *reinterpret_cast<float4*>(sc.sv[cols] + lane * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();   // the weights are complete, Y has been read
    if (h + 1 < sh.h_end) load_adjoint(h + 1);
    cp_async_commit();
    // ---- gx ----
    {
      uint32_t b[4][2];
      load_steps(b, sgy, cols, lane);
      times_scores<2, false, 1>(o, sM, b, part, lane);
      __half* gx = g.gx + (row * g.H + h) * SG_P + cols * 8 + 2 * q;
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int j = row_block<2>(i, part) * 16 + r * 8 + r0;
          const float d = st.dt[j];
          check = fmaf(o[i][0][2 * r], 0.f, fmaf(o[i][0][2 * r + 1], 0.f, check));
          if (j < rows) store_pair(gx + static_cast<size_t>(j) * g.H * SG_P, o[i][0][2 * r] * d, o[i][0][2 * r + 1] * d, g.vec);
        }
    }
    // ---- gC, gB ----
    if (before) {
      float v[2][2][4];
      times_state_n<2>(v, sgy, sH, cols, part, lane);
      row_dots(v, st.grow, sC, cols, sc.su[cols], part, lane);
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e) gC[i][u][e] += v[i][u][e];
    } else if (part == 0 && lane < 16) {
      *reinterpret_cast<float4*>(sc.su[cols] + lane * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    uint32_t b[4][4];   // these columns of B, then of C, over the steps
#pragma unroll
    for (int k = 0; k < 4; ++k) load_b_t<SG_N * 2>(b[k], sB, k * 16, cols * 2, lane);
    times_scores<2, true, 2>(gC, sW, b, part, lane);
#pragma unroll
    for (int k = 0; k < 4; ++k) load_b_t<SG_N * 2>(b[k], sC, k * 16, cols * 2, lane);
    times_scores<2, false, 2>(gB, sW, b, part, lane);
  }
  const size_t bc = static_cast<size_t>(g.B) * g.L * g.G * SG_N;
  float* out = g.gb_part + static_cast<size_t>(sh.split) * 2 * bc + (row * g.G + sh.grp) * SG_N + cols * 16 + 2 * q;
#pragma unroll
  for (int rb = 0; rb < 2; ++rb)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int i = row_block<2>(rb, part) * 16 + r * 8 + r0;
        const float b0 = gB[rb][u][2 * r], b1 = gB[rb][u][2 * r + 1], c0 = gC[rb][u][2 * r], c1 = gC[rb][u][2 * r + 1];
        check = fmaf(b0, 0.f, fmaf(b1, 0.f, fmaf(c0, 0.f, fmaf(c1, 0.f, check))));
        if (i >= rows) continue;
        float* o = out + static_cast<size_t>(i) * g.G * SG_N + u * 8;
        *reinterpret_cast<float2*>(o) = make_float2(b0, b1);
        *reinterpret_cast<float2*>(o + bc) = make_float2(c0, c1);
      }
  const bool again = __syncthreads_or(check != 0.f);
  if (warp == 14) {
    const int n = sh.h_end - 1 - sh.h_first;
    segment_gradients(g, scalars[n & 1], steps[n % 3], sh.h_end - 1, row, rows, unit_of(sh.h_end - 1), lane);
  }
  if (again) {
    __syncthreads();
    if (threadIdx.x < SR_THREADS / 2) segment_reverse_plain(g, reinterpret_cast<float*>(seg_smem), sh.b, sh.seg, sh.grp, sh.split, sh.h_first, sh.h_end);
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
constexpr size_t SG_PLAIN_FORWARD = SG_Q * 2 * (SG_NPITCH + SG_PPITCH) * sizeof(float) + SG_SCALARS;
constexpr size_t SG_PLAIN_REVERSE = (SG_Q * (2 * SG_NPITCH + 5 * SG_PPITCH) + SG_N * SG_P + (2 + 16) * SG_Q + 8) * sizeof(float) + SG_SCALARS;
constexpr size_t SG_SMEM_FORWARD = SF_SMEM > SG_PLAIN_FORWARD ? SF_SMEM : SG_PLAIN_FORWARD;
constexpr size_t SG_SMEM_REVERSE = SR_SMEM > SG_PLAIN_REVERSE ? SR_SMEM : SG_PLAIN_REVERSE;
static_assert(SG_N * SG_P <= SG_Q * SG_NPITCH, "the state takes the place of B");
static_assert(2 * SG_SMEM_FORWARD <= 226 * 1024 && SG_SMEM_REVERSE <= 227 * 1024, "shared memory of an SM");
static_assert(SF_TILES % 128 == 0 && SR_STAGE % 128 == 0, "tiles keep the phase of their chunks");

// Shares of a group's heads: a CTA's time is its heads' and about `setup` heads' worth of loading, scores and writing of gB and gC (which
// are also folded over the shares: `fold` per CTA of the whole grid), `slots` CTAs run at a time.
int segment_splits(int B, int L, int H, int G, int slots, float setup, float fold) {
  const long units = static_cast<long>(B) * ((L + SG_Q - 1) / SG_Q) * G;
  const int hpg = H / G;
  int best = 1;
  float best_cost = 0.f;
  for (int s = 1; s <= hpg; ++s) {
    const int heads = (hpg + s - 1) / s;
    if (s > 1 && heads == (hpg + s - 2) / (s - 1)) continue;   // no fewer heads than with one share less
    const float cost = static_cast<float>((units * s + slots - 1) / slots) * (heads + setup) + fold * units * s;
    if (s == 1 || cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}
int forward_splits(int B, int L, int H, int G) { return segment_splits(B, L, H, G, 2 * 148, 0.7f, 0.f); }
int reverse_splits(int B, int L, int H, int G) { return segment_splits(B, L, H, G, 148, 0.7f, 0.005f); }

struct SegScratch { float* states; float* decay; float* ga_part; float* gb_part; size_t total; };
SegScratch segment_carve(void* base, int B, int L, int H, int G, bool reverse) {
  SegScratch s;
  const size_t start = (256 - (reinterpret_cast<uintptr_t>(base) & 255)) & 255;   // the caller's pointer may have any alignment
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* p = base != nullptr ? static_cast<unsigned char*>(base) + start + off : nullptr;
    off += (bytes + 255) & ~size_t(255);
    return p;
  };
  const size_t units = static_cast<size_t>(B) * H * ((static_cast<size_t>(L) + SG_Q - 1) / SG_Q);
  s.states = reinterpret_cast<float*>(take(units * SG_STATE_BYTES * (reverse ? 2 : 1)));
  s.decay = reinterpret_cast<float*>(take(units * sizeof(float)));
  s.ga_part = reinterpret_cast<float*>(take(reverse ? units * sizeof(float) : 0));
  s.gb_part = reinterpret_cast<float*>(take(reverse ? static_cast<size_t>(reverse_splits(B, L, H, G)) * 2 * B * L * G * SG_N * sizeof(float) : 0));
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
  if (g.nseg == 1) return;
  MP_CUDA_CHECK(cudaFuncSetAttribute(segment_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SS_SMEM)));
  MpLaunch(dim3(g.B * g.H * g.nseg, directions), SS_THREADS, SS_SMEM, st)(segment_states_kernel, g);
  MP_LAUNCH_CHECK();
  MpLaunch(dim3(g.B * g.H * (SG_N * SG_P / 4 / SC_THREADS), directions), SC_THREADS, 0, st)(segment_carry_kernel, g);
  MP_LAUNCH_CHECK();
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
  g.splits = forward_splits(B, L, H, G);
  segment_state_launches(g, 1, st);
  MP_CUDA_CHECK(cudaFuncSetAttribute(segment_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SG_SMEM_FORWARD)));
  MpLaunch(B * g.nseg * G * g.splits, SG_THREADS, SG_SMEM_FORWARD, st)(segment_forward_kernel, g);
  MP_LAUNCH_CHECK();
}

void mp_ssd_segments_reverse(const void* x, const void* dt, const void* A, const void* Bm, const void* Cm, const void* gy, void* gx, void* gdt,
                             void* gA, void* gB, void* gC, void* scratch, int B, int L, int H, int G, cudaStream_t st) {
  SegArgs g = segment_args(x, dt, A, Bm, Cm, segment_carve(scratch, B, L, H, G, true), B, L, H, G);
  g.gy = static_cast<const __half*>(gy); g.gx = static_cast<__half*>(gx); g.gdt = static_cast<float*>(gdt);
  g.splits = reverse_splits(B, L, H, G);
  const bool fold_vec = mp_aligned16(gB) && mp_aligned16(gC);
  g.vec = g.vec && mp_aligned16(gy) && mp_aligned16(gx);
  segment_state_launches(g, 2, st);
  MP_CUDA_CHECK(cudaFuncSetAttribute(segment_reverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SG_SMEM_REVERSE)));
  MpLaunch(B * g.nseg * G * g.splits, SR_THREADS, SG_SMEM_REVERSE, st)(segment_reverse_kernel, g);
  MP_LAUNCH_CHECK();
  const size_t bc = static_cast<size_t>(B) * L * G * SG_N;
  MpLaunch(dim3(static_cast<unsigned>((bc / 4 + SG_THREADS - 1) / SG_THREADS), 2), SG_THREADS, 0, st)(segment_fold_kernel, g.gb_part, static_cast<__half*>(gB),
                                                                                                   static_cast<__half*>(gC), bc, g.splits, fold_vec);
  MpLaunch(H, 32, 0, st)(segment_sum_kernel, g.ga_part, static_cast<float*>(gA), B, H, g.nseg);
  MP_LAUNCH_CHECK();
}
