// What the contraction kernels of gemm.cu (r16) and gemm_r32.cu share: the problem description, the store of blocks that
// TMA cannot write, the split-K fold and the tensor maps.
#pragma once

#include "mp_tcgen05.cuh"

#include <cuda.h>
#include <mutex>

struct GemmArgs {
  const void* bias;   // N values of T (bias_pitch = 0), a full [M, N] matrix (bias_pitch = N), or nullptr
  size_t bias_pitch = 0;
  void* c;            // [M, N] row-major, row pitch ldc
  size_t ldc;
  float alpha, beta;
  int M, N, K;
  int a_mn, b_mn;     // operand major-ness: 0 = K contiguous, 1 = M resp. N contiguous
  int stages;
  int group = 0;      // pair kernel: row blocks per group of tiles (see pair_tile); 0: all of them
  int exact = 0;      // sum as exactly as the FP pipe does (the EXACT forms of the kernels)
  int epi_boxes = 2;  // pair kernel: 64-column staging boxes per epilogue warp
  int split;          // r32 only: 1 = error-compensated hi/lo split (3 MMAs per k-slice), 0 = one tf32 MMA (for timing)
  int ksplit;         // > 1: the K range of every tile is cut into ksplit work units whose raw fp32
  float* partial;     //      accumulators go to partial[unit_split][M][partial_ld]; a fold kernel finishes C
  int partial_ld;     // N rounded up to four columns
  int batch;          // > 1: densely packed [batch, M, K] x [batch, K, N] -> [batch, M, N] over 3-D tensor maps (ksplit = 1)
  uint32_t* status;
};

// An operand as the tensor maps see it: rows of `ld` elements, 16-byte aligned.
template <typename T> struct Operand { const T* p; size_t ld; };

namespace {

constexpr int BM = 128;               // UMMA M (one TMEM lane per output row)
constexpr int SWIZZLE_BYTES = 128;    // one operand row / k-row in shared memory

// One 32 x 32 block of a tile (lane = row, r = its 32 columns) into a C that TMA and 16-byte stores cannot write: odd row
// pitch or base, or the last columns under beta.  A lane's own row is 32 separate sectors per store instruction, so the block is
// turned around through 4 KB of the warp's staging (column XOR row: no bank conflicts either way) and leaves one row per
// instruction; the matrix term and the old C come in the same way.  Eight rows are read before the first of them is written: a row read
// behind the write of the one before it took 200 cycles (r16 [1500, 777] x [777, 1030]: 12 500 of the kernel's 24 600).
template <typename T>
__device__ __forceinline__ void store_block_rows(float* stage, const float* r, int lane, T* c, size_t ldc, int rows, bool col_in, const T* mat,
                                                 size_t mat_ld, float beta) {
#pragma unroll
  for (int j = 0; j < 32; ++j) stage[lane * 32 + (j ^ lane)] = r[j];
  __syncwarp();
  T* p = c + lane;
  const T* q = mat != nullptr ? mat + lane : nullptr;
#pragma unroll 1
  for (int i0 = 0; i0 < rows; i0 += 8) {
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = stage[(i0 + u) * 32 + (lane ^ (i0 + u))];
    const int n = col_in ? min(8, rows - i0) : 0;
    if (q != nullptr) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (u < n) v[u] += mp_up(q[u * mat_ld]);
      q += 8 * mat_ld;
    }
    if (beta != 0.0f) {
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (u < n) v[u] += beta * mp_up(p[u * ldc]);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (u < n) p[u * ldc] = mp_down<T>(v[u]);
    p += 8 * ldc;
  }
  __syncwarp();
}

// The same for r16 results that are neither scaled nor added to: up to 64 columns (two blocks, `second` the right one), staged as words of two
// and written as words.  A row may begin in the middle of one: then its words are put together from neighbours, and its first and last
// element leave alone.  (Two-byte stores take three times as long as words: [1500, 777] x [777, 1030] with its copies 18.0 us with them, 14.7 now.)
__device__ __forceinline__ void stage_half_words(uint32_t* stage, const float* r, int lane, int second) {
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const __half2 h = __floats2half2_rn(r[2 * k], r[2 * k + 1]);
    stage[lane * 32 + ((second * 16 + k) ^ lane)] = *reinterpret_cast<const uint32_t*>(&h);
  }
}
__device__ __forceinline__ void store_half_rows(const uint32_t* stage, int lane, __half* c, size_t ldc, int rows, int cols) {
  __syncwarp();
  unsigned short* p = reinterpret_cast<unsigned short*>(c);
  const int e = 2 * lane;   // this lane's elements: e, e + 1
#pragma unroll 1
  for (int i0 = 0; i0 < rows; i0 += 8) {
    uint32_t v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = stage[(i0 + u) * 32 + (lane ^ (i0 + u))];
#pragma unroll
    for (int u = 0; u < 8; ++u, p += ldc) {
      if (i0 + u >= rows) break;   // (uniform, as is the branch below)
      if ((reinterpret_cast<uintptr_t>(p) & 2u) == 0) {
        if (e + 1 < cols) *reinterpret_cast<uint32_t*>(p + e) = v[u];
        else if (e < cols) p[e] = static_cast<unsigned short>(v[u]);
      } else {
        const uint32_t next = __shfl_down_sync(0xffffffffu, v[u], 1);
        if (e + 2 < cols) *reinterpret_cast<uint32_t*>(p + e + 1) = __byte_perm(v[u], next, 0x5432);
        else if (e + 1 < cols) p[e + 1] = static_cast<unsigned short>(v[u] >> 16);
        if (lane == 0) p[0] = static_cast<unsigned short>(v[u]);
      }
    }
  }
  __syncwarp();
}

// An operand split into hi + lo makes a NaN of every infinite value (lo = inf - inf) and of values that round up to infinity, and with it
// of every result they enter.  A result that comes out as NaN is therefore summed once more from the operands themselves, by fused
// multiply-adds in the order of K: infinities and overflows come out as the FP pipe has them, and what is NaN there remains one.
__device__ __noinline__ float dot_again(const float* a, size_t a_step, const float* b, size_t b_step, int k) {
  float s = 0.f;
#pragma unroll 4
  for (; k > 0; --k) {
    s = fmaf(*a, *b, s);
    if (s != s) break;
    a += a_step;
    b += b_step;
  }
  return s;
}
// The operands of an EXACT r32 contraction, for that.
struct Again {
  const float* a;
  const float* b;
  size_t a_ld, b_ld;
  __device__ __forceinline__ float operator()(const GemmArgs& g, int bz, int row, int col) const { return at(g.a_mn, g.b_mn, g.M, g.N, g.K, bz, row, col); }
  __device__ __forceinline__ float at(int a_mn, int b_mn, int M, int N, int K, int bz, int row, int col) const {
    return dot_again(a + static_cast<size_t>(bz) * (a_mn ? K : M) * a_ld + (a_mn ? row : row * a_ld), a_mn ? a_ld : 1,
                     b + static_cast<size_t>(bz) * (b_mn ? K : N) * b_ld + (b_mn ? col : col * b_ld), b_mn ? b_ld : 1, K);
  }
};
struct AgainFold { Again again; int a_mn, b_mn, K; };   // one problem, K cut into parts
struct NoAgain {};

// C = alpha * sum_s partial[s] + bias + beta * C  (finishes a split-K contraction).  A thread folds four neighbouring columns
// of a row; partial rows have a pitch of whole fours whatever N is.
template <typename T, typename R>
__global__ void __launch_bounds__(256) gemm_fold_kernel(const float* __restrict__ partial, int ksplit, int M, int N, int ld, float alpha,
                                                        const T* __restrict__ bias, float beta, T* c, size_t ldc, size_t bias_pitch,
                                                        const R r) {
  mp_grid_dependency();
  const size_t mn = static_cast<size_t>(M) * ld;
  const size_t i0 = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) * 4;
  if (i0 >= mn) return;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
  for (int sidx = 0; sidx < ksplit; ++sidx) {
    const float4 v = *reinterpret_cast<const float4*>(partial + sidx * mn + i0);
    acc[0] += v.x; acc[1] += v.y; acc[2] += v.z; acc[3] += v.w;
  }
  const int per_row = ld / 4;
  const size_t unit = i0 / 4;
  const size_t row = unit < (size_t(1) << 32) ? static_cast<uint32_t>(unit) / static_cast<uint32_t>(per_row) : unit / per_row;
  const int col = static_cast<int>(unit - row * per_row) * 4;
  T* cr = c + row * ldc + col;
  const T* br = bias != nullptr ? bias + row * bias_pitch + col : nullptr;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (col + e < N) {
      if constexpr (std::is_same<R, AgainFold>::value) {
        if (acc[e] != acc[e]) acc[e] = r.again.at(r.a_mn, r.b_mn, M, N, r.K, 0, static_cast<int>(row), col + e);
      }
      float o = alpha * acc[e];
      if (br != nullptr) o += mp_up(br[e]);
      if (beta != 0.0f) o += beta * mp_up(cr[e]);
      acc[e] = o;
    }
  }
  if (col + 4 <= N && (ldc * sizeof(T)) % 16 == 0 && mp_aligned16(c)) {
    struct alignas(4 * sizeof(T)) Four { T v[4]; } f;
#pragma unroll
    for (int e = 0; e < 4; ++e) f.v[e] = mp_down<T>(acc[e]);
    *reinterpret_cast<Four*>(cr) = f;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (col + e < N) cr[e] = mp_down<T>(acc[e]);
  }
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, []() {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    MP_CUDA_CHECK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres));
    if (p == nullptr || qres != cudaDriverEntryPointSuccess) MP_FATAL("cuTensorMapEncodeTiled is not available");
    fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// 2-D row-major matrix [rows, cols] of T, box = {box_cols (128 bytes), box_rows}, out-of-range
// elements read as zero.
// ld: row pitch in elements.  batch > 1: [batch, rows, ld] as a 3-D tensor, boxes one batch entry deep.
template <typename T>
CUtensorMap make_map(const void* base, size_t rows, size_t cols, size_t ld, uint32_t box_cols, uint32_t box_rows,
                     CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B, size_t batch = 1) {
  CUtensorMap map;
  const cuuint64_t dims[3] = {cols, rows, batch};
  const cuuint64_t strides[2] = {ld * sizeof(T), rows * ld * sizeof(T)};
  const cuuint32_t box[3] = {box_cols, box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUtensorMapDataType dt = sizeof(T) == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  MP_CU_CHECK(encode_tiled()(&map, dt, batch > 1 ? 3 : 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             swizzle,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
  return map;
}

// Row-major [rows, cols] output, box {32 cols, 32 rows} unswizzled, or (wide) {64 cols, 32 rows} of r16 in the
// 128-byte swizzle.
template <typename T>
CUtensorMap make_store_map(void* base, size_t rows, size_t cols, size_t ld, bool wide = false, size_t batch = 1) {
  CUtensorMap map;
  const cuuint64_t dims[3] = {cols, rows, batch};
  const cuuint64_t strides[2] = {ld * sizeof(T), rows * ld * sizeof(T)};
  const cuuint32_t box[3] = {wide ? 64u : 32u, 32, 1};
  const bool swizzle = wide || sizeof(T) == 4;   // 128-byte rows: r16 wide boxes and every r32 box
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUtensorMapDataType dt = sizeof(T) == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  MP_CU_CHECK(encode_tiled()(&map, dt, batch > 1 ? 3 : 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
  return map;
}

template <typename T, typename R>
void launch_fold(const GemmArgs& args, const R& again, cudaStream_t st) {
  const size_t units = static_cast<size_t>(args.M) * args.partial_ld / 4;
  MpLaunch(static_cast<unsigned>((units + 255) / 256), 256, 0, st)(gemm_fold_kernel<T, R>, args.partial, args.ksplit, args.M, args.N, args.partial_ld,
                                                                                args.alpha, static_cast<const T*>(args.bias), args.beta,
                                                                                static_cast<T*>(args.c), args.ldc, args.bias_pitch, again);
  MP_LAUNCH_CHECK();
}

bool env_flag(const char* name) {
  const char* e = getenv(name);
  return e != nullptr && e[0] != '\0' && e[0] != '0';
}

}  // namespace

// gemm_r32.cu: one r32 contraction whose operands TMA can address; picks the tile and the K split itself.
void gemm_run_r32(Operand<float> a, Operand<float> b, GemmArgs args, int sms, void* workspace, size_t workspace_bytes, cudaStream_t st);
// Its estimate in cycles, with the tile and the K split that give it.
double gemm_r32_estimate(const GemmArgs& args, int sms, size_t workspace_bytes, int* bn, int* ksplit);
// gemm_r32_terms.cu: the same from three bf16 terms per value, for any operand alignment; false (and nothing done) where it would take longer than
// `limit_cycles` or its copies do not fit.
bool gemm_run_r32_terms(Operand<float> a, Operand<float> b, GemmArgs args, int sms, void* workspace, size_t workspace_bytes, double limit_cycles,
                        cudaStream_t st);
