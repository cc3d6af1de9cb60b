// bf16 GEMM for at most 64 rows (decode steps of a few sentences), with the RMSNorm in front of
// it and the residual add or gated GELU behind it in the same launch:
//
//   C[M, N] = epi(norm(A)[M, K] * B[K, N])        B row-major (T5X kernel layout), M <= 64
//
// What bounds it: nothing but latency and the weight bytes. A decode step of four sentences of
// T5.1.1 base runs 72 such products of 0.2 to 0.8 us worth of weights each; on the tcgen05
// kernels one took 8 to 10 us (descriptor and TMEM set-up, a 128-row tile of which 124 rows are
// padding, the exchange of split-K partial tiles between SMs) and every norm was a 3.2 us launch
// of its own. Here a CTA owns 16 (wide outputs: 32 or 64) columns and the whole of K, so no
// partial sum leaves the SM:
//   * its eight warps take every eighth 16-deep k step each and copy their weights with cp.async
//     into a ring of their own, 64 KB a CTA, requested before anything else: the weights are on
//     their way while the rows of A are normalised (a programmatic dependent launch requests
//     them before the kernel in front has finished). With register staging, 8 requests ahead, a
//     2048 x 5120 gated product ran at 1.2 TB/s;
//   * A (all rows) sits in shared memory as bf16, normalised in place by one warp per row, or by
//     two, four or eight when there are fewer rows than warps: y = x * rstd * scale, rounded to
//     bf16 exactly as the separate norm kernel stores it;
//   * `mma.sync.m16n8k16` does the products: 16 rows are its natural operand, a tcgen05 tile
//     would be seven eighths padding and the product is bound by the weight stream anyway. The
//     weight tile is read transposed (`ldmatrix.trans`); rows of the A operand beyond M repeat
//     the last one, they only reach rows of C that are not stored;
//   * the warps' fp32 partial tiles are added in shared memory and the epilogue stores 32-byte
//     row pieces.
#include "gemm_common.cuh"
#include "t5x_b200.h"

namespace t5x {
namespace {

constexpr int kRowWarps = 8;
constexpr int kRowThreads = kRowWarps * 32;
constexpr int kRowCols = 16;              // columns of C per CTA and column tile (NT of them)
constexpr int kRowMaxRows = 64;
constexpr int kRowMaxSmem = 224 * 1024;
constexpr int kRowWeightBuf = 512;        // one 16 x 16 bf16 tile
constexpr int kRowRingTiles = 16;         // of a warp's ring: 64 KB of weights in flight per CTA

struct RowGemmParams {
  const __nv_bfloat16* A;
  const __nv_bfloat16* B;
  const __nv_bfloat16* B2;      // gated: second weight
  const float* norm_scale;      // [K] or null
  const __nv_bfloat16* R;       // residual or null
  void* C;
  long long lda, ldb, ldc, ldr;
  int M, N, K;
  int out_fp32;
  float eps, alpha;
  int b_constant;               // B may be requested before the preceding kernel has finished
};

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
      "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void unpack8_bf16(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __bfloat1622float2(h[j]);
    f[2 * j] = t.x;
    f[2 * j + 1] = t.y;
  }
}

// elements between rows of A in shared memory: 16 bytes more than K, so that the eight row
// pieces of an ldmatrix fall into different banks when K is a multiple of 64
__host__ __device__ constexpr int row_pitch(int K) { return K + 8; }

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int MT, int NT, bool GATED>
__global__ void __launch_bounds__(kRowThreads)
    gemm_rows_kernel(const RowGemmParams p) {
  constexpr int kMats = GATED ? 2 : 1;
  constexpr int kPieces = kMats * NT;              // 16 x 16 weight tiles per k step
  constexpr int kAhead = kRowRingTiles / kPieces;  // k steps of a warp in flight
  constexpr int kCols = kRowCols * NT;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __shared__ float s_ss[kRowMaxRows][kRowWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ring = smem_u32(smem_raw) + warp * kRowRingTiles * kRowWeightBuf;
  __nv_bfloat16* sA =
      reinterpret_cast<__nv_bfloat16*>(smem_raw + kRowWarps * kRowRingTiles * kRowWeightBuf);
  const int pitch = row_pitch(p.K);
  const int n0 = blockIdx.x * kCols;
  const int steps = p.K / 16;

  // ---- weights: of each 16 x 16 tile lane l copies 8 columns (half l & 1) of row l >> 1; the
  // tile has 32-byte rows, the halves swapped every four rows (bank conflicts of ldmatrix) ----
  const int wrow = lane >> 1, whalf = lane & 1;
  const long long w_off = static_cast<long long>(wrow) * p.ldb + n0 + whalf * 8;
  const uint32_t w_st = ring + wrow * 32 + ((whalf ^ ((wrow >> 2) & 1)) * 16);
  auto request = [&](int i, int slot) {  // i-th step of this warp
    const int s = warp + i * kRowWarps;
    if (s < steps) {
      const long long off = w_off + static_cast<long long>(s) * 16 * p.ldb;
      const uint32_t dst = w_st + slot * kPieces * kRowWeightBuf;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        cp_async_16(dst + n * kRowWeightBuf, p.B + off + n * kRowCols);
        if (GATED)
          cp_async_16(dst + ((kMats - 1) * NT + n) * kRowWeightBuf, p.B2 + off + n * kRowCols);
      }
    }
    cp_async_commit();  // one group per step, also beyond the last
  };
  chain_release();
  if (!p.b_constant) chain_wait();
#pragma unroll
  for (int i = 0; i < kAhead; ++i) request(i, i);
  if (p.b_constant) chain_wait();

  // ---- A rows -> shared memory: `per_row` warps share a row ----
  const int nvec = p.K / 8;
  const int per_row = p.M <= 1 ? 8 : (p.M <= 2 ? 4 : (p.M <= 4 ? 2 : 1));
  const int first = (warp % per_row) * 32 + lane, stride = per_row * 32;
  for (int r = warp / per_row; r < p.M; r += kRowWarps / per_row) {
    uint4* dst = reinterpret_cast<uint4*>(sA + static_cast<long long>(r) * pitch);
    const uint4* src = reinterpret_cast<const uint4*>(p.A + static_cast<long long>(r) * p.lda);
    float ss = 0.f;
    constexpr int kU = 4;
    for (int v0 = first; v0 < nvec; v0 += kU * stride) {
      uint4 u[kU];
#pragma unroll
      for (int x = 0; x < kU; ++x)
        if (v0 + x * stride < nvec) u[x] = src[v0 + x * stride];
#pragma unroll
      for (int x = 0; x < kU; ++x)
        if (v0 + x * stride < nvec) {
          dst[v0 + x * stride] = u[x];
          float f[8];
          unpack8_bf16(u[x], f);
#pragma unroll
          for (int j = 0; j < 8; ++j) ss += f[j] * f[j];
        }
    }
    if (p.norm_scale != nullptr) {
      ss = warp_sum(ss);
      if (lane == 0) s_ss[r][warp % per_row] = ss;
    }
  }
  __syncthreads();
  if (p.norm_scale != nullptr) {
    for (int r = warp / per_row; r < p.M; r += kRowWarps / per_row) {
      uint4* dst = reinterpret_cast<uint4*>(sA + static_cast<long long>(r) * pitch);
      float ss = 0.f;
      for (int x = 0; x < per_row; ++x) ss += s_ss[r][x];
      const float rstd = rsqrtf(ss / static_cast<float>(p.K) + p.eps);
#pragma unroll 4
      for (int v = first; v < nvec; v += stride) {  // this lane's own pieces again
        const float4 s0 = __ldg(reinterpret_cast<const float4*>(p.norm_scale) + 2 * v);
        const float4 s1 = __ldg(reinterpret_cast<const float4*>(p.norm_scale) + 2 * v + 1);
        const float sc[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
        float f[8];
        unpack8_bf16(dst[v], f);
        uint4 o;
        uint32_t* o32 = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * j] * rstd * sc[2 * j],
                                                         f[2 * j + 1] * rstd * sc[2 * j + 1]);
          o32[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        dst[v] = o;
      }
    }
    __syncthreads();
  }

  // ---- products ----
  float acc[kPieces][MT][2][4];
#pragma unroll
  for (int x = 0; x < kPieces; ++x)
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[x][m][n][e] = 0.f;
  const int lk = ((lane >> 3) & 1) * 8 + (lane & 7);  // row (k) this lane addresses
  const uint32_t w_ld = ring + lk * 32 + (((lane >> 4) ^ ((lk >> 2) & 1)) * 16);
  // A: matrices (rows 0-7, k 0-7), (8-15, 0-7), (0-7, 8-15), (8-15, 8-15)
  uint32_t a_ld[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m)
    a_ld[m] = smem_u32(sA) + (min(m * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), p.M - 1) * pitch +
                              (lane >> 4) * 8) * 2;
  const int mine = (steps - warp + kRowWarps - 1) / kRowWarps;
  for (int i0 = 0; i0 < mine; i0 += kAhead) {
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int i = i0 + u;
      if (i >= mine) break;  // warp-uniform
      cp_async_wait<kAhead - 1>();  // this lane's pieces of step i have landed
      __syncwarp();                 // and every other lane's
      uint32_t b[kPieces][4];
#pragma unroll
      for (int x = 0; x < kPieces; ++x)
        ldsm_x4_trans(w_ld + (u * kPieces + x) * kRowWeightBuf, b[x]);
      __syncwarp();  // the slot may be refilled
      request(i + kAhead, u);
      const int s = warp + i * kRowWarps;
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[4];
        ldsm_x4(a_ld[m] + s * 32, a);
#pragma unroll
        for (int x = 0; x < kPieces; ++x) {
          mma_16816(acc[x][m][0], a, b[x][0], b[x][1]);
          mma_16816(acc[x][m][1], a, b[x][2], b[x][3]);
        }
      }
    }
  }

  // ---- sum over the warps, epilogue ----
  cp_async_wait<0>();
  __syncthreads();  // ring and A are no longer read: their memory holds the partial tiles
  float* red = reinterpret_cast<float*>(smem_raw);  // [warp][matrix][MT * 16 rows][kCols]
  constexpr int kTile = MT * 16 * kCols;
#pragma unroll
  for (int x = 0; x < kPieces; ++x)
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        float* dst = red + (warp * kMats + x / NT) * kTile + (m * 16 + (lane >> 2)) * kCols +
                     (x % NT) * kRowCols + n * 8 + (lane & 3) * 2;
        *reinterpret_cast<float2*>(dst) = make_float2(acc[x][m][n][0], acc[x][m][n][1]);
        *reinterpret_cast<float2*>(dst + 8 * kCols) =
            make_float2(acc[x][m][n][2], acc[x][m][n][3]);
      }
  __syncthreads();
  const int items = min(p.M, MT * 16) * kCols;
  for (int i = threadIdx.x; i < items; i += kRowThreads) {
    const int r = i / kCols, c = n0 + (i & (kCols - 1));
    float v[kMats];
#pragma unroll
    for (int x = 0; x < kMats; ++x) {
      v[x] = 0.f;
#pragma unroll
      for (int g = 0; g < kRowWarps; ++g) v[x] += red[(g * kMats + x) * kTile + i];
    }
    float o = GATED ? gelu_tanh(v[0]) * v[kMats - 1] : v[0] * p.alpha;
    if (p.R != nullptr) o += __bfloat162float(p.R[static_cast<long long>(r) * p.ldr + c]);
    const long long at = static_cast<long long>(r) * p.ldc + c;
    if (p.out_fp32)
      static_cast<float*>(p.C)[at] = o;
    else
      static_cast<__nv_bfloat16*>(p.C)[at] = __float2bfloat16(o);
  }
}

constexpr int round_up_tiles(int M) { return M <= 16 ? 1 : (M <= 32 ? 2 : 4); }

// Column tiles per CTA. Every CTA normalises all of A for itself and reads 32 bytes per weight
// row and tile: wider CTAs where the output still has about one per SM (two for 64 columns).
int column_tiles(int M, int N, bool gated) {
  if (!gated && M <= 16 && N % 64 == 0 && N / 64 >= 2 * num_sms()) return 4;
  return (N % 32 == 0 && N / 32 >= num_sms()) ? 2 : 1;
}

size_t rows_smem(int M, int N, int K, bool gated) {
  const int mt = round_up_tiles(M), mats = gated ? 2 : 1, nt = column_tiles(M, N, gated);
  const size_t a = static_cast<size_t>(M) * row_pitch(K) * 2 +
                   static_cast<size_t>(kRowWarps) * kRowRingTiles * kRowWeightBuf;
  const size_t red = static_cast<size_t>(kRowWarps) * mats * mt * 16 * kRowCols * nt * 4;
  return a > red ? a : red;
}

template <int MT, int NT, bool GATED>
int launch_rows(const RowGemmParams& p, size_t smem, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<MT, NT, GATED>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kRowMaxSmem);
    if (e != cudaSuccess) return set_error("gemm_rows attr: %s", cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  cudaError_t e = launch_chained(gemm_rows_kernel<MT, NT, GATED>, dim3(p.N / (kRowCols * NT)),
                                 dim3(kRowThreads), smem, st, p);
  count_launches(1);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("gemm_rows launch: %s", cudaGetErrorString(e));
  return 0;
}

template <int MT>
int launch_rows_of(const RowGemmParams& p, int nt, size_t smem, cudaStream_t st) {
  if (p.B2 != nullptr)
    return nt == 2 ? launch_rows<MT, 2, true>(p, smem, st) : launch_rows<MT, 1, true>(p, smem, st);
  if (MT == 1 && nt == 4) return launch_rows<1, 4, false>(p, smem, st);
  return nt == 2 ? launch_rows<MT, 2, false>(p, smem, st) : launch_rows<MT, 1, false>(p, smem, st);
}

}  // namespace
}  // namespace t5x

// 1 when t5x_gemm_rows_bf16 covers the shape. Rows: up to 64, while all of A fits in shared memory.
T5X_API int t5x_gemm_rows_ok(int M, int N, int K, int gated) {
  using namespace t5x;
  return M >= 1 && M <= kRowMaxRows && K >= 16 && K % 16 == 0 && N >= 16 && N % 16 == 0 &&
         rows_smem(M, N, K, gated != 0) <= static_cast<size_t>(kRowMaxSmem);
}

// C[M, N] = alpha * norm(A) @ B (+ R), bf16 or fp32; with B2: gelu(norm(A) @ B) * (norm(A) @ B2).
// A [M, K] bf16 (row stride lda), B / B2 [K, N] bf16 row-major (row stride ldb), norm_scale [K]
// fp32 or null (no norm), R [M, N] bf16 or null.
T5X_API int t5x_gemm_rows_bf16(const void* A, const void* B, const void* B2, void* C, int M, int N,
                               int K, long long lda, long long ldb, long long ldc, int out_fp32,
                               const void* norm_scale, float eps, const void* R, long long ldr,
                               float alpha, void* stream) {
  using namespace t5x;
  if (!t5x_gemm_rows_ok(M, N, K, B2 != nullptr))
    return set_error("gemm_rows: M=%d N=%d K=%d is not covered", M, N, K);
  const uintptr_t ptrs = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) |
                         reinterpret_cast<uintptr_t>(B2) | reinterpret_cast<uintptr_t>(norm_scale);
  if ((ptrs & 15) || lda % 8 || ldb % 8)
    return set_error("gemm_rows: operands must start on 16-byte boundaries, row by row");
  RowGemmParams p = {};
  p.A = static_cast<const __nv_bfloat16*>(A);
  p.B = static_cast<const __nv_bfloat16*>(B);
  p.B2 = static_cast<const __nv_bfloat16*>(B2);
  p.norm_scale = static_cast<const float*>(norm_scale);
  p.R = static_cast<const __nv_bfloat16*>(R);
  p.C = C;
  p.lda = lda; p.ldb = ldb; p.ldc = ldc; p.ldr = ldr;
  p.M = M; p.N = N; p.K = K;
  p.out_fp32 = out_fp32;
  p.eps = eps;
  p.alpha = alpha;
  p.b_constant = chained_launches_constant_b() ? 1 : 0;
  const size_t smem = rows_smem(M, N, K, B2 != nullptr);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int mt = round_up_tiles(M), nt = column_tiles(M, N, B2 != nullptr);
  return mt == 1   ? launch_rows_of<1>(p, nt, smem, st)
         : mt == 2 ? launch_rows_of<2>(p, nt, smem, st)
                   : launch_rows_of<4>(p, nt, smem, st);
}
