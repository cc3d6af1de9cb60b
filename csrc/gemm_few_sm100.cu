// bf16 GEMM for a handful of rows (a decode step of a few sentences):
//
//   C[M, N] = A[M, K] * B (+ R),  M <= 64;  B: row-major [K, N]; up to three weights side by side, or
//   gated GELU of two.
//
// What bounds it: nothing but latencies. A step of a decoder layer is a chain of some ten kernels of
// a few microseconds, each of which waits for the one before it; the weights of a product are
// 1 to 20 MB and stream in while it waits (programmatic dependent launches). What counts is the time
// from the last kernel's end to this one's: fetch the rows, multiply, add up the K slices, store.
// So, against the kernels for more rows (gemm_sm100.cu, gemm_skinny_sm100.cu):
//   * tiles of 64 columns (gated: 64 of each weight), so that 2304 columns are 36 CTAs and not 18, and
//     the ring holds most of the K range of a 768-wide product: the tile's weights are requested
//     before the rows exist;
//   * only the M rows are fetched and exchanged, not the 128 of the MMA: the rows of the tile beyond
//     them are whatever the shared memory holds, and end in accumulator rows that nobody reads;
//   * the K slices of a cluster meet by st.async of the few valid rows from registers to the CTA that
//     owns them, without parking a tile in shared memory first;
//   * 112 KB of shared memory at most, so that the next kernel's CTAs fit beside this one's.
// The six products of a layer with three norms between them, four rows, cold weights, chained, us a
// layer, kernels for more rows / these: 512 wide 36.7 / 26.6, 768 45.3 / 30.4, 1024 51.2 / 34.8, 2048
// 79.8 / 50.1; 64 rows of 768 46.7 / 39.1. What is left of a product: 1.8 us from kernel to kernel,
// 0.2 us per 64 of K, 0.6 to 0.8 for the exchange.
//
// The sums are those of the other kernels bit by bit, so that a sentence decodes alike alone and in a
// large batch: the same 128-row MMAs over 64-deep k blocks in order, the same K slices, and the parts
// of a cluster added own part first, then by rank, where the owner of row r is rank r / (128 / S) as
// in gemm_skinny_sm100.cu. (The norm in front as part of this kernel, every CTA computing the normed
// rows for itself, was as fast up to eight rows and slower above: its launch is hidden, the work is
// not.)
#include <algorithm>

#include "gemm_common.cuh"

namespace t5x {
namespace {

constexpr int kFewEpiWarps = 8;
constexpr int kFewThreads = 64 + kFewEpiWarps * 32;
constexpr int kFewMaxRows = 64;
constexpr int kFewMaxStages = 16;
constexpr int kFewBarBytes = 512;
// Two CTAs per SM, so that the next kernel's fit beside this one's while it waits.
constexpr int kFewSmemBudget = 112 * 1024;
constexpr int kFewStageSlots = kFewMaxRows / 32 * 2;  // epilogue warps that hold valid rows
constexpr int kKernelIdGemmFew = 8;

struct FewMaps {
  CUtensorMap a, b[3];
};

struct FewParams {
  int M, N, K;         // N: columns of each weight (gated), of all weights together (else)
  int rows;            // M rounded up to 8: rows of an A block in shared memory
  int split_at[2];     // first column of the second and third weight
  int splits, num_kb;  // cluster size and 64-deep k blocks per CTA
  int slot_rows;       // rows of a part: at most 128 / splits of them meet in one CTA
  int stages;          // of the operand ring
  __nv_bfloat16* C;
  long long ldc;
  const __nv_bfloat16* R;
  long long ldr;
  int b_constant;
  int* status;
};

// 16 bytes to another CTA's shared memory, counted on an mbarrier there.
__device__ __forceinline__ void st_async_v4(uint32_t dst_cluster_addr, const uint32_t* v,
                                            uint32_t bar_cluster_addr) {
  asm volatile(
      "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
      :
      : "r"(dst_cluster_addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar_cluster_addr)
      : "memory");
}
__device__ __forceinline__ void few_epilogue_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kFewEpiWarps * 32) : "memory");
}

template <int EPI>
__global__ void __launch_bounds__(kFewThreads, 2)
    gemm_few_kernel(const __grid_constant__ FewMaps maps, const __grid_constant__ FewParams p) {
  constexpr bool kGated = EPI == kEpiGatedGelu;
  constexpr int BN = kGated ? 128 : 64;
  constexpr int kBBytes = BN * kBK * 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  const int a_bytes = p.rows * 128;
  // A, then B: an MMA reads 16 KB from the start of an A block, the rows beyond it from what follows
  uint8_t* sA = smem;
  uint8_t* sB = smem + p.stages * a_bytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sB + p.stages * kBBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + kFewMaxStages;
  uint64_t* tmem_full = bars + 2 * kFewMaxStages;
  uint64_t* recv_bar = tmem_full + 1;  // counts the bytes of the peers' rows
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // behind the barriers: [S][slot_rows][64] parts of this CTA's rows (clusters), or the warps'
  // staging blocks for whole tiles
  uint8_t* extra = reinterpret_cast<uint8_t*>(bars) + kFewBarBytes;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int S = p.splits;
  const int rank = S > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = blockIdx.x / S;
  const int n0 = tile * 64;
  const int num_kb = p.num_kb;
  const int kb0 = rank * num_kb;
  const int rows_per = kBM / S;                       // accumulator rows that a rank owns
  const int own = min(max(p.M - rank * rows_per, 0), rows_per);  // of them in use

  chain_release();
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tmem_full, 1);
    mbar_init(recv_bar, 1);
    *abort_flag = 0;
    mbar_fence_init();
    if (S > 1 && own > 0) mbar_expect_tx(recv_bar, static_cast<uint32_t>((S - 1) * own * 64 * 4));
    tma_prefetch_desc(&maps.a);
    tma_prefetch_desc(&maps.b[0]);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  // (peers signal this CTA's barriers only after their half of this barrier has completed)
  if (S > 1) cluster_arrive();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      int g = 0, col = n0;  // the weight that holds this tile's columns
      if (!kGated) {
        g = (n0 >= p.split_at[0] ? 1 : 0) + (n0 >= p.split_at[1] ? 1 : 0);
        col = g == 0 ? n0 : n0 - p.split_at[g - 1];
      }
      const CUtensorMap* tb = &maps.b[g];
      auto load_a = [&](int stage, int kb) {
        tma_load_3d(sA + stage * a_bytes, &maps.a, &full[stage], (kb0 + kb) * kBK, 0, 0);
      };
      auto load_b = [&](int stage, int kb) {
        uint8_t* dst = sB + stage * kBBytes;
        const int k0 = (kb0 + kb) * kBK;
        tma_load_3d(dst, tb, &full[stage], col, k0, 0);
        if (kGated) tma_load_3d(dst + 8192, &maps.b[1], &full[stage], col, k0, 0);
      };
      const uint32_t bytes = kBBytes + a_bytes;
      const int first = min(p.stages, num_kb);
      if (!p.b_constant) chain_wait();
      for (int kb = 0; kb < first; ++kb) {
        mbar_expect_tx(&full[kb], bytes);
        load_b(kb, kb);
      }
      // constant weights are requested before the wait for the preceding kernel, the rows after it
      if (p.b_constant) chain_wait();
      for (int kb = 0; kb < first; ++kb) load_a(kb, kb);
      int stage = first == p.stages ? 0 : first;
      uint32_t phase = first == p.stages ? 1 : 0;
      for (int kb = first; kb < num_kb; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag)) {
          report_status(p.status, kStatusTimeoutProducer, kKernelIdGemmFew, tile, kb);
          *abort_flag = 1;
          break;
        }
        mbar_expect_tx(&full[stage], bytes);
        load_a(stage, kb);
        load_b(stage, kb);
        if (++stage == p.stages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    // The whole warp walks the k blocks and one lane issues: with everything uniform the descriptors
    // stay in uniform registers and one addition apart. (An MMA of 64 columns takes less time than
    // building its descriptors in a branch of one lane did: 768 x 768 in one slice, chained, 5.8 us
    // so, 4.1 now.)
    const uint32_t idesc = make_idesc_bf16(kBM, BN, 0, 1);
    const uint64_t a_desc = make_smem_desc_sw128(smem_u32(sA), 16u, 1024);
    const uint64_t b_desc = make_smem_desc_sw128(smem_u32(sB), 8192u, 1024);
    const bool leader = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int kb = 0; kb < num_kb; ++kb) {
      ok = mbar_wait(&full[stage], phase, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const uint64_t ad = a_desc + static_cast<uint32_t>(stage * (a_bytes >> 4));
      const uint64_t bd = b_desc + static_cast<uint32_t>(stage * (kBBytes >> 4));
      if (leader) {
#pragma unroll
        for (int s = 0; s < kBK / 16; ++s)
          umma_bf16(tmem_base, ad + 2 * s, bd + 128 * s, idesc, (kb | s) != 0 ? 1u : 0u);
        umma_commit(&empty[stage]);
      }
      if (++stage == p.stages) {
        stage = 0;
        phase ^= 1;
      }
    }
    ok = __all_sync(0xffffffffu, ok);
    if (ok) {
      if (leader) umma_commit(tmem_full);
    } else {
      if (lane == 0) report_status(p.status, kStatusTimeoutMma, kKernelIdGemmFew, tile, 0);
      *abort_flag = 1;
    }
  }
  __syncwarp();

  const bool acc_ok = mbar_wait(tmem_full, 0, abort_flag);
  if (!acc_ok && threadIdx.x == 64)
    report_status(p.status, kStatusTimeoutEpilogue, kKernelIdGemmFew, tile, 0);
  if (!acc_ok) *abort_flag = 1;
  tc_fence_after();
  chain_wait();  // the residual read and the stores to C come after this
  __syncwarp();
  if (S > 1) cluster_wait();

  const int q = warp & 3, half = (warp - 2) >> 2;
  const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
  if (S > 1) {
    float* parts = reinterpret_cast<float*>(extra);
    const int t = threadIdx.x - 64;  // epilogue threads: 0..255
    if (warp >= 2 && acc_ok && q * 32 < p.M) {
      // each valid row goes to the rank that owns it: this CTA's own rows into its own slot, the
      // others over the cluster
      const int row = q * 32 + lane;
      uint32_t r[32];
      tmem_ld32(t_row + half * 32, r);
      tmem_ld_wait();
      if (row < p.M) {
        const int to = row / rows_per;
        const uint32_t at = static_cast<uint32_t>(
            ((rank * p.slot_rows + row - to * rows_per) * 64 + half * 32) * 4);
        if (to == rank) {
          uint4* dst = reinterpret_cast<uint4*>(extra + at);
#pragma unroll
          for (int i = 0; i < 8; ++i) dst[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
        } else {
          const uint32_t dst = mapa_shared(smem_u32(extra) + at, to);
          const uint32_t bar = mapa_shared(smem_u32(recv_bar), to);
#pragma unroll
          for (int i = 0; i < 8; ++i) st_async_v4(dst + 16 * i, r + 4 * i, bar);
        }
      }
    }
    if (warp >= 2 && own > 0) {
      // columns 4 c .. 4 c + 3 of row t / 16, t / 16 + 16, ..; at most four rows a thread
      const int c = t & 15;
      uint2 res[4];
#pragma unroll
      for (int it = 0; it < 4; ++it) {
        const int lrow = (t >> 4) + 16 * it;
        res[it] = make_uint2(0u, 0u);
        if (p.R != nullptr && lrow < own)
          res[it] = ld_chained(reinterpret_cast<const uint2*>(
              p.R + static_cast<long long>(rank * rows_per + lrow) * p.ldr + n0 + c * 4));
      }
      few_epilogue_sync();  // this CTA's own part is in place
      const bool got = mbar_wait(recv_bar, 0, abort_flag);
      if (!got) {
        if (threadIdx.x == 64)
          report_status(p.status, kStatusTimeoutPeerFlag, kKernelIdGemmFew, tile, rank);
        *abort_flag = 1;
      }
      if (got && acc_ok) {
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const int lrow = (t >> 4) + 16 * it;
          if (lrow >= own) break;
          auto part_of = [&](int s) {
            return *reinterpret_cast<const float4*>(parts + (s * p.slot_rows + lrow) * 64 + c * 4);
          };
          float4 acc = part_of(rank);
          for (int s = 0; s < S; ++s)
            if (s != rank) {
              const float4 o = part_of(s);
              acc.x += o.x, acc.y += o.y;
              acc.z += o.z, acc.w += o.w;
            }
          float o[4] = {acc.x, acc.y, acc.z, acc.w};
          if (p.R != nullptr) {
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&res[it].x));
            const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&res[it].y));
            o[0] += a.x, o[1] += a.y, o[2] += b.x, o[3] += b.y;
          }
          const __nv_bfloat162 lo = __floats2bfloat162_rn(o[0], o[1]);
          const __nv_bfloat162 hi = __floats2bfloat162_rn(o[2], o[3]);
          uint2 u;
          u.x = *reinterpret_cast<const uint32_t*>(&lo);
          u.y = *reinterpret_cast<const uint32_t*>(&hi);
          *reinterpret_cast<uint2*>(p.C + static_cast<long long>(rank * rows_per + lrow) * p.ldc + n0 +
                                    c * 4) = u;
        }
      }
    }
    __syncwarp();
    // nobody leaves while rows may still be on their way into its shared memory
    cluster_arrive();
    cluster_wait();
  } else if (warp >= 2 && acc_ok && q * 32 < p.M) {
    GemmParams gp;
    gp.M = p.M, gp.N = p.N, gp.K = p.K, gp.batch = 1;
    gp.out_fp32 = 0, gp.accumulate = 0;
    gp.C = p.C, gp.ldc = p.ldc, gp.c_batch_stride = 0;
    gp.R = p.R, gp.ldr = p.ldr, gp.r_batch_stride = 0;
    gp.H0 = gp.H1 = nullptr, gp.ldh = 0, gp.h_batch_stride = 0;
    gp.alpha = 1.f;
    const GemmOut out = {p.C, p.ldc, p.N};
    float* stage = reinterpret_cast<float*>(extra + (half * 2 + q) * kEpiStageBytesPerWarp);
    const bool c_vec16 = (p.ldc % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0);
    if (kGated)
      gemm_epilogue_tile<BN, kEpiGatedGelu, 2>(gp, out, t_row, 0, n0, 0, q, half, lane, c_vec16, 0, stage);
    else if (p.R != nullptr)
      gemm_epilogue_tile<BN, kEpiResidual, 2>(gp, out, t_row, 0, n0, 0, q, half, lane, c_vec16, 0, stage);
    else
      gemm_epilogue_tile<BN, kEpiPlain, 2>(gp, out, t_row, 0, n0, 0, q, half, lane, c_vec16, 0, stage);
  }

  // Teardown: loads still in flight after an abort get a bounded time to land.
  __syncwarp();
  if (*abort_flag && warp == 0 && lane == 0) {
    for (int it = 0; it < 2000; ++it) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
}

bool few_map(CUtensorMap* out, const void* ptr, long long inner, long long outer, long long ld,
             uint32_t box_outer) {
  uint64_t dims[3] = {static_cast<uint64_t>(inner), static_cast<uint64_t>(outer), 1};
  uint64_t strides[2] = {static_cast<uint64_t>(ld) * 2, static_cast<uint64_t>(ld) * 2 * outer};
  uint32_t box[3] = {64, box_outer, 1};
  return get_tensor_map(out, ptr, 2, 3, dims, strides, box, 1);
}

template <int EPI>
int launch_few(const FewMaps& maps, FewParams& p, cudaStream_t st) {
  constexpr int kBBytes = (EPI == kEpiGatedGelu ? 128 : 64) * kBK * 2;
  const int a_bytes = p.rows * 128;
  const int extra = p.splits > 1 ? p.splits * p.slot_rows * 64 * 4 : kFewStageSlots * kEpiStageBytesPerWarp;
  const int fixed = 1024 + kFewBarBytes + extra;
  // as many stages as the budget holds, the whole K range if it does
  const int stages = std::min((kFewSmemBudget - fixed) / (kBBytes + a_bytes), kFewMaxStages);
  p.stages = std::max(std::min(stages, p.num_kb), 1);
  // (the MMA of the last A block reads 16 KB from its start)
  const int smem = std::max(fixed + p.stages * (kBBytes + a_bytes),
                            1024 + (p.stages - 1) * a_bytes + kBM * 128);
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(gemm_few_kernel<EPI>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, kFewSmemBudget);
    if (e != cudaSuccess) return set_error("cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    attr_set[dev & 63] = true;
  }
  if (smem > kFewSmemBudget) return set_error("gemm_few: %d bytes of shared memory", smem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.N / 64 * p.splits);
  cfg.blockDim = dim3(kFewThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (p.splits > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = p.splits;
    attr[n].val.clusterDim.y = 1;
    attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (chained_launches()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_few_kernel<EPI>, maps, p);
  count_launches(1);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("gemm_few launch: %s", cudaGetErrorString(e));
  return 0;
}

}  // namespace
}  // namespace t5x

// Whether t5x_gemm_few_bf16 covers M rows x K features against `n` weights of `width` columns (gated: a
// pair of `width`), with K cut into `splits` slices.
T5X_API int t5x_gemm_few_covers(int M, int K, int n, int width, int splits, int gated) {
  using namespace t5x;
  if (M < 1 || M > kFewMaxRows || K < 64 || K % 64 || width < 64 || width % 64) return 0;
  if (splits != 1 && splits != 2 && splits != 4 && splits != 8) return 0;
  if ((K / 64) % splits || n < 1 || n > 3) return 0;
  return !gated || (n == 2 && splits == 1);
}

// C[M, n * width] (bf16, row stride ldc) = A[M, K] * [B_0 | B_1 | B_2] (+ R), M <= 64, B_i row-major
// [K, width] with row stride ldb. gated: C[M, width] = gelu(A B_0) * (A B_1). splits: K slices over a
// cluster, summed as by t5x_gemm_skinny_bf16; 1: summed as by t5x_gemm_bf16. Pointers 16-byte
// aligned, strides multiples of 8 elements (R: 8 bytes, 4 elements).
T5X_API int t5x_gemm_few_bf16(const void* A, const void* const* B, void* C, const void* R, int M, int K,
                              int n, int width, long long lda, long long ldb, long long ldc,
                              long long ldr, int splits, int gated, void* stream) {
  using namespace t5x;
  if (!t5x_gemm_few_covers(M, K, n, width, splits, gated))
    return set_error("gemm_few: %d rows x %d, %d x %d columns, %d slices are not covered", M, K, n, width,
                     splits);
  if (lda % 8 || ldb % 8 || ldc % 8 || (R != nullptr && ldr % 4) || lda < K || ldb < width)
    return set_error("gemm_few: leading dimensions");
  if (((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(C)) & 15) ||
      (reinterpret_cast<uintptr_t>(R) & 7))
    return set_error("gemm_few: misaligned pointer");
  if (R != nullptr && gated) return set_error("gemm_few: no residual with a gate");
  FewParams p = {};
  p.M = M;
  p.K = K;
  p.N = gated ? width : n * width;
  p.rows = (M + 7) / 8 * 8;
  p.split_at[0] = width;
  p.split_at[1] = 2 * width;
  p.splits = splits;
  p.num_kb = K / kBK / splits;
  p.slot_rows = std::min(p.rows, kBM / splits);
  p.C = static_cast<__nv_bfloat16*>(C);
  p.ldc = ldc;
  p.R = static_cast<const __nv_bfloat16*>(R);
  p.ldr = ldr;
  p.b_constant = chained_launches_constant_b() ? 1 : 0;
  p.status = device_status_buffer();
  FewMaps maps;
  if (!few_map(&maps.a, A, K, M, lda, p.rows)) return -1;
  for (int i = 0; i < 3; ++i)
    if (!few_map(&maps.b[i], B[i < n ? i : 0], width, K, ldb, 64)) return -1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return gated ? launch_few<kEpiGatedGelu>(maps, p, st) : launch_few<kEpiPlain>(maps, p, st);
}
