// Pieces shared by the one-CTA and the CTA-pair GEMM kernels: problem description, row
// load/store helpers and the epilogue of one accumulator tile.
#pragma once
#include "common.cuh"

namespace t5x {

constexpr int kBM = 128;
constexpr int kBK = 64;
// Epilogue warps of the plain kernels: two per TMEM lane quarter, each taking half of a tile's
// columns. Four warps (one per quarter) need longer for a 128 x 256 tile than the tensor cores
// need for K < ~1500, so that short-K products ran at the epilogue's pace (see the kernels).
constexpr int kEpiWarps = 8;
constexpr int kGemmThreads = 64 + 32 * kEpiWarps;
constexpr int kTpEpiWarps = 4;  // tensor-parallel kernels: one per quarter
constexpr int kKernelIdGemm = 1;
constexpr int kGemmTraceSlots = 8;
long long* gemm_trace_buffer();  // host: the calling thread's trace buffer, or null
#define T5X_GEMM_TRACE(slot)                                                              \
  do {                                                                                    \
    if (p.trace != nullptr && static_cast<int>(blockIdx.x) < p.trace_ctas)                  \
      p.trace[blockIdx.x * kGemmTraceSlots + (slot)] = global_timer_ns();                   \
  } while (0)

constexpr int kCeTileCols = 128;  // columns that one warp folds into one partial

enum GemmEpilogue : int {
  kEpiPlain = 0,
  kEpiGatedGelu = 1,
  kEpiResidual = 2,
  // The product is a logits matrix that is consumed in the epilogue and never stored:
  kEpiCeStats = 3,  // per (row, column tile) softmax partials for the cross-entropy forward
  kEpiCeGrad = 4,   // gradient of the cross-entropy w.r.t. the logits, written as bf16
  // The product is the gradient of gelu(h0) * h1 and never stored either: h0 and h1 (in H0 and H1) become
  // their gradients.
  kEpiGatedGrad = 5,
  // CTA pairs only: ReLU of the product; the product, zero where R is not positive (ReLU's gradient; a NaN in R
  // lets it through, as torch does).
  kEpiRelu = 6,
  kEpiReluGrad = 7,
};

// Several products in one launch, three at most (the projections that share an input).
//   kGroupColumns  C_i = A B_i: the tile columns of the outputs stand side by side, so that a wave
//                  holds tiles of all of them and the rows of A are read once for all.
//   kGroupSum      C = A_0 B_0 + A_1 B_1 + ...: the k blocks follow one another in one accumulator, so
//                  that C is written once, from fp32 sums, instead of read and rounded in between.
enum GemmGroupKind : int { kGroupNone = 0, kGroupColumns = 1, kGroupSum = 2 };
constexpr int kMaxGroup = 3;
template <bool GROUPED>
struct GemmMaps {  // the operands' tensor maps; gated GELU: wi_0 and wi_1 are b[0] and b[1]
  CUtensorMap a[GROUPED ? kMaxGroup : 1];
  CUtensorMap b[GROUPED ? kMaxGroup : 2];
};
struct GemmOut {  // where a tile goes
  void* C;
  long long ldc;
  int N;
};

struct GemmParams {
  int M, N, K, batch;
  int a_mn, b_mn;
  int out_fp32, accumulate;
  void* C;
  long long ldc, c_batch_stride;  // elements
  const __nv_bfloat16* R;         // residual (bf16), same shape as C
  long long ldr, r_batch_stride;
  __nv_bfloat16* H0;  // gated GELU: optional copies of the two pre-activations; its gradient: in and out
  __nv_bfloat16* H1;
  long long ldh, h_batch_stride;
  float alpha;
  int tiles_m, tiles_n;
  int mt_rot;  // the row-tile walk starts at this tile (tensor-parallel kernels); 0 otherwise
  int split_k;     // CTA pairs: pieces that the tiles of the last wave are cut into (see GemmWork)
  // Groups: the first tile column of each output (kGroupColumns) or the first k block of each product
  // (kGroupSum), INT_MAX where there is none; k blocks in all; the outputs.
  int group_at[kMaxGroup];
  int group_num_kb;
  int vec_ok;              // groups: 16-byte accesses are legal in every bf16 output
  GemmOut out[kMaxGroup];  // out[0] is C, ldc, N
  int b_constant;  // B is not written by any kernel in flight: it may be loaded before chain_wait()
  // Optional phase trace (t5x_gemm_set_trace): 8 timestamps per CTA for its first tile: entry,
  // set-up done, first loads issued, first operands landed, last MMA issued, accumulator
  // complete, epilogue done, exit. Null in normal use.
  long long* trace;
  int trace_ctas;  // CTAs that the buffer has room for: one per SM
  int* status;
  // Cross-entropy epilogues. Column c of the product is vocabulary entry ce_vocab_start + c.
  const long long* ce_targets;  // [M] target ids
  int ce_vocab_start;
  int ce_tiles;            // kEpiCeStats: partials per row, one per kCeTileCols columns
  float* ce_part;          // kEpiCeStats: [M, ce_tiles, 4] = max, sum exp(x - max), sum x, largest x
  int* ce_arg;             // kEpiCeStats: [M, ce_tiles] column of the largest x
  float* ce_target_logit;  // kEpiCeStats: [M], written by the tile that holds the target
  const float* ce_lse;     // kEpiCeGrad: [M] log-sum-exp of the row over the whole vocabulary
  const float* ce_row_scale;  // kEpiCeGrad: [M] upstream gradient of the row's loss
  float ce_z, ce_conf, ce_low;  // z-loss factor, label-smoothing confidences
};

// Tensor-parallel extensions of the CTA-pair GEMM. The rows of A (all-gather) or of C
// (reduce-scatter) are split evenly over `world` ranks, `rows_per_rank` consecutive rows each.
//
// Ordering between ranks needs no separate barrier kernel. Every rank owns a small array of
// signal words in memory that all ranks map; word [kind][r] is written only by rank r, with an
// epoch number that grows by one per call (all ranks make the same calls in the same order).
//   kTpSigRowsReady  rank r's own rows of the A buffer are in place (written by the kernel that
//                    precedes the all-gather GEMM on r's stream). Raised by r's all-gather GEMM
//                    as it starts; awaited by the copy warps before they pull from r.
//   kTpSigScattered  every store of rank r's reduce-scatter GEMM into the inboxes has been
//                    performed. Raised by the last CTA of that GEMM; awaited by the kernel that
//                    sums the inbox slots.
// Waits compare epochs by signed distance (wrap-safe), are bounded, and report a status.
enum GemmTpMode : int { kTpNone = 0, kTpAllGather = 1, kTpReduceScatter = 2 };
constexpr int kTpMaxPeers = 16;
constexpr int kTpSigRowsReady = 0;
constexpr int kTpSigScattered = 1;
constexpr int kTpSigWords = 2 * kTpMaxPeers;
constexpr int kTpGroupRows = 128;  // rows of A whose arrival is tracked by one counter
struct GemmTp {
  int world, rank, rows_per_rank;
  // all-gather -> GEMM: A is this rank's [M, K] buffer; block r of it is pulled from
  // a_src[r] (rank r's buffer as mapped here, same layout) by the copy warps while the tensor
  // cores work on blocks that are already here. flags[r * groups_per_block + g] counts the
  // pieces landed in row group g (kTpGroupRows rows) of block r; the last CTA to leave the
  // kernel clears them again.
  const uint8_t* a_src[kTpMaxPeers];
  uint8_t* a_dst;
  long long block_bytes;
  long long group_bytes;
  int groups_per_block;
  unsigned int* flags;
  // GEMM -> reduce-scatter: rows of block r are stored to c_dst[r] ([rows_per_rank, ldc] bf16,
  // this rank's slot of rank r's inbox as mapped here) instead of C.
  __nv_bfloat16* c_dst[kTpMaxPeers];
  // signal words: this rank's own array and the peers' arrays as mapped here; `epoch` is what
  // this call raises and waits for; `exit_count` counts CTAs that have finished (device word).
  unsigned int* sig_local;
  unsigned int* sig_peer[kTpMaxPeers];
  unsigned int epoch;
  unsigned int* exit_count;
};

__device__ __forceinline__ void st_release_sys_u32(unsigned int* addr, unsigned int v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_sys_u32(const unsigned int* addr) {
  unsigned int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(addr) : "memory");
  return v;
}

__device__ __forceinline__ void store_row_bf16(__nv_bfloat16* dst, const float* v, int n_valid,
                                               bool vec_ok) {
  if (vec_ok && n_valid >= 32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      __nv_bfloat162 p0 = __floats2bfloat162_rn(v[i * 8 + 0], v[i * 8 + 1]);
      __nv_bfloat162 p1 = __floats2bfloat162_rn(v[i * 8 + 2], v[i * 8 + 3]);
      __nv_bfloat162 p2 = __floats2bfloat162_rn(v[i * 8 + 4], v[i * 8 + 5]);
      __nv_bfloat162 p3 = __floats2bfloat162_rn(v[i * 8 + 6], v[i * 8 + 7]);
      uint4 u;
      u.x = *reinterpret_cast<uint32_t*>(&p0);
      u.y = *reinterpret_cast<uint32_t*>(&p1);
      u.z = *reinterpret_cast<uint32_t*>(&p2);
      u.w = *reinterpret_cast<uint32_t*>(&p3);
      reinterpret_cast<uint4*>(dst)[i] = u;
    }
  } else {
    // unrolled: an index known only at run time would put the caller's array in local memory
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (i < n_valid) dst[i] = __float2bfloat16(v[i]);
  }
}

__device__ __forceinline__ void load_row_bf16(const __nv_bfloat16* src, float* v, int n_valid,
                                              bool vec_ok) {
  if (vec_ok && n_valid >= 32) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 u = ld_chained(reinterpret_cast<const uint4*>(src) + i);
      const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 f = __bfloat1622float2(p[j]);
        v[i * 8 + j * 2] = f.x;
        v[i * 8 + j * 2 + 1] = f.y;
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = (i < n_valid) ? __bfloat162float(ld_chained(src + i)) : 0.f;
  }
}

// Coalesced epilogue stores. A lane holds 32 consecutive columns of ONE accumulator row, so a
// store straight from registers sends 16-byte pieces of 32 different rows per warp
// instruction: 32 separate 128-byte lines each time, which the load/store unit serialises (a
// 128 x 128 fp32 tile of split-K atomics took 7 us that way). Instead the warp parks its
// 32 x 32 block in shared memory (`stage`: 4 KB of this warp, 16-byte chunks XOR-swizzled by
// row so that neither side has bank conflicts) and writes it out as whole row segments:
// four rows of 128 bytes (fp32) or eight rows of 64 bytes (bf16) per instruction.
constexpr int kEpiStageBytesPerWarp = 32 * 128;

// v: this lane's row (32 floats). out: &C[first row of the warp's block][first column], fp32.
// MODE 0: plain store, 1: add to what is there (one writer per element), 2: atomic add; a
// template argument so that every variant is straight-line code (with the mode as a run-time
// value the atomic variant ran almost four times slower). Rows >= rows_valid are skipped. All
// lanes must call it.
template <int MODE>
__device__ __forceinline__ void staged_store_f32(float* stage, const float (&v)[32], float* out,
                                                 long long ldc, int rows_valid, int lane) {
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<float4*>(stage + lane * 32 + ((c ^ (lane & 7)) * 4)) =
        make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
  __syncwarp();
  const int c = lane & 7;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int row = j * 4 + (lane >> 3);
    const float4 o = *reinterpret_cast<const float4*>(stage + row * 32 + ((c ^ (row & 7)) * 4));
    if (row < rows_valid) {
      float4* dst = reinterpret_cast<float4*>(out + static_cast<long long>(row) * ldc + c * 4);
      if (MODE == 2) {
        atomicAdd(dst, o);
      } else if (MODE == 1) {
        const float4 old = *dst;
        *dst = make_float4(o.x + old.x, o.y + old.y, o.z + old.z, o.w + old.w);
      } else {
        *dst = o;
      }
    }
  }
  __syncwarp();
}

// The same for a bf16 output: the staged block is 32 rows x 64 bytes (the first half of each
// 128-byte staging row), written out as eight 64-byte row segments per instruction.
__device__ __forceinline__ void staged_store_bf16(float* stage, const float (&v)[32],
                                                  __nv_bfloat16* out, long long ldc,
                                                  int rows_valid, int lane) {
  uint4* st4 = reinterpret_cast<uint4*>(stage);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    __nv_bfloat162 p0 = __floats2bfloat162_rn(v[c * 8 + 0], v[c * 8 + 1]);
    __nv_bfloat162 p1 = __floats2bfloat162_rn(v[c * 8 + 2], v[c * 8 + 3]);
    __nv_bfloat162 p2 = __floats2bfloat162_rn(v[c * 8 + 4], v[c * 8 + 5]);
    __nv_bfloat162 p3 = __floats2bfloat162_rn(v[c * 8 + 6], v[c * 8 + 7]);
    uint4 u;
    u.x = *reinterpret_cast<uint32_t*>(&p0);
    u.y = *reinterpret_cast<uint32_t*>(&p1);
    u.z = *reinterpret_cast<uint32_t*>(&p2);
    u.w = *reinterpret_cast<uint32_t*>(&p3);
    // row `lane`, 16-byte chunk c of 4, swizzled over the 8 chunk slots of the 128-byte row
    st4[lane * 8 + ((c ^ (lane & 7)))] = u;
  }
  __syncwarp();
  const int c = lane & 3;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = j * 8 + (lane >> 2);
    const uint4 u = st4[row * 8 + (c ^ (row & 7))];
    if (row < rows_valid)
      *reinterpret_cast<uint4*>(out + static_cast<long long>(row) * ldc + c * 8) = u;
  }
  __syncwarp();
}

// Reads a 32 x 32 bf16 block (rows `ldr` elements apart) into the staging block as 64-byte row
// segments, and adds one row of it to a lane's 32 values. A residual read straight from its row
// by each lane costs 32 separate lines per instruction, as described above.
__device__ __forceinline__ void staged_load_bf16(float* stage, const __nv_bfloat16* src,
                                                 long long ldr, int rows_valid, int lane) {
  uint4* st4 = reinterpret_cast<uint4*>(stage);
  const int c = lane & 3;
  uint4 u[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = j * 8 + (lane >> 2);
    u[j] = make_uint4(0u, 0u, 0u, 0u);
    if (row < rows_valid)
      u[j] = ld_chained(reinterpret_cast<const uint4*>(src + static_cast<long long>(row) * ldr + c * 8));
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = j * 8 + (lane >> 2);
    st4[row * 8 + (c ^ (row & 7))] = u[j];
  }
  __syncwarp();
}

__device__ __forceinline__ void staged_keep_positive(const float* stage, float (&v)[32], int lane) {
  const uint4* st4 = reinterpret_cast<const uint4*>(stage);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint4 u = st4[lane * 8 + (c ^ (lane & 7))];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      v[c * 8 + j * 2] = f.x <= 0.f ? 0.f : v[c * 8 + j * 2];
      v[c * 8 + j * 2 + 1] = f.y <= 0.f ? 0.f : v[c * 8 + j * 2 + 1];
    }
  }
  __syncwarp();  // the block may be overwritten
}

__device__ __forceinline__ void staged_add_row(const float* stage, float (&v)[32], int lane) {
  const uint4* st4 = reinterpret_cast<const uint4*>(stage);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const uint4 u = st4[lane * 8 + (c ^ (lane & 7))];
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      v[c * 8 + j * 2] += f.x;
      v[c * 8 + j * 2 + 1] += f.y;
    }
  }
  __syncwarp();  // the block may be overwritten
}

// Tile order: groups of kRasterGroup row tiles are walked column by column, so that the tiles
// in flight at one time (one per SM or SM pair) share a few A row blocks and a few B column
// blocks instead of one A block and every B block; the operands of a wave then fit in L2.
constexpr int kRasterGroup = 8;
__device__ __forceinline__ void gemm_tile_coords(const GemmParams& p, int tile, int tiles_per_batch,
                                                 int& b, int& mt, int& nt) {
  b = tile / tiles_per_batch;
  const int rem = tile - b * tiles_per_batch;
  const int per_group = kRasterGroup * p.tiles_n;
  const int g = rem / per_group;
  const int first_m = g * kRasterGroup;
  const int gsz = min(kRasterGroup, p.tiles_m - first_m);
  const int r = rem - g * per_group;
  nt = r / gsz;
  mt = first_m + (r - nt * gsz);
  if (p.mt_rot) {
    mt += p.mt_rot;
    if (mt >= p.tiles_m) mt -= p.tiles_m;
  }
}

// Which output (product) tile column (k block) `at` belongs to.
__device__ __forceinline__ int gemm_group_of(const GemmParams& p, int at) {
  return (at >= p.group_at[1] ? 1 : 0) + (at >= p.group_at[2] ? 1 : 0);
}

// The work of a CTA pair, in order: every num_units-th tile, whole, except that with split_k > 1
// the tiles of the last wave, which would leave most of the chip idle (160 tiles on 74 pairs: 2.16
// waves of work in the time of 3), are cut into split_k pieces along K and dealt out piece by
// piece; the pieces of a tile are added to fp32 memory with atomics. Pieces of the same k range
// run at the same time, so they share operands in L2. (Equal shares of all k blocks laid end to
// end balance better, but every pair is then at another k: 2048 x 2048 x 32768 went from 193 to
// 265 us on operand traffic.)
struct GemmWork {
  int at, step, whole, total, tail, splits, num_kb;
  __device__ GemmWork(const GemmParams& p, int unit, int num_units, int total_tiles, int num_kb_)
      : at(unit), step(num_units), whole(total_tiles), total(total_tiles), tail(0), splits(1),
        num_kb(num_kb_) {
    if (p.split_k > 1) {
      tail = total_tiles % num_units;
      whole = total_tiles - tail;
      splits = p.split_k;
      total = whole + tail * splits;
    }
  }
  // Next piece of work: k blocks [kb0, kb1) of `tile`; false when there is none.
  __device__ __forceinline__ bool next(int& tile, int& kb0, int& kb1) {
    if (at >= total) return false;
    if (at < whole) {
      tile = at;
      kb0 = 0;
      kb1 = num_kb;
    } else {
      const int piece = at - whole, s = piece / tail;
      tile = whole + piece - s * tail;
      kb0 = static_cast<int>(static_cast<long long>(num_kb) * s / splits);
      kb1 = static_cast<int>(static_cast<long long>(num_kb) * (s + 1) / splits);
    }
    at += step;
    return true;
  }
};

// Epilogue of one 128-row accumulator tile held in TMEM columns [t_cols, t_cols + BN): the
// calling warp owns lane quarter q (rows m0 + 32q .. +31) and part `part` of PARTS of the tile's
// columns of output `o`, `c_vec_ok` says whether 16-byte accesses to a bf16 C are legal in every batch.
template <int BN, int EPI, int PARTS>
__device__ __forceinline__ void gemm_epilogue_tile(const GemmParams& p, const GemmOut& o, uint32_t t_row, int m0,
                                                   int n0, int b, int q, int part, int lane,
                                                   bool c_vec_ok, int accumulate,
                                                   float* stage = nullptr) {
  const int row = m0 + q * 32 + lane;
  const bool row_ok = row < p.M;
  const int rows_valid = p.M - (m0 + q * 32);  // of this warp's 32 rows (may exceed 32 or be <= 0)

  if (EPI == kEpiGatedGelu) {
    constexpr int kHalf = BN / 2;
    __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(o.C) + b * p.c_batch_stride +
                         static_cast<long long>(row) * o.ldc;
#pragma unroll 1
    for (int c = part * (kHalf / 32 / PARTS); c < (part + 1) * (kHalf / 32 / PARTS); ++c) {
      if (n0 + c * 32 >= o.N) break;  // warp-uniform: columns beyond the output
      uint32_t r0[32], r1[32];
      tmem_ld32(t_row + c * 32, r0);
      tmem_ld32(t_row + kHalf + c * 32, r1);
      tmem_ld_wait();
      const int col = n0 + c * 32;
      const int n_valid = o.N - col;
      const bool hv16 = p.H0 == nullptr ||
                        ((p.ldh % 8 == 0) && (p.h_batch_stride % 8 == 0) &&
                        ((reinterpret_cast<uintptr_t>(p.H0) |
                                               reinterpret_cast<uintptr_t>(p.H1)) & 15) == 0);
      if (stage != nullptr && n_valid >= 32 && rows_valid > 0 && c_vec_ok && hv16) {
        // whole 32-column blocks: row-contiguous stores through the staging block
        float g[32], h0[32], h1[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          h0[i] = __uint_as_float(r0[i]);
          h1[i] = __uint_as_float(r1[i]);
          g[i] = gelu_tanh(h0[i]) * h1[i];
        }
        const long long first_row = m0 + q * 32;
        staged_store_bf16(stage, g,
                          reinterpret_cast<__nv_bfloat16*>(o.C) + b * p.c_batch_stride +
                              first_row * o.ldc + col,
                          o.ldc, rows_valid, lane);
        if (p.H0 != nullptr) {
          const long long at = b * p.h_batch_stride + first_row * p.ldh + col;
          staged_store_bf16(stage, h0, p.H0 + at, p.ldh, rows_valid, lane);
          staged_store_bf16(stage, h1, p.H1 + at, p.ldh, rows_valid, lane);
        }
        continue;
      }
      if (row_ok && n_valid > 0) {
        float g[32], h0[32], h1[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          h0[i] = __uint_as_float(r0[i]);
          h1[i] = __uint_as_float(r1[i]);
          g[i] = gelu_tanh(h0[i]) * h1[i];
        }
        store_row_bf16(out + col, g, n_valid, c_vec_ok);
        if (p.H0 != nullptr) {
          const long long at = b * p.h_batch_stride + static_cast<long long>(row) * p.ldh + col;
          store_row_bf16(p.H0 + at, h0, n_valid, hv16);
          store_row_bf16(p.H1 + at, h1, n_valid, hv16);
        }
      }
    }
  } else {
    const bool f32_vec_ok = o.ldc % 4 == 0 && p.c_batch_stride % 4 == 0 &&
                            (reinterpret_cast<uintptr_t>(o.C) & 15) == 0;
    constexpr bool kReadsR = EPI == kEpiResidual || EPI == kEpiReluGrad;
    const bool r_vec_ok = kReadsR && p.ldr % 8 == 0 && p.r_batch_stride % 8 == 0 &&
                          (reinterpret_cast<uintptr_t>(p.R) & 15) == 0;
#pragma unroll 1
    for (int c = part * (BN / 32 / PARTS); c < (part + 1) * (BN / 32 / PARTS); ++c) {
      const int col = n0 + c * 32;
      const int n_valid = o.N - col;
      if (n_valid <= 0) break;  // warp-uniform: columns beyond the output
      uint32_t r[32];
      tmem_ld32(t_row + c * 32, r);
      // whole 32-column blocks go out through the staging buffer (warp-uniform condition)
      const bool staged = stage != nullptr && n_valid >= 32 && rows_valid > 0 &&
                          (p.out_fp32 ? f32_vec_ok
                                      : (c_vec_ok && (accumulate == 0 || EPI != kEpiResidual)));
      if (staged) {
        if (kReadsR && r_vec_ok)
          staged_load_bf16(stage, p.R + b * p.r_batch_stride +
                                      static_cast<long long>(m0 + q * 32) * p.ldr + col,
                           p.ldr, rows_valid, lane);
        const long long first = b * p.c_batch_stride +
                                static_cast<long long>(m0 + q * 32) * o.ldc + col;
        // bf16 C += : what is there comes in the same way as a residual (65536 x 768 x 768
        // 118 us with 16-byte reads of 32 rows, 94 so)
        const bool add_c = EPI != kEpiResidual && accumulate != 0 && !p.out_fp32;
        if (add_c)
          staged_load_bf16(stage, reinterpret_cast<const __nv_bfloat16*>(o.C) + first, o.ldc,
                           rows_valid, lane);
        tmem_ld_wait();
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * p.alpha;
        if (add_c) staged_add_row(stage, v, lane);
        if (EPI == kEpiRelu) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = v[i] < 0.f ? 0.f : v[i];  // (a NaN stays)
        }
        if (EPI == kEpiReluGrad && r_vec_ok) staged_keep_positive(stage, v, lane);
        if (EPI == kEpiReluGrad && !r_vec_ok && row_ok) {
          float rr[32];
          load_row_bf16(p.R + b * p.r_batch_stride + static_cast<long long>(row) * p.ldr + col, rr, n_valid, false);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = rr[i] <= 0.f ? 0.f : v[i];
        }
        if (EPI == kEpiResidual) {
          if (r_vec_ok) {
            staged_add_row(stage, v, lane);
          } else if (row_ok) {
            float rr[32];
            load_row_bf16(p.R + b * p.r_batch_stride + static_cast<long long>(row) * p.ldr + col,
                          rr, n_valid, false);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += rr[i];
          }
        }
        if (p.out_fp32) {
          float* dst = reinterpret_cast<float*>(o.C) + first;
          if (accumulate == 2)
            staged_store_f32<2>(stage, v, dst, o.ldc, rows_valid, lane);
          else if (accumulate == 1)
            staged_store_f32<1>(stage, v, dst, o.ldc, rows_valid, lane);
          else
            staged_store_f32<0>(stage, v, dst, o.ldc, rows_valid, lane);
        } else
          staged_store_bf16(stage, v, reinterpret_cast<__nv_bfloat16*>(o.C) + first, o.ldc,
                            rows_valid, lane);
        continue;
      }
      tmem_ld_wait();
      if (row_ok) {
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * p.alpha;
        if (EPI == kEpiRelu) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = v[i] < 0.f ? 0.f : v[i];
        }
        if (EPI == kEpiReluGrad) {
          float rr[32];
          load_row_bf16(p.R + b * p.r_batch_stride + static_cast<long long>(row) * p.ldr + col, rr, n_valid,
                        r_vec_ok);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = rr[i] <= 0.f ? 0.f : v[i];
        }
        if (EPI == kEpiResidual) {
          float rr[32];
          load_row_bf16(p.R + b * p.r_batch_stride + static_cast<long long>(row) * p.ldr + col,
                        rr, n_valid, r_vec_ok);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] += rr[i];
        }
        if (p.out_fp32) {
          float* out = reinterpret_cast<float*>(o.C) + b * p.c_batch_stride +
                       static_cast<long long>(row) * o.ldc + col;
          if (f32_vec_ok && n_valid >= 32) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              float4 w = make_float4(v[i * 4], v[i * 4 + 1], v[i * 4 + 2], v[i * 4 + 3]);
              if (accumulate == 2) {  // several CTAs (split K) add into the same tile
                atomicAdd(reinterpret_cast<float4*>(out) + i, w);
                continue;
              }
              if (accumulate) {
                float4 old = reinterpret_cast<float4*>(out)[i];
                w.x += old.x;
                w.y += old.y;
                w.z += old.z;
                w.w += old.w;
              }
              reinterpret_cast<float4*>(out)[i] = w;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              if (i >= n_valid) break;
              if (accumulate == 2)
                atomicAdd(out + i, v[i]);
              else
                out[i] = accumulate ? out[i] + v[i] : v[i];
            }
          }
        } else {
          __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(o.C) + b * p.c_batch_stride +
                               static_cast<long long>(row) * o.ldc + col;
          if (accumulate) {
            float old[32];
            load_row_bf16(out, old, n_valid, c_vec_ok);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += old[i];
          }
          store_row_bf16(out, v, n_valid, c_vec_ok);
        }
      }
    }
  }
}

// Epilogue of the gradient of gelu(h0) * h1 (kEpiGatedGrad): the accumulator holds dg; 32 columns at a time h0 and
// h1 come in, and dg h1 gelu'(h0) and dg gelu(h0) go out in their place, rows 64 bytes at a time through the
// warp's staging block. `GatedRows` holds a block that is on its way: two of them are, across the ends of tiles
// (one of them within a tile: 335 us below; the reads wait for memory, the arithmetic costs nothing).
//
// As a pass of its own this reads dg, h0 and h1 and writes two of them, at the rate of memory; here two fifths of
// that traffic are gone and the rest runs under the MMAs of other tiles (us, product and pass / in one: 65536 x
// 768 x 2048 415 / 324, 14592 x 768 x 2048 101 / 92, 16384 x 4096 x 10240 1380 / 1100, 16384 x 1472 x 3584
// 332 / 250, 3024 x 1472 x 3584 80 / 70). With K = 768 the epilogue is the slower side, by its traffic.
struct GatedRows {
  uint4 h0[4], h1[4];
};
__device__ __forceinline__ void gated_request(const GemmParams& p, int first_row, int col, int rows_valid, int lane,
                                              GatedRows& in) {
  const long long at = static_cast<long long>(first_row + (lane >> 2)) * p.ldh + col + (lane & 3) * 8;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    in.h0[j] = in.h1[j] = make_uint4(0u, 0u, 0u, 0u);
    if (j * 8 + (lane >> 2) < rows_valid) {
      in.h0[j] = ld_chained(reinterpret_cast<const uint4*>(p.H0 + at + j * 8 * p.ldh));
      in.h1[j] = ld_chained(reinterpret_cast<const uint4*>(p.H1 + at + j * 8 * p.ldh));
    }
  }
}
// One block: 32 accumulator columns from t_cols on, columns col.. of the rows from first_row on. `next` requests what
// is to take the place of `in`.
template <typename Next>
__device__ __forceinline__ void gated_block(const GemmParams& p, uint32_t t_cols, int first_row, int col, int lane,
                                            float* stage, GatedRows& in, Next next) {
  const int rows_valid = p.M - first_row;
  uint4* st4 = reinterpret_cast<uint4*>(stage);  // 32 rows of 8 pieces: 0..3 h0, 4..7 h1, exchanged by row
  uint32_t r[32];
  tmem_ld32(t_cols, r);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = j * 8 + (lane >> 2);
    st4[row * 8 + ((lane & 3) ^ (row & 7))] = in.h0[j];
    st4[row * 8 + (((lane & 3) + 4) ^ (row & 7))] = in.h1[j];
  }
  __syncwarp();
  next();
  tmem_ld_wait();
#pragma unroll
  for (int k = 0; k < 4; ++k) {  // eight columns of this lane's row
    uint4& u0 = st4[lane * 8 + (k ^ (lane & 7))];
    uint4& u1 = st4[lane * 8 + ((k + 4) ^ (lane & 7))];
    uint4 a = u0, b = u1;
    __nv_bfloat162* ha = reinterpret_cast<__nv_bfloat162*>(&a);
    __nv_bfloat162* hb = reinterpret_cast<__nv_bfloat162*>(&b);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 x = __bfloat1622float2(ha[e]), y = __bfloat1622float2(hb[e]);
      const float g0 = __uint_as_float(r[k * 8 + e * 2]), g1 = __uint_as_float(r[k * 8 + e * 2 + 1]);
      float v0, v1, d0, d1;
      gelu_tanh_both(x.x, v0, d0);
      gelu_tanh_both(x.y, v1, d1);
      ha[e] = __floats2bfloat162_rn(g0 * y.x * d0, g1 * y.y * d1);
      hb[e] = __floats2bfloat162_rn(g0 * v0, g1 * v1);
    }
    u0 = a;
    u1 = b;
  }
  __syncwarp();
  const long long at = static_cast<long long>(first_row + (lane >> 2)) * p.ldh + col + (lane & 3) * 8;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int row = j * 8 + (lane >> 2);
    if (row < rows_valid) {
      *reinterpret_cast<uint4*>(p.H0 + at + j * 8 * p.ldh) = st4[row * 8 + ((lane & 3) ^ (row & 7))];
      *reinterpret_cast<uint4*>(p.H1 + at + j * 8 * p.ldh) = st4[row * 8 + (((lane & 3) + 4) ^ (row & 7))];
    }
  }
  __syncwarp();  // the block may be overwritten
}

// Cross-entropy forward epilogue of kCeTileCols columns (part `part` of the tile) of an
// accumulator tile: the calling thread owns one row of logits x = alpha * acc and folds them into
// (max, sum exp(x - max), sum x, largest x and its column), which a small kernel merges over the
// partials of a row afterwards. The logits themselves are never stored.
//
// Bound by the instructions per logit: whole 32-column chunks run without bounds checks, the
// column of the maximum comes from one compare-and-select per logit, and the target is looked for
// only in the chunk that holds it.
template <int BN>
__device__ __forceinline__ void gemm_epilogue_ce_stats(const GemmParams& p, uint32_t t_row, int m0,
                                                       int n0, int q, int part, int lane) {
  const int row = m0 + q * 32 + lane;
  const bool row_ok = row < p.M;
  const long long tgt = row_ok ? p.ce_targets[row] - p.ce_vocab_start : -1;
  float mx = -3.0e38f, se = 0.f, sx = 0.f;
  int best_col = 0;
  const int first = n0 + part * kCeTileCols;
  if (first >= p.N) return;  // warp-uniform: no such partial
#pragma unroll 1
  for (int c = 0; c < kCeTileCols / 32; ++c) {
    const int col = first + c * 32;
    const int n_valid = p.N - col;
    if (n_valid <= 0) break;  // warp-uniform
    uint32_t r[32];
    tmem_ld32(t_row + part * kCeTileCols + c * 32, r);
    tmem_ld_wait();
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * p.alpha;
    float s0 = 0.f, s1 = 0.f;
    if (n_valid >= 32) {
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        s0 += v[i];
        s1 += v[i + 1];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        if (i < n_valid) s0 += v[i];
        else v[i] = -INFINITY;  // never the maximum, exp gives zero even where every logit is -inf
      }
    }
    sx += s0 + s1;
    float cm = v[0], cm1 = v[1];
#pragma unroll
    for (int i = 2; i < 32; i += 2) {
      cm = fmaxf(cm, v[i]);
      cm1 = fmaxf(cm1, v[i + 1]);
    }
    cm = fmaxf(cm, cm1);
    int ci = 0;
#pragma unroll
    for (int i = 31; i >= 0; --i) ci = v[i] == cm ? i : ci;
    if (cm > mx) best_col = col + ci;
    const long long off = tgt - col;
    if (off >= 0 && off < 32 && off < n_valid) {
      float t = v[0];
#pragma unroll
      for (int i = 1; i < 32; ++i) t = off == i ? v[i] : t;
      p.ce_target_logit[row] = t;
    }
    const float nm = fmaxf(mx, cm);
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      a0 += __expf(v[i] - nm);
      a1 += __expf(v[i + 1] - nm);
    }
    se = se * __expf(mx - nm) + (a0 + a1);
    mx = nm;
  }
  if (row_ok) {
    const long long at = static_cast<long long>(row) * p.ce_tiles + first / kCeTileCols;
    reinterpret_cast<float4*>(p.ce_part)[at] = make_float4(mx, se, sx, mx);
    p.ce_arg[at] = best_col + p.ce_vocab_start;
  }
}

// Cross-entropy backward epilogue: the logits tile is recomputed by the GEMM and turned into
//   dlogits = row_scale * ((1 + 2 z lse) * exp(x - lse) - soft_target)        (bf16)
// which the two gradient GEMMs of the projection read next. C is the bf16 [M, N] output; whole
// chunks leave through the warp's staging block as 64-byte row segments.
template <int BN, int PARTS>
__device__ __forceinline__ void gemm_epilogue_ce_grad(const GemmParams& p, uint32_t t_row, int m0,
                                                      int n0, int q, int part, int lane,
                                                      bool c_vec_ok, float* stage) {
  const int row = m0 + q * 32 + lane;
  const bool row_ok = row < p.M;
  const int rows_valid = p.M - (m0 + q * 32);
  const float lse = row_ok ? p.ce_lse[row] : 0.f;
  const float g = row_ok ? p.ce_row_scale[row] : 0.f;
  const float zf = 1.f + 2.f * p.ce_z * lse;
  const long long tgt = row_ok ? p.ce_targets[row] - p.ce_vocab_start : -1;
  __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.C);
#pragma unroll 1
  for (int c = part * (BN / 32 / PARTS); c < (part + 1) * (BN / 32 / PARTS); ++c) {
    const int col = n0 + c * 32;
    const int n_valid = p.N - col;
    if (n_valid <= 0) break;  // warp-uniform
    uint32_t r[32];
    tmem_ld32(t_row + c * 32, r);
    tmem_ld_wait();
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i)
      v[i] = g * (zf * __expf(__uint_as_float(r[i]) * p.alpha - lse) - p.ce_low);
    const long long off = tgt - col;
    if (off >= 0 && off < 32) {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (off == i)
          v[i] = g * (zf * __expf(__uint_as_float(r[i]) * p.alpha - lse) - p.ce_conf);
    }
    if (g == 0.f) {  // a token without weight: exactly zero, whatever its logits are
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = 0.f;
    }
    if (n_valid >= 32 && c_vec_ok && rows_valid > 0)
      staged_store_bf16(stage, v, out + static_cast<long long>(m0 + q * 32) * p.ldc + col, p.ldc,
                        rows_valid, lane);
    else if (row_ok)
      store_row_bf16(out + static_cast<long long>(row) * p.ldc + col, v, n_valid, c_vec_ok);
  }
}

// Reduce-scatter epilogue of one 128-row accumulator tile: each row of the bf16 partial product
// (+ local residual) goes to the inbox of the rank that owns the row, mostly peer memory. A
// lane holds one row of the accumulator, so storing straight from registers would send 16-byte
// pieces of 32 different rows per instruction; over NVLink that is one small packet each.
// Instead 128 columns at a time are staged in shared memory (`stage`: 8 KB of this warp, 16-byte
// chunks XOR-swizzled by row so that neither side has bank conflicts) and written out as
// 256-byte row segments, two rows per warp instruction. Requires N % 8 == 0 and ldc % 8 == 0.
constexpr int kRsGroupCols = 128;
constexpr int kRsStageBytesPerWarp = 32 * kRsGroupCols * 2;
template <int BN, int EPI>
__device__ __forceinline__ void gemm_epilogue_tile_rs(const GemmParams& p, const GemmTp& tp,
                                                      uint32_t t_row, int m0, int n0, int q,
                                                      int lane, uint8_t* stage) {
  const int row = m0 + q * 32 + lane;
  const bool row_ok = row < p.M;
#pragma unroll 1
  for (int g = 0; g < BN / kRsGroupCols; ++g) {
    const int gcol = n0 + g * kRsGroupCols;
#pragma unroll 1
    for (int c = 0; c < kRsGroupCols / 32; ++c) {
      uint32_t r[32];
      tmem_ld32(t_row + g * kRsGroupCols + c * 32, r);
      tmem_ld_wait();
      const int col = gcol + c * 32;
      const int n_valid = p.N - col;
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) * p.alpha;
      if (EPI == kEpiResidual && row_ok && n_valid > 0) {
        float rr[32];
        const bool rv = (p.ldr % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.R) & 15) == 0);
        load_row_bf16(p.R + static_cast<long long>(row) * p.ldr + col, rr, n_valid, rv);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] += rr[i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {  // four 16-byte chunks of this lane's row
        __nv_bfloat162 p0 = __floats2bfloat162_rn(v[i * 8 + 0], v[i * 8 + 1]);
        __nv_bfloat162 p1 = __floats2bfloat162_rn(v[i * 8 + 2], v[i * 8 + 3]);
        __nv_bfloat162 p2 = __floats2bfloat162_rn(v[i * 8 + 4], v[i * 8 + 5]);
        __nv_bfloat162 p3 = __floats2bfloat162_rn(v[i * 8 + 6], v[i * 8 + 7]);
        uint4 u;
        u.x = *reinterpret_cast<uint32_t*>(&p0);
        u.y = *reinterpret_cast<uint32_t*>(&p1);
        u.z = *reinterpret_cast<uint32_t*>(&p2);
        u.w = *reinterpret_cast<uint32_t*>(&p3);
        const int chunk = (c * 4 + i) ^ (lane & 15);
        *reinterpret_cast<uint4*>(stage + lane * (kRsGroupCols * 2) + chunk * 16) = u;
      }
    }
    __syncwarp();
    // 16 instructions, each: lanes 0-15 one row, lanes 16-31 the next, 16 bytes per lane
    const int chunk = lane & 15;
    const int ccol = gcol + chunk * 8;
#pragma unroll 4
    for (int it = 0; it < 16; ++it) {
      const int rloc = it * 2 + (lane >> 4);
      const int grow = m0 + q * 32 + rloc;
      if (grow < p.M && ccol < p.N) {
        const uint4 u = *reinterpret_cast<const uint4*>(stage + rloc * (kRsGroupCols * 2) +
                                                        ((chunk ^ (rloc & 15)) * 16));
        const int owner = grow / tp.rows_per_rank;
        __nv_bfloat16* dst = tp.c_dst[owner] +
                             static_cast<long long>(grow - owner * tp.rows_per_rank) * p.ldc + ccol;
        *reinterpret_cast<uint4*>(dst) = u;
      }
    }
    __syncwarp();
  }
}

}  // namespace t5x
