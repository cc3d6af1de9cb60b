// Flash attention forward on sm_100a for few heads of 64 channels: softmax(Q K^T + bias(k - q) + mask) V, bias and
// masks as in attention_common.cuh (hidden scores take the value -1e10; no 1/sqrt(d) scaling).
//
// One CTA per head and example of 16 softmax warps, four threads a row: K and V stay in shared memory while the
// CTA walks the 128-query blocks; S = Q K^T for the whole key range sits in TMEM (up to 512 keys), and the score
// MMAs of the next query block are issued as soon as the softmax warps release the columns.
//
// What bounds it is the chain of steps of one query block. attention_fwd_rows_sm100.cu hides the chains of four
// groups of warps behind one another, which takes heads enough for two CTAs per SM; where the SMs are not filled,
// sixteen warps on one block are through sooner (`forward_kernel` in t5x_b200/ops/attention.py has the figures). The exact maximum
// comes first and the sums are taken in the same order, so that results are those of that kernel bit for bit.
#include "attention_common.cuh"
#include "t5x_ops.h"

namespace t5x {
namespace {

struct FewSmem {
  static constexpr int kTile = 128 * 128;  // bytes of a [128 x 64] bf16 tile
  static constexpr int kQ = 0;
  static constexpr int kK = kTile;              // up to 4 tiles
  static constexpr int kV = kK + 4 * kTile;     // up to 4 tiles
  static constexpr int kP = kV + 4 * kTile;     // 2 buffers x 2 tiles
  static constexpr int kRel = kP + 4 * kTile;   // bias by (k - q): up to 512 + 512 floats
  static constexpr int kStat = kRel + 1024 * 4; // 128 x 4 floats (row max parts), then sums
  static constexpr int kKeySeg = kStat + 128 * 4 * 4 * 2;  // 512 ints: segment id of key k
  static constexpr int kKeyWord = kKeySeg + 512 * 4;  // 16 words: bit x of word w, key 32 w + x is visible
  static constexpr int kBars = kKeyWord + 16 * 4;
  static constexpr int kTotal = kBars + 256 + 1024;
};
constexpr int kFewMax = 512;  // queries and keys: sRel covers (k - q) for that many

__global__ void __launch_bounds__(kAttnThreads, 1)
    attn_fwd_few_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sQ = smem + FewSmem::kQ;
  uint8_t* sK = smem + FewSmem::kK;
  uint8_t* sV = smem + FewSmem::kV;
  uint8_t* sP = smem + FewSmem::kP;
  float* sRel = reinterpret_cast<float*>(smem + FewSmem::kRel);
  float* sStat = reinterpret_cast<float*>(smem + FewSmem::kStat);
  int* sKeySeg = reinterpret_cast<int*>(smem + FewSmem::kKeySeg);
  uint32_t* sKeyWord = reinterpret_cast<uint32_t*>(smem + FewSmem::kKeyWord);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FewSmem::kBars);
  uint64_t* bar_q = bars;           // Q tile landed (once per query block)
  uint64_t* bar_kv = bars + 1;      // 4: K_j and V_j landed (once per CTA)
  uint64_t* bar_s = bars + 5;       // 4: S block j ready in TMEM (once per query block)
  uint64_t* bar_p = bars + 9;       // 4: P block j written to smem, S block j released
  uint64_t* bar_pv = bars + 13;     // 4: PV MMA of block j finished (P buffer reusable)
  uint64_t* bar_qfree = bars + 17;  // all S MMAs of this query block done: Q smem reusable
  uint64_t* bar_oread = bars + 18;  // O accumulator of this query block has been read out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, b = blockIdx.y;
  const int nblk = (p.Lk + 127) / 128;
  const int nq = (p.Lq + 127) / 128;
  const int lq_pad = nq * 128;
  const int o_col = (nblk * 128) & 511;  // TMEM column of O (reuses S block 0 when Lk fills TMEM)

  if (threadIdx.x == 0) {
    mbar_init(bar_q, 1);
    mbar_init(bar_qfree, 1);
    mbar_init(bar_oread, kSoftmaxWarps);
    for (int j = 0; j < 4; ++j) {
      mbar_init(&bar_kv[j], 1);
      mbar_init(&bar_s[j], 1);
      mbar_init(&bar_p[j], kSoftmaxWarps);
      mbar_init(&bar_pv[j], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kCtrlWarp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == kCtrlWarp) {
    if (lane == 0) {
      bool ok = true;
      mbar_expect_tx(bar_q, FewSmem::kTile);
      tma_load_4d(sQ, &tmQ, bar_q, 0, h, 0, b);
      for (int j = 0; j < nblk; ++j) {
        mbar_expect_tx(&bar_kv[j], 2 * FewSmem::kTile);
        tma_load_4d(sK + j * FewSmem::kTile, &tmK, &bar_kv[j], 0, h, j * 128, b);
        tma_load_4d(sV + j * FewSmem::kTile, &tmV, &bar_kv[j], 0, h, j * 128, b);
      }
      const uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
      const uint32_t idesc_o = make_idesc_bf16(128, 64, 0, 1);
      const uint32_t qa = smem_u32(sQ);
      for (int i = 0; i < nq && ok; ++i) {
        const uint32_t ph = i & 1;
        // ---- S_j = Q_i K_j^T, as soon as the previous query block released the columns ----
        ok = mbar_wait(bar_q, ph, abort_flag);
        for (int j = 0; j < nblk && ok; ++j) {
          if (i == 0) ok = mbar_wait(&bar_kv[j], 0, abort_flag);
          if (ok && i > 0) {
            ok = mbar_wait(&bar_p[j], ph ^ 1, abort_flag);
            // the O accumulator of the previous block may live in S block 0's columns
            if (ok && j * 128 == o_col) ok = mbar_wait(bar_oread, ph ^ 1, abort_flag);
          }
          if (!ok) break;
          tc_fence_after();
          const uint32_t ka = smem_u32(sK + j * FewSmem::kTile);
#pragma unroll
          for (int s = 0; s < 4; ++s)
            umma_bf16(tmem_base + j * 128, make_smem_desc_sw128(qa + s * 32, 16, 1024),
                      make_smem_desc_sw128(ka + s * 32, 16, 1024), idesc_s, s != 0);
          umma_commit(&bar_s[j]);
        }
        if (!ok) break;
        // Q smem is free once the S MMAs are done: prefetch the next query block.
        if (i + 1 < nq) {
          umma_commit(bar_qfree);
          ok = mbar_wait(bar_qfree, ph, abort_flag);
          if (!ok) break;
          mbar_expect_tx(bar_q, FewSmem::kTile);
          tma_load_4d(sQ, &tmQ, bar_q, 0, h, (i + 1) * 128, b);
        }
        // ---- O_i += P_j V_j ----
        if (i > 0 && o_col >= nblk * 128) {
          // O has its own columns: they must have been read out before being overwritten
          ok = mbar_wait(bar_oread, ph ^ 1, abort_flag);
          if (!ok) break;
        }
        for (int j = 0; j < nblk && ok; ++j) {
          ok = mbar_wait(&bar_p[j], ph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint32_t pa = smem_u32(sP + (j & 1) * 2 * FewSmem::kTile);
          const uint32_t va = smem_u32(sV + j * FewSmem::kTile);
#pragma unroll
          for (int s = 0; s < 8; ++s)
            umma_bf16(tmem_base + o_col,
                      make_smem_desc_sw128(pa + (s >> 2) * FewSmem::kTile + (s & 3) * 32, 16, 1024),
                      make_smem_desc_sw128(va + s * 2048, 8192, 1024), idesc_o, (j | s) != 0);
          umma_commit(&bar_pv[j]);
        }
      }
      if (!ok) {
        report_status(p.status, kStatusTimeoutMma, kKernelIdAttnFwd, blockIdx.x, blockIdx.y);
        *abort_flag = 1;
      }
    }
  } else {
    // ------------------------------ softmax warps ------------------------------
    // (the operand loads and the first score MMAs are under way while these tables are filled)
    // Bias by relative offset for this head: sRel[u], u = (k - q) + lq_pad - 1.
    if (p.rel_bias != nullptr) {
      const float* tab = p.rel_bias + static_cast<long long>(h) * p.num_buckets;
      for (int u = threadIdx.x; u < lq_pad + nblk * 128; u += kSoftmaxThreads)
        sRel[u] = rel_bias_at(p, tab, u - (lq_pad - 1) + p.rel_off);
    }
    // Per-key metadata: segment id (0 when unpacked), and whether the key exists and is not masked.
    for (int k = threadIdx.x; k < 512; k += kSoftmaxThreads) {
      const long long off = static_cast<long long>(b) * p.Lk + k;
      sKeySeg[k] = k < p.Lk && p.kv_seg != nullptr ? p.kv_seg[off] : 0;
      const uint32_t word =
          __ballot_sync(0xffffffffu, k < p.Lk && (p.key_mask == nullptr || p.key_mask[off] != 0));
      if (lane == 0) sKeyWord[k >> 5] = word;
    }
    softmax_bar_sync();
    const int quarter = warp & 3, part = warp >> 2;  // 4 threads per row, 32 columns each
    const int r = quarter * 32 + lane;               // row of the tile == TMEM lane
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const bool has_bias = p.rel_bias != nullptr;
    bool ok = true;
    // Key-only visibility (padding / key mask) and in-range bits, fixed for the whole CTA.
    uint32_t kvis[4], inr[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int left = p.Lk - (j * 128 + part * 32);  // keys from this chunk's first to the end
      kvis[j] = sKeyWord[j * 4 + part];
      inr[j] = left >= 32 ? 0xffffffffu : (left <= 0 ? 0u : ((1u << left) - 1u));
    }
    // (past a wait that gave up the group barriers are passed all the same, and nothing is stored)
    for (int i = 0; i < nq; ++i) {
      const uint32_t ph = i & 1;
      const int q = i * 128 + r;
      const int qseg = (p.q_seg != nullptr && q < p.Lq) ? p.q_seg[static_cast<long long>(b) * p.Lq + q] : 0;
      const int kmax = p.causal ? q + p.causal_off : 0x7fffffff;
      // Visibility bits of this thread's keys: chunk j covers keys j*128 + part*32 .. +31.
      uint32_t vis[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint32_t mvis = kvis[j];
        if (p.causal) {
          const int n = kmax - (j * 128 + part * 32) + 1;  // number of leading visible keys
          mvis &= n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : ((1u << n) - 1u));
        }
        if (p.kv_seg != nullptr && j < nblk) {
          uint32_t ms = 0;
          for (int x = 0; x < 32; ++x)
            ms |= (sKeySeg[j * 128 + part * 32 + x] == qseg ? 1u : 0u) << x;
          mvis &= ms;
        }
        vis[j] = mvis;
      }
      // ---- pass 1: row max ----
      float m = -3.0e38f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j >= nblk || !ok) break;
        ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&bar_s[j], ph, abort_flag));
        if (!ok) break;
        tc_fence_after();
        uint32_t v[32];
        const int col0 = j * 128 + part * 32;
        tmem_ld32(t_row + col0, v);
        tmem_ld_wait();
        const float* rel = sRel + (col0 - q + lq_pad - 1);
        if (vis[j] == 0xffffffffu) {
#pragma unroll
          for (int x = 0; x < 32; ++x) {
            float sc = __uint_as_float(v[x]);
            if (has_bias) sc += rel[x];
            m = fmaxf(m, sc);
          }
        } else {
          const uint32_t mv = vis[j], mi = inr[j];
#pragma unroll
          for (int x = 0; x < 32; ++x) {
            float sc = __uint_as_float(v[x]);
            if (has_bias) sc += rel[x];
            sc = ((mv >> x) & 1u) ? sc : kMaskValue;
            if ((mi >> x) & 1u) m = fmaxf(m, sc);
          }
        }
      }
      sStat[r * 4 + part] = m;
      softmax_bar_sync();
      m = fmaxf(fmaxf(sStat[r * 4], sStat[r * 4 + 1]), fmaxf(sStat[r * 4 + 2], sStat[r * 4 + 3]));
      const float m2 = m * kLog2e;
      // ---- pass 2: probabilities -> smem (bf16), row sums ----
      float l = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j >= nblk || !ok) break;
        // P buffer (j & 1) was last read by the PV MMA of block j-2 (this query block) or of
        // the last block with the same parity of the previous query block.
        if (j >= 2) {
          ok = mbar_wait_relaxed(&bar_pv[j - 2], ph, abort_flag);
        } else if (i > 0) {
          const int jp = ((nblk - 1 - j) & ~1) + j;  // last block index with parity j
          if (jp < nblk) ok = mbar_wait_relaxed(&bar_pv[jp], ph ^ 1, abort_flag);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        uint8_t* ptile = sP + (j & 1) * 2 * FewSmem::kTile + (part >> 1) * FewSmem::kTile;
        uint32_t v[32];
        const int col0 = j * 128 + part * 32;
        tmem_ld32(t_row + col0, v);
        tmem_ld_wait();
        const float* rel = sRel + (col0 - q + lq_pad - 1);
        float pr[32];
        if (vis[j] == 0xffffffffu) {
#pragma unroll
          for (int x = 0; x < 32; ++x) {
            float sc = __uint_as_float(v[x]);
            if (has_bias) sc += rel[x];
            const float e = exp2f(fmaf(sc, kLog2e, -m2));
            pr[x] = e;
            l += e;
          }
        } else {
          const uint32_t mv = vis[j], mi = inr[j];
#pragma unroll
          for (int x = 0; x < 32; ++x) {
            float sc = __uint_as_float(v[x]);
            if (has_bias) sc += rel[x];
            sc = ((mv >> x) & 1u) ? sc : kMaskValue;
            // subtract first: a fully masked row has sc == m == -1e10 and must give exp2(0)
            const float e = ((mi >> x) & 1u) ? exp2f((sc - m) * kLog2e) : 0.f;
            pr[x] = e;
            l += e;
          }
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) store_swizzled_chunk(ptile, r, (part & 1) * 4 + g, pr + g * 8);
        tc_fence_before();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_p[j]);
      }
      sStat[512 + r * 4 + part] = l;
      softmax_bar_sync();
      l = (sStat[512 + r * 4] + sStat[512 + r * 4 + 1]) + (sStat[512 + r * 4 + 2] + sStat[512 + r * 4 + 3]);
      // ---- epilogue: O / l (each of the 4 threads of a row writes 16 of the 64 columns) ----
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&bar_pv[nblk - 1], ph, abort_flag));
      if (ok) {
        tc_fence_after();
        uint32_t v[16];
        tmem_ld16(t_row + o_col + part * 16, v);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_oread);
        if (q < p.Lq) {
          __nv_bfloat16* dst =
              p.O + b * p.o_sb + static_cast<long long>(q) * p.o_sl + h * p.o_sh + part * 16;
          store16_bf16(dst, v, 1.f / l);
          if (part == 0 && p.lse != nullptr)
            p.lse[(static_cast<long long>(b) * p.H + h) * p.Lq + q] = m + __logf(l);
        }
      }
      // sStat is rewritten by the next query block only after everyone read the sums
      softmax_bar_sync();
    }
    if (!ok && lane == 0) {
      report_status(p.status, kStatusTimeoutEpilogue, kKernelIdAttnFwd, blockIdx.x, blockIdx.y);
      *abort_flag = 1;
    }
  }
  if (*abort_flag && threadIdx.x == 0)
    for (int it = 0; it < 2000; ++it) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == kCtrlWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}
}  // namespace
}  // namespace t5x

using namespace t5x;

// As t5x_attention_fwd, for up to 512 queries and keys without a prefix mask.
T5X_API int t5x_attention_fwd_few(const void* q, const void* k, const void* v, void* o, void* lse, int B,
                              int H, int Lq, int Lk, long long q_sb, long long q_sl, long long q_sh,
                              long long k_sb, long long k_sl, long long k_sh, long long v_sb,
                              long long v_sl, long long v_sh, long long o_sb, long long o_sl,
                              long long o_sh, const void* rel_bias, const void* rel_bucket,
                              int num_buckets, int nrel, int rel_off, const void* key_mask,
                              const void* q_seg, const void* kv_seg, int causal, int causal_off,
                              void* stream) {
  if (B <= 0 || H <= 0 || Lq <= 0 || Lk <= 0) return 0;
  if (Lq > kFewMax || Lk > kFewMax || causal == 2)
    return set_error("attention_fwd_few: %d queries, %d keys, mask %d are not covered", Lq, Lk, causal);
  if (B > 65535) return set_error("attention_fwd_few: B beyond the grid limit");
  if ((o_sb | o_sl | o_sh) & 7 || !aligned_to(16, {o}))
    return set_error("attention_fwd_few: output rows must be 16-byte aligned");
  CUtensorMap tq, tk, tv;
  if (!bhld_map(&tq, q, B, Lq, H, q_sb, q_sl, q_sh) || !bhld_map(&tk, k, B, Lk, H, k_sb, k_sl, k_sh) ||
      !bhld_map(&tv, v, B, Lk, H, v_sb, v_sl, v_sh))
    return -1;
  AttnParams p = {};
  p.B = B; p.H = H; p.Lq = Lq; p.Lk = Lk;
  p.rel_bias = static_cast<const float*>(rel_bias);
  p.rel_bucket = static_cast<const int*>(rel_bucket);
  p.num_buckets = num_buckets;
  p.nrel = nrel; p.rel_off = rel_off;
  p.key_mask = static_cast<const uint8_t*>(key_mask);
  p.q_seg = static_cast<const int*>(q_seg);
  p.kv_seg = static_cast<const int*>(kv_seg);
  p.causal = causal; p.causal_off = causal_off;
  p.O = static_cast<__nv_bfloat16*>(o);
  p.o_sb = o_sb; p.o_sl = o_sl; p.o_sh = o_sh;
  p.lse = static_cast<float*>(lse);
  p.status = device_status_buffer();
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_few_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         FewSmem::kTotal);
    if (e != cudaSuccess) return set_error("attention_fwd_few attr: %s", cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  dim3 grid(H, B);
  attn_fwd_few_kernel<<<grid, kAttnThreads, FewSmem::kTotal, static_cast<cudaStream_t>(stream)>>>(
      tq, tk, tv, p);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("attention_fwd_few: %s", cudaGetErrorString(e));
  return 0;
}
