// Flash attention backward on sm_100a, head_dim 64 or 128, up to 4096 queries: the gradients of softmax(Q K^T +
// bias(k - q) + mask) V, no 1/sqrt(d) scaling (T5 folds it into the query initialiser).
//
// All five GEMMs run on tcgen05 with accumulators in TMEM; Q/K/V/dO tiles arrive by TMA (128-byte swizzle, no
// multicast) and the P and dS tiles are written by the softmax warps straight into the swizzled shared layout
// that the next MMA reads. The [b,h,q,k] score matrix never exists in global memory. Bias and masks are
// generated in-kernel from per-token metadata:
//   bias      : rel_bias[h][rel_bucket[(k - q) + rel_off]]  (the T5 bucket table; the bucket of
//               each relative position comes from the host, bit-identical to the oracle)
//   masks     : key padding [B,Lk], causal (k <= q + causal_off), packed-segment ids.
// Masked logits take the value -1e10 (not -inf): a fully masked row gives a uniform distribution, exactly
// like the additive-mask formulation of the reference.
//
// One CTA per (128-key block, head, batch), looping over query blocks; dK/dV accumulate in TMEM, dQ partial
// tiles are added to an fp32 buffer with vector red.global.add. (attention_bwd_head_sm100.cu is the faster one
// for 64 channels where there are heads enough.)
#include "attention_common.cuh"
#include "t5x_ops.h"

namespace t5x {

// ---------------------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------------------
// delta[b,h,q] = sum_d dO[b,q,h,d] * O[b,q,h,d]
template <int D>
__global__ void __launch_bounds__(256)
    attn_delta_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O,
                      float* __restrict__ delta, int B, int H, int Lq, long long do_sb,
                      long long do_sl, long long do_sh, long long o_sb, long long o_sl,
                      long long o_sh) {
  // D / 8 lanes per (b, q, h): one 16-byte load per lane and tensor; four items in flight per
  // thread. Requires 16-byte aligned rows (strides multiples of 8 elements).
  constexpr int kLanes = D / 8;           // 8 or 16
  constexpr int kShift = (D == 64) ? 3 : 4;
  const long long total = static_cast<long long>(B) * Lq * H;
  const int sub = threadIdx.x & (kLanes - 1);
  const long long first = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) >> kShift;
  const long long stride = (static_cast<long long>(gridDim.x) * blockDim.x) >> kShift;
  // the lane groups of a warp leave the loop together (the shuffles use the full mask)
  const int group = (threadIdx.x & 31) >> kShift;
  for (long long w0 = first; w0 - group < total; w0 += 4 * stride) {
    uint4 a[4], c[4];
    long long out[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const long long w = w0 + u * stride;
      out[u] = -1;
      if (w < total) {
        const int hh = static_cast<int>(w % H);
        const long long t = w / H;
        const int q = static_cast<int>(t % Lq);
        const int bb = static_cast<int>(t / Lq);
        a[u] = *reinterpret_cast<const uint4*>(dO + bb * do_sb + static_cast<long long>(q) * do_sl +
                                               hh * do_sh + sub * 8);
        c[u] = *reinterpret_cast<const uint4*>(O + bb * o_sb + static_cast<long long>(q) * o_sl +
                                               hh * o_sh + sub * 8);
        out[u] = (static_cast<long long>(bb) * H + hh) * Lq + q;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      float s = 0.f;
      if (out[u] >= 0) {
        const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a[u]);
        const __nv_bfloat162* pc = reinterpret_cast<const __nv_bfloat162*>(&c[u]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 fa = __bfloat1622float2(pa[j]), fc = __bfloat1622float2(pc[j]);
          s += fa.x * fc.x + fa.y * fc.y;
        }
      }
      if (kLanes == 16) s += __shfl_xor_sync(0xffffffffu, s, 8);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if (sub == 0 && out[u] >= 0) delta[out[u]] = s;
    }
  }
}

constexpr int kSmemBuckets = 128;  // tables with more buckets add to memory directly
// P and dS of 16 scores of one key that all count: rel points at the bias of the first, the next
// ones lie below it.
template <bool kBias>
__device__ __forceinline__ void visible_scores(const uint32_t (&sv)[16], const uint32_t (&dpv)[16],
                                               const float* rel, const float (&lse)[16],
                                               const float (&delta)[16], float (&pr)[16],
                                               float (&ds)[16]) {
#pragma unroll
  for (int x = 0; x < 16; ++x) {
    float s = __uint_as_float(sv[x]);
    if (kBias) s += rel[-x];
    s = fmaxf(s, kMaskValue);
    pr[x] = exp2f(fmaf(s, kLog2e, -lse[x]));
    ds[x] = pr[x] * (__uint_as_float(dpv[x]) - delta[x]);
  }
}

// head_dim 64: Q / dO double-buffered, the scores of the next query block are issued while the
// softmax warps work, dQ partial tiles alternate between two TMEM buffers. head_dim 128: operand
// tiles are twice as large and dK, dV take twice the TMEM columns, so Q / dO have one stage, dQ
// reuses the columns of S^T and the query blocks run one after the other.
template <int D>
struct BwdSmem {
  static constexpr int kTile = 128 * 128;  // bytes of a [128 x 64] bf16 panel
  static constexpr int kPanels = D / 64;
  static constexpr int kStages = (D == 64) ? 2 : 1;
  static constexpr int kK = 0;
  static constexpr int kV = kK + kPanels * kTile;
  static constexpr int kQ = kV + kPanels * kTile;                 // kStages x kPanels
  static constexpr int kDO = kQ + kStages * kPanels * kTile;      // kStages x kPanels
  static constexpr int kPT = kDO + kStages * kPanels * kTile;     // P^T : 2 panels (128 keys x 128 queries)
  static constexpr int kDST = kPT + 2 * kTile;                    // dS^T: 2 panels
  static constexpr int kVec = kDST + 2 * kTile;     // 2 stages x {lse[128], delta[128], qseg[128]}
  static constexpr int kRel = kVec + 2 * 3 * 128 * 4;   // bias by rel for the (i, j) pair: 2 x 256 floats
  static constexpr int kDRel = kRel + 2 * 256 * 4;      // d bias by rel accumulators: (Lq_pad + 128) floats
  static constexpr int kBucket = kDRel + (4096 + 128) * 4;  // bias gradient by bucket
  static constexpr int kBars = kBucket + kSmemBuckets * 4;
  static constexpr int kTotal = kBars + 256 + 1024;
};

// kAhead: causal self-attention, where query blocks may be passed over (a variant of its own: the
// first block held in a register costs the other one spills).
template <int D, bool kAhead>
__global__ void __launch_bounds__(kAttnThreads, 1)
    attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                    const AttnParams p) {
  using Smem = BwdSmem<D>;
  constexpr int kPanels = Smem::kPanels;
  constexpr int kStageBytes = kPanels * Smem::kTile;  // one Q (or dO) stage
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* sK = smem + Smem::kK;
  uint8_t* sV = smem + Smem::kV;
  uint8_t* sQ = smem + Smem::kQ;
  uint8_t* sDO = smem + Smem::kDO;
  uint8_t* sPT = smem + Smem::kPT;
  uint8_t* sDST = smem + Smem::kDST;
  float* sVec = reinterpret_cast<float*>(smem + Smem::kVec);
  float* sRelAll = reinterpret_cast<float*>(smem + Smem::kRel);
  float* sDRel = reinterpret_cast<float*>(smem + Smem::kDRel);
  float* sBucket = reinterpret_cast<float*>(smem + Smem::kBucket);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Smem::kBars);
  uint64_t* bar_kv = bars;          // 1
  uint64_t* bar_qdo = bars + 1;     // 2 (full, per stage)
  uint64_t* bar_free = bars + 3;    // 2 (stage consumed by the MMAs)
  uint64_t* bar_s = bars + 5;       // S^T and dP^T ready
  uint64_t* bar_p = bars + 6;       // P^T / dS^T written, S^T / dP^T released
  uint64_t* bar_dq = bars + 7;      // dQ partial ready (also: P^T/dS^T smem consumed)
  uint64_t* bar_dq_read = bars + 8; // dQ partial consumed
  uint64_t* bar_sfree = bars + 9;   // S^T / dP^T columns read into registers
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 10);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k0 = blockIdx.x * 128, h = blockIdx.y, b = blockIdx.z;
  const int lq_pad = (p.Lq + 127) / 128 * 128;
  // TMEM columns
  // dQ partial tiles alternate between two 64-column buffers, so that the tile of query block
  // i is read out while the MMAs of block i + 1 run.
  constexpr int cS = 0, cDP = 128;
  constexpr int cDQ = (D == 64) ? 256 : 0;     // head_dim 128: dQ takes over the columns of S^T
  constexpr int cDK = (D == 64) ? 384 : 256;
  constexpr int cDV = (D == 64) ? 448 : 384;
  constexpr int kColsPerPart = D / 4;          // output columns per thread of a row

  if (threadIdx.x == 0) {
    mbar_init(bar_kv, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar_qdo[s], 1);
      mbar_init(&bar_free[s], 1);
    }
    mbar_init(bar_s, 1);
    mbar_init(bar_p, kSoftmaxWarps);
    mbar_init(bar_dq, 1);
    mbar_init(bar_dq_read, kSoftmaxWarps);
    mbar_init(bar_sfree, kSoftmaxWarps);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kCtrlWarp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  // The block's key mask, where it alone hides keys: requested here, so that it arrives during the set-up
  // (128 x 12 heads x 114 x 512, all keys visible, us without a look / with / so: 479 / 489 / 482).
  int shown = key_mask_alone(p) ? 0 : 1;
  if (!shown && threadIdx.x < 128 && k0 + static_cast<int>(threadIdx.x) < p.Lk)
    shown = p.key_mask[static_cast<long long>(b) * p.Lk + k0 + threadIdx.x];
  if (p.d_rel_bias != nullptr) {
    for (int t = threadIdx.x; t < lq_pad + 128; t += kAttnThreads) sDRel[t] = 0.f;
    if (threadIdx.x < kSmemBuckets) sBucket[threadIdx.x] = 0.f;
  }
  tc_fence_before();
  const bool any_shown = __syncthreads_or(shown);
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // A block of hidden keys (the padding of a batch) has exact zeros for P and dS wherever a query sees
  // any key. With nothing but a key mask all queries do or none does, as the first one's lse tells.
  // (Keys of which 60 to 100 % are visible, us before / so: 32 x 64 heads x 512 x 512 1480 / 1352, 16 x
  // 6 x 1024 x 1024 326 / 284, 8 x 32 x 1024 x 1024 of 128 features 979 / 861; none hidden: 1140 / 1140.)
  const bool idle = !any_shown &&  // (then the key mask stands alone)
                    p.lse[(static_cast<long long>(b) * p.H + h) * p.Lq] >= -5e9f;

  // Of causal self-attention the query blocks ahead of this key block see nothing of it (unless both
  // lie in the prefix of a prefix LM), and where each of their queries sees itself their P and dS are
  // exact zeros: the walk starts at the first block behind them. (us before / so: causal, 8 x 32 heads
  // of 128 x 1024 1205 / 838, 32 x 12 x 256 182 / 170; prefix LM, 16 x 12 x 1024, 600 tokens in the
  // prefix, 730 / 612, but 4 x 12 x 300 109 / 114: from more than kAheadKeys keys on.)
  int q_first = 0;
  if (kAhead && k0 > 0) {
    bool keep = false;
    for (int q = threadIdx.x; q < k0 + 128 && q < p.Lk; q += kAttnThreads)
      keep = keep || (q < k0 ? !sees_itself(p, b, q) : in_prefix(p, b, q));
    if (!__syncthreads_or(keep)) q_first = k0;
  }
  const int nq = (lq_pad - (kAhead ? q_first : 0)) / 128;

  if (idle) {
    for (int i = threadIdx.x; i < 128 * (D / 8); i += kAttnThreads) {
      const int k = k0 + i / (D / 8);
      if (k < p.Lk) {
        const long long off = b * p.dk_sb + static_cast<long long>(k) * p.dk_sl + h * p.dk_sh + i % (D / 8) * 8;
        *reinterpret_cast<uint4*>(p.dK + off) = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(p.dV + off) = make_uint4(0u, 0u, 0u, 0u);
      }
    }
  } else if (warp == kCtrlWarp) {
    if (lane == 0) {
      bool ok = true;
      mbar_expect_tx(bar_kv, 2 * kStageBytes);
      for (int c = 0; c < kPanels; ++c) {
        tma_load_4d(sK + c * Smem::kTile, &tmK, bar_kv, c * 64, h, k0, b);
        tma_load_4d(sV + c * Smem::kTile, &tmV, bar_kv, c * 64, h, k0, b);
      }
      auto load_qdo = [&](int i, int st) {
        mbar_expect_tx(&bar_qdo[st], 2 * kStageBytes);
        for (int c = 0; c < kPanels; ++c) {
          tma_load_4d(sQ + st * kStageBytes + c * Smem::kTile, &tmQ, &bar_qdo[st], c * 64, h,
                      (kAhead ? q_first : 0) + i * 128, b);
          tma_load_4d(sDO + st * kStageBytes + c * Smem::kTile, &tmDO, &bar_qdo[st], c * 64, h,
                      (kAhead ? q_first : 0) + i * 128, b);
        }
      };
      for (int i = 0; i < nq && i < Smem::kStages; ++i) load_qdo(i, i);
      const uint32_t idesc_kq = make_idesc_bf16(128, 128, 0, 0);  // [keys x queries], K = d
      const uint32_t idesc_kd = make_idesc_bf16(128, D, 0, 1);    // [keys x d], K = queries (B MN-major)
      const uint32_t idesc_qd = make_idesc_bf16(128, D, 1, 1);    // [queries x d], A and B MN-major
      const uint32_t ka = smem_u32(sK), va = smem_u32(sV);
      const uint32_t pta = smem_u32(sPT), dsta = smem_u32(sDST);

      auto issue_scores = [&](int st) {  // S^T = K Q_i^T ; dP^T = V dO_i^T
        const uint32_t qa = smem_u32(sQ + st * kStageBytes);
        const uint32_t doa = smem_u32(sDO + st * kStageBytes);
#pragma unroll
        for (int s = 0; s < D / 16; ++s)
          umma_bf16(tmem_base + cS,
                    make_smem_desc_sw128(ka + (s >> 2) * Smem::kTile + (s & 3) * 32, 16, 1024),
                    make_smem_desc_sw128(qa + (s >> 2) * Smem::kTile + (s & 3) * 32, 16, 1024),
                    idesc_kq, s != 0);
#pragma unroll
        for (int s = 0; s < D / 16; ++s)
          umma_bf16(tmem_base + cDP,
                    make_smem_desc_sw128(va + (s >> 2) * Smem::kTile + (s & 3) * 32, 16, 1024),
                    make_smem_desc_sw128(doa + (s >> 2) * Smem::kTile + (s & 3) * 32, 16, 1024),
                    idesc_kq, s != 0);
        umma_commit(bar_s);
      };
      // dV += P^T dO ; dK += dS^T Q ; dQ_i = dS K. The B operands hold d contiguous (MN-major):
      // 64-channel groups are one panel apart, 16 rows of the K dimension 2048 bytes.
      auto issue_grads = [&](int i, int st, int dq_col) {
        const uint32_t qa = smem_u32(sQ + st * kStageBytes);
        const uint32_t doa = smem_u32(sDO + st * kStageBytes);
#pragma unroll
        for (int s = 0; s < 8; ++s)
          umma_bf16(tmem_base + cDV,
                    make_smem_desc_sw128(pta + (s >> 2) * Smem::kTile + (s & 3) * 32, 16, 1024),
                    make_smem_desc_sw128(doa + s * 2048, Smem::kTile, 1024), idesc_kd, (i | s) != 0);
#pragma unroll
        for (int s = 0; s < 8; ++s)
          umma_bf16(tmem_base + cDK,
                    make_smem_desc_sw128(dsta + (s >> 2) * Smem::kTile + (s & 3) * 32, 16, 1024),
                    make_smem_desc_sw128(qa + s * 2048, Smem::kTile, 1024), idesc_kd, (i | s) != 0);
        // A = dS (M = queries) read from the dS^T tiles as an MN-major operand: 64-query groups
        // are kTile apart (LBO), 8-key groups 1024 B apart (SBO); K advances 16 keys = 2048 B.
#pragma unroll
        for (int s = 0; s < 8; ++s)
          umma_bf16(tmem_base + dq_col,
                    make_smem_desc_sw128(dsta + s * 2048, Smem::kTile, 1024),
                    make_smem_desc_sw128(ka + s * 2048, Smem::kTile, 1024), idesc_qd, s != 0);
        umma_commit(bar_dq);
      };

      ok = mbar_wait(bar_kv, 0, abort_flag) && mbar_wait(&bar_qdo[0], 0, abort_flag);
      if (ok) {
        tc_fence_after();
        issue_scores(0);
      }
      if constexpr (D == 64) {
        // Order per query block i: the scores of block i + 1 are issued as soon as the softmax
        // warps hold those of block i in registers (bar_sfree), so they are computed while the
        // warps do their arithmetic; the gradient MMAs of block i follow when P^T / dS^T are
        // in shared memory (bar_p).
        for (int i = 0; i < nq && ok; ++i) {
          const int st = i & 1;
          const uint32_t ph = (i >> 1) & 1;
          ok = mbar_wait(bar_sfree, i & 1, abort_flag);
          if (ok && i + 1 < nq) {
            ok = mbar_wait(&bar_qdo[(i + 1) & 1], ((i + 1) >> 1) & 1, abort_flag);
            if (ok) {
              tc_fence_after();
              issue_scores((i + 1) & 1);
            }
          }
          if (ok) ok = mbar_wait(bar_p, i & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          issue_grads(i, st, cDQ + (i & 1) * 64);
          umma_commit(&bar_free[st]);
          // The softmax warps read dQ_{i-1} right after they signalled bar_p for block i; once
          // they have, its buffer is free for dQ_{i+1}. (Waiting here, not before the next
          // block's MMAs, keeps at most one completion of bar_dq_read ahead of this wait.)
          if (i >= 1 && i + 1 < nq) {
            ok = mbar_wait(bar_dq_read, (i - 1) & 1, abort_flag);
            if (!ok) break;
          }
          // refill this stage with query block i + 2
          if (i + 2 < nq) {
            ok = mbar_wait(&bar_free[st], ph, abort_flag);
            if (!ok) break;
            load_qdo(i + 2, st);
          }
        }
      } else {
        // One query block at a time: scores, softmax, gradient MMAs, dQ read-out (from the
        // columns of S^T), then the next block's operands and scores.
        for (int i = 0; i < nq && ok; ++i) {
          ok = mbar_wait(bar_p, i & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          issue_grads(i, 0, cDQ);
          umma_commit(&bar_free[0]);
          if (i + 1 < nq) {
            ok = mbar_wait(&bar_free[0], i & 1, abort_flag);
            if (!ok) break;
            load_qdo(i + 1, 0);
            ok = mbar_wait(bar_dq_read, i & 1, abort_flag) &&
                 mbar_wait(&bar_qdo[0], (i + 1) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            issue_scores(0);
          }
        }
      }
      if (!ok) {
        report_status(p.status, kStatusTimeoutMma, kKernelIdAttnBwd, blockIdx.x, blockIdx.y);
        *abort_flag = 1;
      }
    }
  } else {
    // ------------------------------ softmax / gradient warps ------------------------------
    const int quarter = warp & 3, part = warp >> 2;  // 4 threads per key row, 32 queries each
    const int r = quarter * 32 + lane;               // key row of the tile == TMEM lane
    const int k = k0 + r;
    const bool k_ok = k < p.Lk;
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    bool kvis = k_ok;
    if (p.key_mask && k_ok) kvis = p.key_mask[static_cast<long long>(b) * p.Lk + k] != 0;
    // causal == 2: prefix LM (segment codes carry "inside the prefix" in bit 30; a key inside
    // the prefix is visible to every query inside the prefix)
    const bool prefix_lm = p.causal == 2;
    const int seg_mask = prefix_lm ? 0x3fffffff : -1;
    const int kcode = (p.kv_seg && k_ok) ? p.kv_seg[static_cast<long long>(b) * p.Lk + k] : 0;
    const int kseg = kcode & seg_mask;
    const bool k_pre = prefix_lm && ((kcode >> 30) & 1);
    const float inv_lk = 1.f / static_cast<float>(p.Lk);
    const bool has_bias = p.rel_bias != nullptr;
    const bool simple_mask = !p.causal && p.kv_seg == nullptr;
    bool ok = true;

    // Per-query vectors of block i go to stage (i & 1) of shared memory; all softmax threads
    // cooperate (thread t < 128: lse, delta and segment id of query t; the next 255 threads:
    // the bias by relative position over the (key block, query block) pair, index
    // u = r - c + 127). `fetch` issues the global loads early, `publish` stores them after the
    // arithmetic of the current block, so their latency is off the critical path.
    float pf_a = 0.f, pf_b = 0.f;
    int pf_c = 0;
    const float* head_table =
        has_bias ? p.rel_bias + static_cast<long long>(h) * p.num_buckets : nullptr;
    auto fetch_vectors = [&](int i) {
      const int qb = (kAhead ? q_first : 0) + i * 128;
      const int t = threadIdx.x;
      if (t < 128) {
        const int q = qb + t;
        const long long off = (static_cast<long long>(b) * p.H + h) * p.Lq + q;
        pf_a = (q < p.Lq) ? p.lse[off] * kLog2e : 0.f;
        pf_b = (q < p.Lq) ? p.delta[off] : 0.f;
        pf_c = (p.q_seg && q < p.Lq) ? p.q_seg[static_cast<long long>(b) * p.Lq + q] : 0;
      } else if (t < 128 + 255 && has_bias) {
        const int u = t - 128;
        const int idx = (k0 - qb) + (u - 127) + p.rel_off;
        pf_c = (idx >= 0 && idx < p.nrel) ? __ldg(p.rel_bucket + idx) : -1;
      }
    };
    // bucket -> bias, once the bucket has arrived and still ahead of its use
    auto resolve_bias = [&]() {
      if (has_bias && threadIdx.x >= 128 && threadIdx.x < 128 + 255)
        pf_a = pf_c >= 0 ? __ldg(head_table + pf_c) : 0.f;
    };
    auto publish_vectors = [&](int i) {
      float* sLse = sVec + (i & 1) * 384;
      float* sDelta = sLse + 128;
      int* sQseg = reinterpret_cast<int*>(sDelta + 128);
      float* sRel = sRelAll + (i & 1) * 256;
      const int t = threadIdx.x;
      if (t < 128) {
        sLse[t] = pf_a;
        sDelta[t] = pf_b;
        sQseg[t] = pf_c;
      } else if (t < 128 + 255 && has_bias) {
        sRel[t - 128] = pf_a;
      }
    };

    auto read_dq = [&](int blk, bool release) {
      uint32_t v[kColsPerPart];
      if constexpr (D == 64) {
        tmem_ld16(t_row + cDQ + (blk & 1) * 64 + part * 16, v);
      } else {
        tmem_ld32(t_row + cDQ + part * 32, v);
      }
      tmem_ld_wait();
      if (release) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_dq_read);
      }
      // Four lanes exchange their 16-byte pieces, so that an instruction adds 64 contiguous bytes
      // of 8 rows instead of 16 of 32 (128 x 12 heads x 512 x 512 1009 / 976 us).
      const int q0 = (kAhead ? q_first : 0) + blk * 128 + quarter * 32 + (lane & ~3);
      float* dst = p.dQ + ((static_cast<long long>(b) * p.Lq + q0) * p.H + h) * D +
                   part * kColsPerPart + (lane & 3) * 4;
      const long long row_step = static_cast<long long>(p.H) * D;
#pragma unroll
      for (int x = 0; x < kColsPerPart; x += 16) {
        transpose_pieces(v + x, lane);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (q0 + i < p.Lq)
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(
                             dst + i * row_step + x),
                         "f"(__uint_as_float(v[x + 4 * i])), "f"(__uint_as_float(v[x + 4 * i + 1])),
                         "f"(__uint_as_float(v[x + 4 * i + 2])),
                         "f"(__uint_as_float(v[x + 4 * i + 3]))
                         : "memory");
      }
    };

    fetch_vectors(0);
    resolve_bias();
    publish_vectors(0);
    softmax_bar_sync();
    for (int i = 0; i < nq && ok; ++i) {
      const int qb = (kAhead ? q_first : 0) + i * 128;
      const float* sLse = sVec + (i & 1) * 384;
      const float* sDelta = sLse + 128;
      const int* sQseg = reinterpret_cast<const int*>(sDelta + 128);
      const float* sRel = sRelAll + (i & 1) * 256;
      if (i + 1 < nq) fetch_vectors(i + 1);  // published before the sync at the loop end
      const int col0 = part * 32;  // query column within the block
      // visibility of (this key, queries col0..col0+31)
      uint32_t mv;
      if (simple_mask) {
        mv = kvis ? 0xffffffffu : 0u;
      } else {
        mv = 0;
        for (int x = 0; x < 32; ++x) {
          const int q = qb + col0 + x;
          bool v = kvis;
          const int qcode = sQseg[col0 + x];
          if (p.causal) v = v && (k <= q + p.causal_off || (k_pre && ((qcode >> 30) & 1)));
          if (p.kv_seg) v = v && (kseg == (qcode & seg_mask));
          mv |= (v ? 1u : 0u) << x;
        }
      }
      ok = mbar_wait_relaxed(bar_s, i & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      // 16 columns (queries) at a time keeps the working set in registers: scores and dP of
      // the chunk, its per-query statistics, and the packed bf16 results.
      const float* rel = sRel + (r - col0 + 127);
      // The kernel is bound by the instructions per score (42 with every case in one body, at half
      // of the issue slots). Where all of a warp's 32 x 32 block counts, and no query in it has all
      // its keys hidden, it takes a body without any of those cases (us: 128 x 12 heads x 512 x 512
      // 976 / 925, 8 x 32 x 1024 x 1024 of 128 features 880 / 805).
      const bool fast = qb + col0 + 32 <= p.Lq &&
                        __all_sync(0xffffffffu,
                                   mv == 0xffffffffu && sLse[col0 + lane] >= -5e9f);
      uint8_t* pt_tile = sPT + (part >> 1) * Smem::kTile;
      uint8_t* dst_tile = sDST + (part >> 1) * Smem::kTile;
      // Bias gradient: dS[key r][query c] belongs to bin (r - c). Within the warp's 32 x 32
      // block (lane = key row, x = query column) lane L collects diagonal L and diagonal L - 32:
      // at column x it fetches the value of lane (L + x) mod 32, which lies on diagonal L when
      // L + x < 32 and on diagonal L - 32 otherwise. The 32 shuffles are independent of each
      // other, and the block costs two shared-memory atomics per lane instead of 32. (Masks
      // are additive, so the bias receives dS everywhere.)
      const bool want_drel = p.d_rel_bias != nullptr;
      float* bins = sDRel + (quarter * 32 - qb - col0 + lq_pad);  // bins[lane - x]
      float diag_pos = 0.f, diag_neg = 0.f;
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        uint32_t sv[16], dpv[16];
        tmem_ld16(t_row + cS + col0 + hc * 16, sv);
        tmem_ld16(t_row + cDP + col0 + hc * 16, dpv);
        tmem_ld_wait();
        if (hc == 1) {
          // all of S^T / dP^T of this block is in registers: the scores of the next block may
          // overwrite the columns while the arithmetic below runs
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_sfree);
        }
        float lse_c[16], del_c[16];
#pragma unroll
        for (int g = 0; g < 4; ++g) {  // 16-byte broadcast loads of the per-query statistics
          const float4 a = reinterpret_cast<const float4*>(sLse + col0 + hc * 16)[g];
          const float4 d = reinterpret_cast<const float4*>(sDelta + col0 + hc * 16)[g];
          lse_c[4 * g] = a.x, lse_c[4 * g + 1] = a.y, lse_c[4 * g + 2] = a.z, lse_c[4 * g + 3] = a.w;
          del_c[4 * g] = d.x, del_c[4 * g + 1] = d.y, del_c[4 * g + 2] = d.z, del_c[4 * g + 3] = d.w;
        }
        float pr[16], ds[16];
        if (fast) {
          if (has_bias)
            visible_scores<true>(sv, dpv, rel - hc * 16, lse_c, del_c, pr, ds);
          else
            visible_scores<false>(sv, dpv, rel, lse_c, del_c, pr, ds);
        } else {
#pragma unroll
          for (int x = 0; x < 16; ++x) {
            const int xx = hc * 16 + x;
            float s = __uint_as_float(sv[x]);
            if (has_bias) s += rel[-xx];
            s = ((mv >> xx) & 1u) ? s : kMaskValue;
            float e = exp2f(fmaf(s, kLog2e, -lse_c[x]));
            // A row with every key masked has lse = -1e10 + log(Lk), which fp32 rounds to -1e10:
            // its probabilities are uniform over the Lk keys.
            if (lse_c[x] < -5e9f) e = inv_lk;
            if (!k_ok || qb + col0 + xx >= p.Lq) e = 0.f;
            pr[x] = e;
            ds[x] = e * (__uint_as_float(dpv[x]) - del_c[x]);
          }
        }
        if (want_drel) {
#pragma unroll
          for (int x = 0; x < 16; ++x) {
            const int xx = hc * 16 + x;
            const float v = __shfl_sync(0xffffffffu, ds[x], lane + xx);  // (modulo 32)
            if (lane + xx < 32) {
              diag_pos += v;
            } else {
              diag_neg += v;
            }
          }
        }
        if (hc == 0 && i + 1 < nq) resolve_bias();
        if (D == 64 && hc == 0 && i > 0) {
          // the gradient MMAs of block i - 1 still read P^T / dS^T; they also produce dQ_{i-1}
          // (head_dim 128 has waited for them already, at the end of block i - 1)
          ok = mbar_wait_relaxed(bar_dq, (i - 1) & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          store_swizzled_chunk(pt_tile, r, (part & 1) * 4 + hc * 2 + g, pr + g * 8);
          store_swizzled_chunk(dst_tile, r, (part & 1) * 4 + hc * 2 + g, ds + g * 8);
        }
      }
      if (want_drel) {
        atomicAdd(bins + lane, diag_pos);
        if (lane != 0) atomicAdd(bins + (lane - 32), diag_neg);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_p);
      if (!ok) break;
      // dQ partial of the previous block (its MMAs were waited for above), while the MMAs of
      // this block run: rows are queries here (TMEM lane = query within the block), 16 columns
      // per thread.
      if constexpr (D == 64) {
        if (i > 0) read_dq(i - 1, true);
      } else {
        // dQ_i sits in the columns of S^T: out before the next block's scores may be issued
        ok = mbar_wait_relaxed(bar_dq, i & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        read_dq(i, true);
      }
      if (i + 1 < nq) publish_vectors(i + 1);  // other stage than the one block i used
      softmax_bar_sync();  // the vectors of block i+1 are complete; those of block i are dead
    }
    // the bucket of this thread's first relative position, requested before the last MMAs are
    // waited for
    int first_bucket = -1;
    if (p.d_rel_bias != nullptr) {
      const int idx = k0 + (static_cast<int>(threadIdx.x) - lq_pad) + p.rel_off;
      if (idx >= 0 && idx < p.nrel) first_bucket = __ldg(p.rel_bucket + idx);
    }
    if (D == 64 && ok) {
      ok = mbar_wait_relaxed(bar_dq, (nq - 1) & 1, abort_flag);
      if (ok) {
        tc_fence_after();
        read_dq(nq - 1, false);
      }
    }
    if (ok) {
      // dK, dV accumulators are complete once the last bar_dq fired (same commit group).
#pragma unroll
      for (int c = 0; c < kColsPerPart / 16; ++c) {
        uint32_t vk[16], vv[16];
        tmem_ld16(t_row + cDK + part * kColsPerPart + c * 16, vk);
        tmem_ld16(t_row + cDV + part * kColsPerPart + c * 16, vv);
        tmem_ld_wait();
        if (k_ok) {
          const long long off = b * p.dk_sb + static_cast<long long>(k) * p.dk_sl + h * p.dk_sh +
                                part * kColsPerPart + c * 16;
          store16_bf16(p.dK + off, vk, 1.f);
          store16_bf16(p.dV + off, vv, 1.f);
        }
      }
      softmax_bar_sync();
      if (p.d_rel_bias != nullptr) {
        // sDRel[t] holds sum dS over (k - q) = k0 + t - lq_pad for this key block. The relative
        // positions are folded into their buckets here (a few dozen sums per head), so that one
        // CTA adds num_buckets values to memory and no expanded gradient exists.
        // Neighbouring positions share buckets (far ones a single bucket): each run of equal
        // buckets in a warp is summed by shuffles and added once.
        float* out = p.d_rel_bias + static_cast<long long>(h) * p.num_buckets;
        const bool in_smem = p.num_buckets <= kSmemBuckets;
        float* bucket_sum = in_smem ? sBucket : out;
        for (int t = threadIdx.x; t < lq_pad + 128; t += kSoftmaxThreads) {  // whole warps
          float g = sDRel[t];
          const int idx = k0 + (t - lq_pad) + p.rel_off;  // (k - q) + rel_off
          const int bucket =
              t == threadIdx.x ? first_bucket
                               : ((idx >= 0 && idx < p.nrel) ? __ldg(p.rel_bucket + idx) : -1);
          const int before = __shfl_up_sync(0xffffffffu, bucket, 1);
          const bool head = lane == 0 || before != bucket;
          const uint32_t heads = __ballot_sync(0xffffffffu, head);
          const uint32_t later = lane == 31 ? 0u : heads >> (lane + 1);
          const int run_end = later ? lane + __ffs(later) : 32;  // first lane of the next run
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float v = __shfl_down_sync(0xffffffffu, g, o);
            if (lane + o < run_end) g += v;
          }
          if (head && bucket >= 0 && g != 0.f) atomicAdd(bucket_sum + bucket, g);
        }
        if (in_smem) {
          softmax_bar_sync();
          for (int t = threadIdx.x; t < p.num_buckets; t += kSoftmaxThreads)
            if (bucket_sum[t] != 0.f) atomicAdd(out + t, bucket_sum[t]);
        }
      }
    } else if (lane == 0) {
      report_status(p.status, kStatusTimeoutEpilogue, kKernelIdAttnBwd, blockIdx.x, blockIdx.y);
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

}  // namespace t5x

using namespace t5x;

namespace t5x {
template <int D, bool kAhead>
static int launch_attention_bwd(const void* d_o, const void* o, void* delta, const CUtensorMap* tq,
                                const CUtensorMap* tk, const CUtensorMap* tv,
                                const CUtensorMap* tdo, const AttnParams& p, long long do_sb,
                                long long do_sl, long long do_sh, long long o_sb, long long o_sl,
                                long long o_sh, cudaStream_t st) {
  long long items = static_cast<long long>(p.B) * p.Lq * p.H;
  long long blocks = (items * (D / 8) / 4 + 255) / 256;
  long long cap = static_cast<long long>(num_sms()) * 8;
  attn_delta_kernel<D><<<static_cast<int>(blocks > cap ? cap : blocks), 256, 0, st>>>(
      static_cast<const __nv_bfloat16*>(d_o), static_cast<const __nv_bfloat16*>(o),
      static_cast<float*>(delta), p.B, p.H, p.Lq, do_sb, do_sl, do_sh, o_sb, o_sl, o_sh);
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_kernel<D, kAhead>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         BwdSmem<D>::kTotal);
    if (e != cudaSuccess) return set_error("attention_bwd attr: %s", cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  dim3 grid((p.Lk + 127) / 128, p.H, p.B);
  attn_bwd_kernel<D, kAhead><<<grid, kAttnThreads, BwdSmem<D>::kTotal, st>>>(*tq, *tk, *tv, *tdo, p);
  count_launches(2);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("attention_bwd: %s", cudaGetErrorString(e));
  return 0;
}
}  // namespace t5x

// dq_f32 [B,Lq,H,D] fp32 contiguous, zero on entry. delta [B,H,Lq] fp32 scratch. D = 64 or 128.
T5X_API int t5x_attention_bwd(const void* q, const void* k, const void* v, const void* o,
                              const void* d_o, const void* lse, void* delta, void* dq_f32, void* dk,
                              void* dv, int B, int H, int Lq, int Lk, int D, long long q_sb,
                              long long q_sl, long long q_sh, long long k_sb, long long k_sl,
                              long long k_sh, long long v_sb, long long v_sl, long long v_sh,
                              long long o_sb, long long o_sl, long long o_sh, long long do_sb,
                              long long do_sl, long long do_sh, long long dk_sb, long long dk_sl,
                              long long dk_sh, const void* rel_bias, const void* rel_bucket,
                              void* d_rel_bias, int num_buckets, int nrel, int rel_off,
                              const void* key_mask, const void* q_seg,
                              const void* kv_seg, int causal, int causal_off, void* stream) {
  if (B <= 0 || H <= 0 || Lq <= 0 || Lk <= 0) return 0;
  if (D != 64 && D != 128) return set_error("attention_bwd: head_dim %d not in {64, 128}", D);
  if (Lq > 4096) return set_error("attention_bwd: Lq=%d > 4096 is not covered by this kernel", Lq);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  CUtensorMap tq, tk, tv, tdo;
  if (!bhld_map(&tq, q, B, Lq, H, q_sb, q_sl, q_sh, D) || !bhld_map(&tk, k, B, Lk, H, k_sb, k_sl, k_sh, D) ||
      !bhld_map(&tv, v, B, Lk, H, v_sb, v_sl, v_sh, D) ||
      !bhld_map(&tdo, d_o, B, Lq, H, do_sb, do_sl, do_sh, D))
    return -1;
  if ((do_sb | do_sl | do_sh | o_sb | o_sl | o_sh | dk_sb | dk_sl | dk_sh) & 7)
    return set_error("attention_bwd: dO / O / dK strides must be multiples of 8 elements");
  AttnParams p = {};
  p.B = B; p.H = H; p.Lq = Lq; p.Lk = Lk;
  p.rel_bias = static_cast<const float*>(rel_bias);
  p.rel_bucket = static_cast<const int*>(rel_bucket);
  p.num_buckets = num_buckets;
  p.d_rel_bias = static_cast<float*>(d_rel_bias);
  p.nrel = nrel; p.rel_off = rel_off;
  p.key_mask = static_cast<const uint8_t*>(key_mask);
  p.q_seg = static_cast<const int*>(q_seg);
  p.kv_seg = static_cast<const int*>(kv_seg);
  p.causal = causal; p.causal_off = causal_off;
  p.lse = const_cast<float*>(static_cast<const float*>(lse));
  p.delta = static_cast<const float*>(delta);
  p.dQ = static_cast<float*>(dq_f32);
  p.dK = static_cast<__nv_bfloat16*>(dk);
  p.dV = static_cast<__nv_bfloat16*>(dv);
  p.dk_sb = dk_sb; p.dk_sl = dk_sl; p.dk_sh = dk_sh;
  p.status = device_status_buffer();
  const bool ahead = causal && Lq == Lk && causal_off == 0 && Lq > (causal == 2 ? kAheadKeys : 128);
  const auto launch = D == 128 ? (ahead ? launch_attention_bwd<128, true> : launch_attention_bwd<128, false>)
                               : (ahead ? launch_attention_bwd<64, true> : launch_attention_bwd<64, false>);
  return launch(d_o, o, delta, &tq, &tk, &tv, &tdo, p, do_sb, do_sl, do_sh, o_sb, o_sl, o_sh, st);
}
