// Flash attention forward on sm_100a for head_dim 64: softmax(Q K^T + bias(k - q) + mask) V, bias and masks as
// in attention_common.cuh (hidden scores take the value -1e10; no 1/sqrt(d) scaling).
//
// A softmax group of four warps owns 128 query rows, a thread a row: nothing is exchanged between threads. A
// CTA has two groups (256 queries of a head; of 128 queries or fewer the groups take every other block of 64
// keys), and two CTAs share an SM. What bounds the kernel is the chain of
// steps of a group (scores from TMEM, exponentials, probabilities to shared memory, fences, barriers): four
// groups in different phases fill one another's gaps (52 % of the issue slots are taken with 16 x 12 heads x 512 x
// 512). Where heads leave SMs idle, attention_fwd_few_sm100.cu is the faster one.
// (us, T5-like scores; one CTA of 16 warps per SM with the scores of all keys in TMEM / here: 128 x 12 heads x
// 512 x 512 with bias, 60 to 100 % of the keys visible 410 / 305, 114 x 512 without bias 117 / 103, 114 x 114
// causal 80 / 60. Two groups of four warps per SM in blocks of 128 keys, the kernel in attention_fwd_sm100.cu /
// here: 16 x 6 x 1024 x 1024 148 / 89, 16 x 12 x 1024 prefix LM 341 / 184, 16 x 6 x 189 x 1024 52 / 37.)
//
// A step is 32 keys of a row. P goes to a panel of 64 keys, in halves; the P V products are issued by halves.
// Of long key ranges the maximum in use is raised only by scores that exceed it by more than 8 ln 2 (until then
// every exponential stays below 256, exact in fp32 sums), so O in TMEM is rescaled rarely; of up to 512 keys
// the exact maximum comes first (kShort).
//
//   warps 0-3 / 4-7  groups 0 / 1
//   warp 8           issues the MMAs of both groups
//   warp 9           TMA: Q, then K and V in blocks of 64 keys through a ring of two stages (three where the
//                    groups share the queries: the third is where other queries would be)
//
// TMEM (256 columns): group g: S at 64 g, O at 128 + 64 g.
#include <type_traits>

#include "attention_common.cuh"
#include "t5x_ops.h"

namespace t5x {
namespace {

constexpr int kRowsThreads = 320;
constexpr int kRowsMma = 8, kRowsTma = 9;
constexpr int kMaxSteps = 64;       // of 32 keys
constexpr int kCopy = 872;          // floats of one of four copies of the bias table (8 banks further each)
constexpr int kTable = 4 * kCopy;
constexpr int kShortKeys = 512;
static_assert(256 + kShortKeys <= kCopy && 256 + 32 * kMaxSteps <= kTable, "the bias tables");
constexpr int kRowsKernelId = 13;
constexpr float kGap = 5.5451774f;  // 8 ln 2

struct RowsSmem {
  static constexpr int kPanel = 128 * 128;  // [128 x 64] bf16
  static constexpr int kBlock = 64 * 128;   // [64 x 64] bf16
  static constexpr int kQ = 0;                      // 2 panels
  static constexpr int kP = kQ + 2 * kPanel;        // 2 panels
  static constexpr int kKV = kP + 2 * kPanel;       // 2 stages x (K, V)
  static constexpr int kRel = kKV + 4 * kBlock;     // bias by (k - q)
  static constexpr int kVis = kRel + kTable * 4;    // bit x of word s: key 32 s + x may be seen
  static constexpr int kPre = kVis + kMaxSteps * 4;  // ... lies in the prefix (prefix LM)
  static constexpr int kSeg = kPre + kMaxSteps * 4;  // the segment of all keys of a step, or kMixedSeg
  static constexpr int kJoin = kSeg + kMaxSteps * 4;  // maximum and sum of group 1's rows (queries shared)
  static constexpr int kFlat = kJoin + 256 * 4;       // by t / 32: the bias is one value over these 32
  static constexpr int kBars = kFlat + (kTable / 32 + 7) / 8 * 8;
  static constexpr int kTotal = kBars + 28 * 8 + 1024;
};
static_assert(2 * (RowsSmem::kTotal + 1024) <= 233472, "two CTAs per SM");
static_assert(RowsSmem::kBars % 8 == 0, "barriers are 8-byte words");
constexpr int kMixedSeg = 0x7fffffff;

__device__ __forceinline__ uint32_t first_bits(int n) {  // n ones, n clamped to 0..32
  return n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : ((1u << n) - 1u));
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void add_to(uint32_t& a, float x) {
  a = __float_as_uint(__uint_as_float(a) + x);
}

// kShort (up to 512 keys): the exact maximum of a row comes first, from a walk of its own over all scores, which
// are then computed again: the largest probability is exactly one, and with it the error of O is 2.06e-3 where
// the maximum in use gives 2.32e-3 (64-bit reference, scores of standard deviation 1.4, 512 keys). That walk has
// two buffers for scores (O is not in use yet) and costs some 60 of 300 us. The bias table stands four times,
// shifted by 0..3, so that a thread reads its 32 consecutive entries 16 bytes at a time whatever its row.
// Otherwise (up to 2048 keys) the maximum is the one in use, and the table stands once.
template <bool kShort>
__global__ void __launch_bounds__(kRowsThreads, 2)
    attn_fwd_rows_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                         const __grid_constant__ AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  float* sRel = reinterpret_cast<float*>(smem + RowsSmem::kRel);
  uint32_t* sVis = reinterpret_cast<uint32_t*>(smem + RowsSmem::kVis);
  uint32_t* sPre = reinterpret_cast<uint32_t*>(smem + RowsSmem::kPre);
  int* sSeg = reinterpret_cast<int*>(smem + RowsSmem::kSeg);
  float* sJoin = reinterpret_cast<float*>(smem + RowsSmem::kJoin);
  uint8_t* sFlat = smem + RowsSmem::kFlat;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + RowsSmem::kBars);
  uint64_t* bar_q = bars;            // Q landed
  uint64_t* bar_kv = bars + 1;       // 3: K and V of a block landed
  uint64_t* bar_kvfree = bars + 4;   // 3: ... and are no longer read
  uint64_t* bar_s = bars + 7;        // per group and buffer: S of a block is in TMEM
  uint64_t* bar_sfree = bars + 11;   // per group and buffer: ... and in registers
  uint64_t* bar_p = bars + 15;       // per group and half: P is in shared memory
  uint64_t* bar_pv = bars + 19;      // per group and half: P V is done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 23);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* sFlags = reinterpret_cast<int*>(tmem_slot + 2);  // per group: a query that does not see itself, one in
                                                        // the prefix; [4]: last prefix key + 1

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.y, b = blockIdx.z;
  const int q_base = blockIdx.x * 256;
  const bool pair = p.Lq - q_base > 128;  // each group has queries of its own
  const int all_blocks = (p.Lk + 63) / 64;
  // groups that share their queries, and the maximum, add to one O, in the order of the keys
  const bool one_o = kShort && !pair;
  const bool once = kShort && all_blocks == 1;  // the scores stay where they are for the second walk
  constexpr int cO = 128;

  if (threadIdx.x == 0) {
    mbar_init(bar_q, 1);
    for (int i = 0; i < 3; ++i) {
      mbar_init(&bar_kv[i], 1);
      mbar_init(&bar_kvfree[i], 1);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&bar_s[i], 1);
      mbar_init(&bar_sfree[i], 4);
      mbar_init(&bar_p[i], 4);
      mbar_init(&bar_pv[i], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (threadIdx.x < 5) sFlags[threadIdx.x] = 0;
  if (warp == kRowsMma) {
    tmem_alloc(tmem_slot, 256);
    tmem_relinquish();
  }
  // the n-th load's stage of the ring, which use of the stage it is, and where the stage is
  const int ring = pair ? 2 : 3;
  auto stage_of = [&](int n) { return pair ? n & 1 : n % 3; };
  auto use_of = [&](int n) { return pair ? n >> 1 : n / 3; };
  auto place_of = [&](int st) {
    return st < 2 ? RowsSmem::kKV + st * 2 * RowsSmem::kBlock : RowsSmem::kQ + RowsSmem::kPanel;
  };
  auto load_block = [&](int n, int j, bool values) {
    const int st = stage_of(n);
    uint8_t* at = smem + place_of(st);
    mbar_expect_tx(&bar_kv[st], (values ? 2 : 1) * RowsSmem::kBlock);
    tma_load_4d(at, &tmK, &bar_kv[st], 0, h, j * 64, b);
    if (values) tma_load_4d(at + RowsSmem::kBlock, &tmV, &bar_kv[st], 0, h, j * 64, b);
  };
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (warp == kRowsTma && lane == 0) {  // (the first block always counts)
    mbar_expect_tx(bar_q, (pair ? 2 : 1) * RowsSmem::kPanel);
    tma_load_4d(smem + RowsSmem::kQ, &tmQ, bar_q, 0, h, q_base, b);
    if (pair) tma_load_4d(smem + RowsSmem::kQ + RowsSmem::kPanel, &tmQ, bar_q, 0, h, q_base + 128, b);
    load_block(0, 0, !kShort || once);
  }
  __syncwarp();

  // ---- tables, while the operands travel ----
  const int group = warp >> 2;  // (of the first eight warps)
  const int r = (warp & 3) * 32 + lane;  // row of the tile == TMEM lane
  const int q0 = q_base + (pair ? group * 128 : 0);
  const int q = q0 + r;
  const bool prefix_lm = p.causal == 2;
  const int seg_mask = prefix_lm ? 0x3fffffff : -1;
  const bool has_bias = p.rel_bias != nullptr;
  // table index t: k - q = t - t_zero
  const int t_zero = 255 + q_base, rels = 256 + all_blocks * 64;
  int qcode = 0;
  if (warp < 8) {
    if (p.q_seg != nullptr && q < p.Lq) qcode = p.q_seg[static_cast<long long>(b) * p.Lq + q];
    for (int s = warp; s < all_blocks * 2; s += 8) {
      const int k = s * 32 + lane;
      const long long at = static_cast<long long>(b) * p.Lk + k;
      const bool vis = k < p.Lk && (p.key_mask == nullptr || p.key_mask[at] != 0);
      const int code = (k < p.Lk && p.kv_seg != nullptr) ? p.kv_seg[at] : 0;
      const uint32_t v = __ballot_sync(0xffffffffu, vis);
      const uint32_t pre = __ballot_sync(0xffffffffu, prefix_lm && ((code >> 30) & 1));
      const int seg = code & seg_mask, first = __shfl_sync(0xffffffffu, seg, 0);
      const bool one = __all_sync(0xffffffffu, seg == first);
      if (lane == 0) {
        sVis[s] = v;
        sPre[s] = pre;
        sSeg[s] = one ? first : kMixedSeg;
        if (pre != 0u) atomicMax(&sFlags[4], s * 32 + 32 - __clz(pre));
      }
    }
    if (p.causal) {
      const bool self = p.Lq == p.Lk && p.causal_off == 0;
      if (q < p.Lq && !(self && sees_itself(p, b, q))) sFlags[2 * group] = 1;
      if (q < p.Lq && prefix_lm && ((qcode >> 30) & 1)) sFlags[2 * group + 1] = 1;
    }
    if (has_bias) {
      const float* tab = p.rel_bias + static_cast<long long>(h) * p.num_buckets;
      for (int t1 = warp * 32 + lane; t1 - lane < rels; t1 += 4 * 256) {  // (whole warps; four loads at a time)
        int bucket[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int t = t1 + c * 256, idx = t - t_zero + p.rel_off;
          bucket[c] = t < rels && idx >= 0 && idx < p.nrel ? __ldg(p.rel_bucket + idx) : -1;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int t = t1 + c * 256;
          if (t - lane >= rels) break;
          const float x = bucket[c] >= 0 ? __ldg(tab + bucket[c]) : 0.f;
          if (kShort) {
#pragma unroll
            for (int m = 0; m < 4; ++m)  // copy m holds entry i + m at i
              if (t >= m) sRel[m * kCopy + t - m] = x;
          } else {
            sRel[t] = x;
          }
          const bool one = __all_sync(0xffffffffu, x == __shfl_sync(0xffffffffu, x, 0));
          if (lane == 0) sFlat[t >> 5] = one;
        }
      }
    }
  }
  __syncthreads();
  // Blocks of 64 keys that a group walks. What lies behind them is hidden from all its queries, each of which
  // sees some key, so that it would contribute exact zeros: the end of a key mask, or what lies ahead of a
  // causal tile.
  auto blocks_of = [&](int g) {
    int n = all_blocks;
    const int last_q = min(p.Lq, q_base + (pair ? g * 128 : 0) + 128) - 1;
    if (p.causal) {
      if (p.key_mask == nullptr && p.kv_seg == nullptr) {
        if (p.causal_off >= 0) n = static_cast<int>(min(static_cast<long long>(n),
                                                      (static_cast<long long>(last_q) + p.causal_off) / 64 + 1));
      } else if (!sFlags[2 * g]) {
        n = min(n, max(last_q, sFlags[2 * g + 1] ? sFlags[4] - 1 : -1) / 64 + 1);
      }
    } else if (p.key_mask != nullptr && p.kv_seg == nullptr) {
      int s = 2 * all_blocks - 1;
      while (s >= 0 && sVis[s] == 0u) --s;
      if (s >= 0) n = s / 2 + 1;
    }
    return n;
  };
  // (in a CTA of one tile group 0 takes the even blocks, group 1 the odd ones)
  const int n0 = blocks_of(0), n1 = pair ? blocks_of(1) : n0;
  const int blocks = max(n0, n1);

  if (warp == kRowsTma) {
    if (lane == 0) {
      bool ok = true;
      for (int n = 1; n < (kShort && !once ? 2 : 1) * blocks && ok; ++n) {
        if (n >= ring) ok = mbar_wait(&bar_kvfree[stage_of(n)], (use_of(n) - 1) & 1, abort_flag);
        const bool values = !kShort || n >= blocks;
        if (ok) load_block(n, kShort && values ? n - blocks : n, values);
      }
      if (!ok) {
        report_status(p.status, kStatusTimeoutProducer, kRowsKernelId, blockIdx.x, blockIdx.y);
        *abort_flag = 1;
      }
    }
  } else if (warp == kRowsMma) {
    // The whole warp walks and one lane issues (descriptors in uniform registers, an addition apart).
    const bool leader = elect_one();
    const uint32_t idesc_s = make_idesc_bf16(128, 64, 0, 0);
    const uint32_t idesc_o = make_idesc_bf16(128, 64, 0, 1);
    const uint64_t row_major = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
    const uint64_t col_major = make_smem_desc_sw128(smem_u32(smem), RowsSmem::kBlock, 1024);
    constexpr uint32_t kP16 = RowsSmem::kPanel >> 4, kB16 = RowsSmem::kBlock >> 4;
    const int count[2] = {pair ? n0 : (n0 + 1) / 2, pair ? n1 : n0 / 2};  // blocks of the group
    bool ok = mbar_wait(bar_q, 0, abort_flag);
    // The scores of the i-th block of a group (of the first walk, in two buffers in turn; where they stay, the
    // first buffer goes on).
    auto issue_scores = [&](int g, int i, bool walk) {
      if (i >= count[g] || !ok || (once && !walk)) return;
      const int j = pair ? i : 2 * i + g;
      const int n = walk || !kShort ? j : blocks + j, st = stage_of(n);
      const int buf = walk ? i & 1 : 0;
      const int use = walk ? i >> 1 : (kShort ? (count[g] + 1) / 2 : 0) + i;  // of the buffer
      ok = mbar_wait(&bar_kv[st], use_of(n) & 1, abort_flag) &&
           (use == 0 || mbar_wait(&bar_sfree[2 * g + buf], (use - 1) & 1, abort_flag));
      if (!ok) return;
      tc_fence_after();
      const uint64_t qd = row_major + (RowsSmem::kQ >> 4) + (pair ? g : 0) * kP16;
      const uint64_t kd = row_major + static_cast<uint32_t>(place_of(st) >> 4);
      const bool last = walk && !once && (!pair || g == 1 || i >= count[1]);
      if (leader) {
#pragma unroll
        for (int s = 0; s < 4; ++s)
          umma_bf16(tmem_base + g * 64 + buf * cO, qd + 2 * s, kd + 2 * s, idesc_s, s != 0);
        umma_commit(&bar_s[2 * g + buf]);
        if (last) umma_commit(&bar_kvfree[st]);
      }
    };
    // P V of half of it; the last product that reads the block gives its place in the ring free
    auto issue_values = [&](int g, int i, int half) {
      if (i >= count[g] || !ok) return;
      ok = mbar_wait(&bar_p[g * 2 + half], i & 1, abort_flag);
      if (!ok) return;
      tc_fence_after();
      const int j = pair ? i : 2 * i + g;
      const uint64_t pd = row_major + (RowsSmem::kP >> 4) + g * kP16 + static_cast<uint32_t>(half) * 4;
      const int st = stage_of(kShort && !once ? blocks + j : j);
      const uint64_t vd = col_major + static_cast<uint32_t>(place_of(st) >> 4) + kB16 +
                          static_cast<uint32_t>(half) * 256;
      const bool last = half == 1 && (!pair || g == 1 || i >= count[1]);
      if (leader) {
#pragma unroll
        for (int s = 0; s < 2; ++s)
          umma_bf16(tmem_base + cO + (one_o ? 0 : g * 64), pd + 2 * s, vd + 128 * s, idesc_o,
                    ((one_o ? j : i) | half | s) != 0);
        umma_commit(&bar_pv[g * 2 + half]);
        if (last) umma_commit(&bar_kvfree[st]);
      }
    };
    if (kShort) {
      for (int i = 0; i < max(count[0], count[1]) && ok; ++i) {
        issue_scores(0, i, true);
        issue_scores(1, i, true);
      }
    }
    issue_scores(0, 0, false);
    issue_scores(1, 0, false);
    for (int i = 0; i < max(count[0], count[1]) && ok; ++i) {
      issue_values(0, i, 0);
      if (!one_o) issue_values(1, i, 0);
      issue_scores(0, i + 1, false);
      issue_values(0, i, 1);
      if (one_o) issue_values(1, i, 0);
      issue_scores(1, i + 1, false);
      issue_values(1, i, 1);
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0) report_status(p.status, kStatusTimeoutMma, kRowsKernelId, blockIdx.x, blockIdx.y);
      *abort_flag = 1;
    }
  } else {
    const int g = group;
    const uint32_t t_s = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + g * 64;
    const uint32_t t_o = t_s + cO;
    uint8_t* p_row = smem + RowsSmem::kP + g * RowsSmem::kPanel + r * 128;
    const int qseg = qcode & seg_mask;
    const bool q_pre = prefix_lm && ((qcode >> 30) & 1);
    const int mine = g == 0 ? n0 : n1;
    const uint64_t log2e2 = pair_of(kLog2e, kLog2e);
    // The steps whose bias is one value for the warp (bits of lo, hi: steps 0..31, 32..63), and those whose
    // keys all count.
    uint32_t flat_steps[2] = {0xffffffffu, 0xffffffffu}, full_steps[2];
    const int t_warp = t_zero - (q0 + (warp & 3) * 32);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int step = c * 32 + lane;
      const bool there = step < 2 * all_blocks;
      full_steps[c] = __ballot_sync(0xffffffffu, there && sVis[step] == 0xffffffffu);
      if (has_bias) {
        const int t0 = step * 32 + t_warp, a = (t0 - 31) >> 5;
        flat_steps[c] = __ballot_sync(
            0xffffffffu, there && sFlat[a] && sFlat[a + 1] && sRel[t0 - 31] == sRel[t0 + 1]);
      }
    }
    const bool by_row = p.causal || p.kv_seg != nullptr;  // visibility differs from row to row
    bool ok = true;
    float m = 0.f;  // the maximum, exact or in use
    // the row's sum, in four parts: 32 keys to each in turn (of a row whose keys two groups share, two and two)
    float sum = 0.f, sum1 = 0.f, sum2 = 0.f, sum3 = 0.f;
    // which keys of a step this row sees; whether all rows of the warp see all of them
    auto seen = [&](int step, bool& fast) {
      const int k0 = step * 32;
      const bool full = ((step < 32 ? full_steps[0] : full_steps[1]) >> (step & 31)) & 1u;
      uint32_t mv = 0xffffffffu;
      fast = full;
      if (!full) mv = sVis[step];
      if (p.kv_seg != nullptr) {
        const int seg = sSeg[step];
        if (seg != kMixedSeg) {
          mv = seg == qseg ? mv : 0u;
        } else {
          const int k = k0 + lane;
          const int code = k < p.Lk ? p.kv_seg[static_cast<long long>(b) * p.Lk + k] & seg_mask : 0;
          uint32_t same = 0u;
#pragma unroll 4
          for (int x = 0; x < 32; ++x) same |= (__shfl_sync(0xffffffffu, code, x) == qseg ? 1u : 0u) << x;
          mv &= same;
        }
      }
      if (p.causal) {
        const long long n = static_cast<long long>(q) + p.causal_off - k0 + 1;
        const uint32_t behind = first_bits(n > 32 ? 32 : (n < 0 ? 0 : static_cast<int>(n)));
        mv &= q_pre ? (behind | sPre[step]) : behind;
      }
      if (by_row) fast = __all_sync(0xffffffffu, mv == 0xffffffffu);
      return mv;
    };
    // The walk or two, 32 keys at a time. (Everything stands here once, unrolled over 32 scores and no more: with
    // the halves of a block side by side, or the masked case with exponentials of its own, the kernel waits for
    // its instructions, 297 us and more against 272.)
    const int blocks_here = pair ? mine : (mine - g + 1) / 2;
    int i = 0;      // blocks walked
    int uses = 0;   // of the first buffer, before the last walk
    if (kShort) m = -3.0e38f;
#pragma unroll 1
    for (int walk = kShort ? 0 : 1; walk < 2 && ok; ++walk) {
      const bool look = kShort && walk == 0;
#pragma unroll 1
      for (i = 0; i < blocks_here && ok; ++i) {
        const int buf = look ? i & 1 : 0;
        if (look || !once)
          ok = __all_sync(0xffffffffu, mbar_wait(&bar_s[2 * g + buf], (look ? i >> 1 : uses + i) & 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
          const int step = 2 * (pair ? i : 2 * i + g) + half, k0 = step * 32;
          uint32_t v[32];
          tmem_ld32(t_s + buf * cO + half * 32, v);
          bool fast;
          const uint32_t mv = seen(step, fast);
          const int at = k0 + t_warp - lane;  // table index of this row and the first key
          tmem_ld_wait();
          if (half == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar_sfree[2 * g + buf]);
          }
          // (single additions: in pairs, add.f32x2, 343 us instead of 305)
          float later = 0.f;  // a bias that is added to the maximum alone: rounding keeps the order of scores
          if (((step < 32 ? flat_steps[0] : flat_steps[1]) >> (step & 31)) & 1u) {
            if (has_bias) {
              const float one = sRel[at];
              if (look && fast) {
                later = one;
              } else {
#pragma unroll
                for (int x = 0; x < 32; ++x) add_to(v[x], one);
              }
            }
          } else if (kShort) {
            const float4* rel = reinterpret_cast<const float4*>(sRel + (at & 3) * kCopy + (at & ~3));
#pragma unroll
            for (int x = 0; x < 32; x += 4) {
              const float4 bias = rel[x / 4];
              add_to(v[x], bias.x);
              add_to(v[x + 1], bias.y);
              add_to(v[x + 2], bias.z);
              add_to(v[x + 3], bias.w);
            }
          } else {
#pragma unroll
            for (int x = 0; x < 32; ++x) add_to(v[x], sRel[at + x]);
          }
          if (!fast) {
            const uint32_t inside = first_bits(p.Lk - k0);
#pragma unroll
            for (int x = 0; x < 32; ++x) {
              const float hidden = ((inside >> x) & 1u) ? kMaskValue : -3.0e38f;  // beyond the last key: for nothing
              v[x] = ((mv >> x) & 1u) ? v[x] : __float_as_uint(hidden);
            }
          }
          float fix = 1.f;
          if (look || !kShort) {
            float top = -3.0e38f, top2 = -3.0e38f;
#pragma unroll
            for (int x = 0; x < 32; x += 4) {
              top = max3(top, __uint_as_float(v[x]), __uint_as_float(v[x + 1]));
              top2 = max3(top2, __uint_as_float(v[x + 2]), __uint_as_float(v[x + 3]));
            }
            top = fmaxf(top, top2) + later;
            if (look) {
              m = fmaxf(m, top);
              continue;
            }
            if (i == 0 && half == 0) {
              m = top;
            } else if (top > m + kGap) {
              fix = exp2f((m - top) * kLog2e);
              m = top;
              sum *= fix;
              sum1 *= fix;
              sum2 *= fix;
              sum3 *= fix;
            }
          }
          // the product that read this half of the panel last
          if (i > 0) ok = mbar_wait(&bar_pv[g * 2 + half], (i - 1) & 1, abort_flag);
          if (!kShort && __any_sync(0xffffffffu, fix != 1.f)) {
            // O is rescaled once the products issued so far are in it
            if (half == 1) ok = mbar_wait(&bar_pv[g * 2], i & 1, abort_flag) && ok;
            if (half == 0) ok = mbar_wait(&bar_pv[g * 2 + 1], (i - 1) & 1, abort_flag) && ok;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < 64; c += 16) {
              uint32_t o[16];
              tmem_ld16(t_o + c, o);
              tmem_ld_wait();
#pragma unroll
              for (int x = 0; x < 16; ++x) o[x] = __float_as_uint(__uint_as_float(o[x]) * fix);
              tmem_st16(t_o + c, o);
            }
            tmem_st_wait();
          }
          if (!ok) break;
          // Probabilities, rounded into the panel, and their sum, one after the other (in pairs 322 -> 335 us).
          // Where a row does not see all keys the difference comes before the product: without visible keys
          // each of its scores is m, -1e10, and gives one.
          const bool whole = mv == 0xffffffffu;
          const float less = whole ? -m * kLog2e : 0.f;
          const uint64_t m2 = pair_of(less, less);
          if (!fast) {
            const float before = whole ? 0.f : m;
#pragma unroll
            for (int x = 0; x < 32; ++x) v[x] = __float_as_uint(__uint_as_float(v[x]) - before);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t pp[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int x = 8 * c + 2 * e;
              const uint64_t t = fma2(pair_of(__uint_as_float(v[x]), __uint_as_float(v[x + 1])), log2e2, m2);
              const float e0 = exp2f(low_of(t)), e1 = exp2f(high_of(t));
              sum += e0;
              sum += e1;
              pp[e] = pack_bf16x2(e0, e1);
            }
            *reinterpret_cast<uint4*>(p_row + (((half * 4 + c) ^ (r & 7)) << 4)) =
                make_uint4(pp[0], pp[1], pp[2], pp[3]);
          }
          const float turn = sum;
          sum = sum1;
          sum1 = pair ? sum2 : turn;
          sum2 = sum3;
          sum3 = pair ? turn : 0.f;
          tc_fence_before();
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar_p[g * 2 + half]);
        }
      }
      if (look) {
        uses = (blocks_here + 1) / 2;
        if (!pair) {  // the maximum over the keys of both groups
          sJoin[2 * r + g] = m;
          asm volatile("bar.sync 3, 256;" ::: "memory");
          m = fmaxf(sJoin[2 * r], sJoin[2 * r + 1]);
          asm volatile("bar.sync 3, 256;" ::: "memory");  // (before sums take their place)
        }
      }
    }
    i = blocks_here;
    if (ok && i > 0) ok = __all_sync(0xffffffffu, mbar_wait(&bar_pv[g * 2 + 1], (i - 1) & 1, abort_flag));
    tc_fence_after();
    // ---- O / sum ----
    // (past a wait that gave up the group barriers are passed all the same, and nothing is stored)
    float l = (sum + sum1) + (sum2 + sum3), mine_by = 1.f, other_by = 0.f;
    if (!pair) {
      // group 1 leaves its maxima and sums; its O (if it has one) is in the same lanes of TMEM
      if (g == 1) {
        tc_fence_before();
        sJoin[2 * r] = i > 0 ? m : -3.0e38f;
        sJoin[2 * r + 1] = i > 0 ? l : 0.f;
        asm volatile("bar.arrive 3, 256;" ::: "memory");
      } else {
        asm volatile("bar.sync 3, 256;" ::: "memory");
        tc_fence_after();
        const float m1 = sJoin[2 * r], l1 = sJoin[2 * r + 1], all = fmaxf(m, m1);
        const float a = exp2f((m - all) * kLog2e), c = l1 > 0.f ? exp2f((m1 - all) * kLog2e) : 0.f;
        l = a * l + c * l1;
        m = all;
        mine_by = a;
        other_by = c;
      }
    }
    const bool joined = !pair && !one_o && n0 > 1;  // (group 1 has had a block)
    const float scale = 1.f / l;
    if (pair || g == 0) {
#pragma unroll 1
      for (int c = 0; c < 64; c += 16) {
        uint32_t o[16];
        tmem_ld16(t_o + c, o);
        tmem_ld_wait();
        float out[16];
#pragma unroll
        for (int x = 0; x < 16; ++x) out[x] = __uint_as_float(o[x]) * mine_by;
        if (joined) {
          tmem_ld16(t_o + 64 + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 16; ++x) out[x] = fmaf(__uint_as_float(o[x]), other_by, out[x]);
        }
#pragma unroll
        for (int x = 0; x < 16; ++x) out[x] *= scale;
        // (P is no longer read)
        store_swizzled_chunk(smem + RowsSmem::kP + g * RowsSmem::kPanel, r, c / 8, out);
        store_swizzled_chunk(smem + RowsSmem::kP + g * RowsSmem::kPanel, r, c / 8 + 1, out + 8);
      }
      if (p.lse != nullptr && ok && q < p.Lq)
        p.lse[(static_cast<long long>(b) * p.H + h) * p.Lq + q] = m + __logf(l);
      fence_proxy_async_smem();
      if (g == 0)
        asm volatile("bar.sync 1, 128;" ::: "memory");
      else
        asm volatile("bar.sync 2, 128;" ::: "memory");
      if (ok && (threadIdx.x & 127) == 0 && q0 < p.Lq) {
        tma_store_4d(&tmO, smem + RowsSmem::kP + g * RowsSmem::kPanel, 0, h, q0, b);
        bulk_commit();
        bulk_store_wait_all();
      }
    }
    if (!ok && lane == 0) {
      report_status(p.status, kStatusTimeoutEpilogue, kRowsKernelId, blockIdx.x, blockIdx.y);
      *abort_flag = 1;
    }
  }
  if (*abort_flag && threadIdx.x == 0)
    for (int it = 0; it < 2000; ++it) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == kRowsMma) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

template <bool kShort>
int launch_rows(const CUtensorMap* tq, const CUtensorMap* tk, const CUtensorMap* tv, const CUtensorMap* to,
                const AttnParams& p, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_rows_kernel<kShort>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         RowsSmem::kTotal);
    if (e != cudaSuccess) return set_error("attention_fwd attr: %s", cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  attn_fwd_rows_kernel<kShort>
      <<<dim3((p.Lq + 255) / 256, p.H, p.B), kRowsThreads, RowsSmem::kTotal, st>>>(*tq, *tk, *tv, *to, p);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("attention_fwd: %s", cudaGetErrorString(e));
  return 0;
}
}  // namespace
}  // namespace t5x

using namespace t5x;

// q [B,Lq,H,64], k/v [B,Lk,H,64] bf16 with element strides (sb, sl, sh), innermost contiguous.
// rel_bias [H, num_buckets] fp32 or null, rel_bucket [nrel] int32 in [0, num_buckets):
// bias = rel_bias[h][rel_bucket[(k - q) + rel_off]]. lse [B,H,Lq] fp32 or null.
T5X_API int t5x_attention_fwd(const void* q, const void* k, const void* v, void* o, void* lse, int B,
                              int H, int Lq, int Lk, long long q_sb, long long q_sl, long long q_sh,
                              long long k_sb, long long k_sl, long long k_sh, long long v_sb,
                              long long v_sl, long long v_sh, long long o_sb, long long o_sl,
                              long long o_sh, const void* rel_bias, const void* rel_bucket,
                              int num_buckets, int nrel, int rel_off, const void* key_mask,
                              const void* q_seg, const void* kv_seg, int causal, int causal_off,
                              void* stream) {
  if (B <= 0 || H <= 0 || Lq <= 0 || Lk <= 0) return 0;
  if (Lk > kMaxSteps * 32)
    return set_error("attention_fwd: Lk=%d > %d is not covered by this kernel", Lk, kMaxSteps * 32);
  if (B > 65535 || H > 65535) return set_error("attention_fwd: B or H beyond the grid limit");
  if ((o_sb | o_sl | o_sh) & 7 || !aligned_to(16, {o}))
    return set_error("attention_fwd: output rows must be 16-byte aligned");
  CUtensorMap tq, tk, tv, to;
  if (!bhld_map(&tq, q, B, Lq, H, q_sb, q_sl, q_sh) || !bhld_map(&tk, k, B, Lk, H, k_sb, k_sl, k_sh, 64, 64) ||
      !bhld_map(&tv, v, B, Lk, H, v_sb, v_sl, v_sh, 64, 64) || !bhld_map(&to, o, B, Lq, H, o_sb, o_sl, o_sh))
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
  p.lse = static_cast<float*>(lse);
  p.status = device_status_buffer();
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return (Lk <= kShortKeys ? launch_rows<true> : launch_rows<false>)(&tq, &tk, &tv, &to, p, st);
}
