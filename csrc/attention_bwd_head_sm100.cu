// Flash attention backward on sm_100a for head_dim 64: one CTA per head, example and 512 queries.
//
// The CTA walks the key blocks of its head and, inside each, the queries 64 at a time. dQ of all (up to
// four) query blocks stays in TMEM for the whole walk, dK and dV of a key block for its part of it, so all
// three gradients leave the chip once and in bf16: no fp32 dQ in memory that is cleared, added to and cast,
// and rowsum(dO * O) is computed while the first operands travel instead of by a kernel of its own.
//
// TMEM (512 columns): S^T 0..63, dP^T 64..127, dQ of query block i 128 + 64 i, dK 384, dV 448.
// Shared memory: K and V of two key blocks, Q and dO of three 64-query units, P^T of two units, dS^T of two
// query blocks. The MMA warp issues the scores of unit u + 1 as soon as the 16 softmax warps hold those of
// unit u in registers, and the gradient products of unit u - 1 while they do their arithmetic on unit u; the
// softmax warps never wait for one another inside the walk.
//
// One CTA per 128-key block (attention_sm100.cu) spends 14k cycles on setting up and tearing down a CTA and
// 6.7k on a 128 x 128 tile. Here a CTA takes some 14k and a 128 x 64 unit 2 to 3k, bound by what a softmax warp
// does one after the other for a unit (us, with rowsum(dO * O), clearing and casting of dQ where there are any,
// before / now: 128 x 12 heads x 512 x 512 1081 / 610, 114 x 512 without a bias 385 / 202, 114 x 114 causal
// 184 / 113, 24 x 12 x 509 packed 258 / 157, 32 x 64 x 512 x 512 1327 / 792). Of the 610, the bias gradient
// takes 100 (40 its additions to shared memory, which are loops around a compare-and-swap), the bias 35, the
// exponentials 8.
#include <algorithm>
#include <type_traits>

#include "attention_common.cuh"
#include "t5x_ops.h"

namespace t5x {
namespace {

constexpr int kMaxQ = 512;        // queries: 4 x 64 columns of TMEM for dQ
// Padded queries and keys together, with a bias table; and stages of Q and dO. Where the queries are cut into
// parts the tables are longer, in the place of a stage.
template <bool kParts>
constexpr int kMaxRelOf = kParts ? 1664 : 1152;
template <bool kParts>
constexpr int kRingOf = kParts ? 2 : 3;
constexpr int kMaxKeys = 4096;    // a bit per key block
constexpr int kBuckets = 128;     // bias tables of more buckets take the other kernel
constexpr int kOutside = 255, kMixed = 254;  // in tables of buckets: none, several
constexpr int kThreads = kSoftmaxThreads + 64;  // + MMA warp + TMA warp
constexpr int kMmaWarp = kSoftmaxWarps, kTmaWarp = kSoftmaxWarps + 1;
constexpr int kKernelId = 12;

template <bool kParts>
struct HeadSmem {
  static constexpr int kMaxRel = kMaxRelOf<kParts>, kRing = kRingOf<kParts>;
  static constexpr int kPanel = 128 * 128;  // [128 x 64] bf16
  static constexpr int kHalf = 64 * 128;    // [64 x 64] bf16
  static constexpr int kK = 0;              // 2 stages
  static constexpr int kV = kK + 2 * kPanel;
  static constexpr int kQ = kV + 2 * kPanel;       // kRing stages
  static constexpr int kDO = kQ + kRing * kHalf;   // kRing stages
  static constexpr int kP = kDO + kRing * kHalf;   // 2 x [128 keys x 64 queries]
  static constexpr int kDS = kP + 2 * kPanel;      // 2 query blocks x 2 x [128 keys x 64 queries]
  static constexpr int kVec = kDS + 4 * kPanel;    // -lse * log2(e), -rowsum(dO * O), query codes
  static constexpr int kRel = kVec + 3 * kMaxQ * 4;  // bias by (k - q)
  static constexpr int kDRel = kRel + kMaxRel * 4;   // its gradient
  static constexpr int kChange = kDRel + kMaxRel * 4;  // bit t: another bucket than at t - 1
  static constexpr int kBucketAt = kChange + (kMaxRel / 32 + 2) * 4;  // bucket by (k - q), 255: outside the table
  // by t / 16: the bucket of all positions t - 15 .. t + 31, or kMixed
  static constexpr int kFlat = kBucketAt + kMaxRel;
  static constexpr int kBucket = kFlat + (kMaxRel / 16 + 7) / 8 * 8;  // bias gradient by bucket
  static constexpr int kWords = kBucket + kBuckets * 4;  // block flags
  static constexpr int kBars = kWords + 6 * 4;
  static constexpr int kTotal = kBars + 24 * 8 + 1024;
};
static_assert(HeadSmem<false>::kTotal <= 232448 && HeadSmem<true>::kTotal <= 232448, "shared memory of a CTA");
static_assert(HeadSmem<false>::kBars % 8 == 0 && HeadSmem<true>::kBars % 8 == 0, "barriers are 8-byte words");

struct HeadParams {
  AttnParams a;
  const __nv_bfloat16* O;
  const __nv_bfloat16* dO;
  long long o_sb, o_sl, o_sh, do_sb, do_sl, do_sh;
  int ahead;  // CTAs that run at a time
  float *dK32, *dV32;  // kParts: [B, Lk, H, 64], added to
};

// Waits for the loads from TMEM into these registers.
__device__ __forceinline__ void tmem_wait_into(uint32_t (&a)[16], uint32_t (&c)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                 "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15])
               :
               : "memory");
  asm volatile("" : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7]),
                    "+r"(c[8]), "+r"(c[9]), "+r"(c[10]), "+r"(c[11]), "+r"(c[12]), "+r"(c[13]), "+r"(c[14]), "+r"(c[15]));
}

// kAhead: causal self-attention over more than one block, where key blocks ahead of a query block are
// passed over (see attn_bwd_kernel for the conditions).
// kParts: more than 512 queries, a CTA for each 512 of them. dQ leaves as above; dK and dV of the parts are added in
// fp32 memory (two buffers of [B, Lk, H, 64]) and cast afterwards. The parts arrive in any order: up to two of them
// give the same sums whatever it is, of more than 1024 queries dK and dV can differ from run to run in the last
// bits (by key blocks in attention_sm100.cu dQ does). (us, by key blocks / so, with all launches: prefix LM, 16 x 12
// heads x 1024, 591 / 400.)
template <bool kAhead, bool kParts>
__global__ void __launch_bounds__(kThreads, 1)
    attn_bwd_head_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                         const __grid_constant__ CUtensorMap tmDQ, const __grid_constant__ CUtensorMap tmDK,
                         const __grid_constant__ CUtensorMap tmDV, const __grid_constant__ CUtensorMap tmO,
                         const __grid_constant__ HeadParams hp) {
  using HeadSmem = HeadSmem<kParts>;
  constexpr int kMaxRel = HeadSmem::kMaxRel, kRing = HeadSmem::kRing;
  const AttnParams& p = hp.a;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  float* sLse = reinterpret_cast<float*>(smem + HeadSmem::kVec);
  float* sDelta = sLse + kMaxQ;
  int* sQseg = reinterpret_cast<int*>(sDelta + kMaxQ);
  float* sRel = reinterpret_cast<float*>(smem + HeadSmem::kRel);
  float* sDRel = reinterpret_cast<float*>(smem + HeadSmem::kDRel);
  uint32_t* sChange = reinterpret_cast<uint32_t*>(smem + HeadSmem::kChange);
  uint8_t* sBucketAt = smem + HeadSmem::kBucketAt;
  uint8_t* sFlat = smem + HeadSmem::kFlat;
  float* sBucket = reinterpret_cast<float*>(smem + HeadSmem::kBucket);
  uint32_t* sWords = reinterpret_cast<uint32_t*>(smem + HeadSmem::kWords);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + HeadSmem::kBars);
  uint64_t* bar_kv = bars;            // 2: K and V of a key block landed
  uint64_t* bar_staged = bars + 2;    // 2: dK and dV of it have taken their place
  uint64_t* bar_q = bars + 4;         // kRing: Q and dO of a unit landed
  uint64_t* bar_qfree = bars + 7;     // kRing: ... and are no longer read
  uint64_t* bar_s = bars + 10;        // S^T and dP^T of a unit are in TMEM
  uint64_t* bar_sfree = bars + 11;    // ... and in registers
  uint64_t* bar_p = bars + 12;        // 2: P^T and dS^T of a unit are in shared memory
  uint64_t* bar_g = bars + 14;        // 2: the gradient products of a unit are done
  uint64_t* bar_dq = bars + 16;       // dQ of all query blocks is in shared memory
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.x, b = blockIdx.y;
  const int nkb = (p.Lk + 127) / 128;
  // queries count from here (the last part first: of causal attention it has the most keys)
  const int q_base = kParts ? static_cast<int>(gridDim.z - 1 - blockIdx.z) * kMaxQ : 0;
  const int lq = kParts ? min(p.Lq - q_base, kMaxQ) : p.Lq;
  const int lq_pad = (lq + 127) / 128 * 128;
  const int units = (lq + 63) / 64;  // of a key block
  constexpr int cS = 0, cDP = 64, cDQ = 128, cDK = 384, cDV = 448;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&bar_kv[s], 1);
      mbar_init(&bar_staged[s], kSoftmaxWarps);
      mbar_init(&bar_p[s], kSoftmaxWarps);
      mbar_init(&bar_g[s], 1);
    }
    for (int s = 0; s < kRing; ++s) {
      mbar_init(&bar_q[s], 1);
      mbar_init(&bar_qfree[s], 1);
    }
    mbar_init(bar_s, 1);
    mbar_init(bar_sfree, kSoftmaxWarps);
    mbar_init(bar_dq, kSoftmaxWarps);
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (threadIdx.x < 6) sWords[threadIdx.x] = 0u;
  if (warp == kMmaWarp) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (warp == kTmaWarp && lane == 0) {
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  // The softmax warps request what their tables are made of: the buckets of up to three relative
  // positions a thread (and, in a warp's first lane, of the position before), and a query's statistics.
  constexpr int kRelRounds = (kMaxRel + 32 + kSoftmaxThreads - 1) / kSoftmaxThreads;
  const int rels = lq_pad + nkb * 128;  // table index t: k - q = t - lq_pad - q_base
  int bucket[kRelRounds], left[kRelRounds];
  // ... and of rowsum(dO * O): eight lanes a query, the first four of eight rounds of queries.
  constexpr int kRows = kSoftmaxThreads / 8;
  float lse = 0.f;
  int code = 0;
  uint4 xo[4], xd[4];
  const int sub = threadIdx.x & 7;
  const __nv_bfloat16* o_row = hp.O + b * hp.o_sb + q_base * hp.o_sl + h * hp.o_sh + sub * 8;
  const __nv_bfloat16* do_row = hp.dO + b * hp.do_sb + q_base * hp.do_sl + h * hp.do_sh + sub * 8;
  auto request_rows = [&](int q0) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int q = q0 + c * kRows;
      xo[c] = xd[c] = make_uint4(0u, 0u, 0u, 0u);
      if (q < lq) {
        xo[c] = *reinterpret_cast<const uint4*>(o_row + static_cast<long long>(q) * hp.o_sl);
        xd[c] = *reinterpret_cast<const uint4*>(do_row + static_cast<long long>(q) * hp.do_sl);
      }
    }
  };
  if (warp < kSoftmaxWarps) {
    request_rows(threadIdx.x >> 3);
#pragma unroll
    for (int c = 0; c < kRelRounds; ++c) {
      const int t = threadIdx.x + c * kSoftmaxThreads, idx = t - lq_pad - q_base + p.rel_off;
      bucket[c] = left[c] = -1;
      if (p.rel_bias != nullptr && t <= rels) {
        if (t < rels && idx >= 0 && idx < p.nrel) bucket[c] = __ldg(p.rel_bucket + idx);
        if (lane == 0 && t > 0 && idx >= 1 && idx <= p.nrel) left[c] = __ldg(p.rel_bucket + idx - 1);
      }
    }
    const int q = threadIdx.x;
    if (q < lq) {
      lse = p.lse[(static_cast<long long>(b) * p.H + h) * p.Lq + q_base + q];
      if (p.q_seg) code = p.q_seg[static_cast<long long>(b) * p.Lq + q_base + q];
    }
  }
  // Key blocks that a key mask alone hides whole (words[0]: blocks with a visible key), and of causal
  // self-attention the query blocks with a query that does not see itself (words[1]) and the key blocks
  // with a prefix key (words[2]): what may be passed over, as in attn_bwd_kernel.
  const bool look = key_mask_alone(p);
  uint32_t shown = 0u, unseen = 0u, prefix = 0u;
  float lse0 = 0.f;
  if (look) {
    const uint8_t* row = p.key_mask + static_cast<long long>(b) * p.Lk;
    lse0 = p.lse[(static_cast<long long>(b) * p.H + h) * p.Lq];
    for (int k0 = warp * 32; k0 < p.Lk; k0 += kThreads)
      if (__any_sync(0xffffffffu, k0 + lane < p.Lk && row[k0 + lane] != 0)) shown |= 1u << (k0 >> 7);
  }
  if (kAhead) {
    for (int k0 = warp * 32; k0 < p.Lk; k0 += kThreads) {
      const int k = k0 + lane;
      if (__any_sync(0xffffffffu, k < p.Lk && !sees_itself(p, b, k))) unseen |= 1u << (k0 >> 7);
      if (__any_sync(0xffffffffu, k < p.Lk && in_prefix(p, b, k))) prefix |= 1u << (k0 >> 7);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  uint32_t idle = 0u;
  if (look || kAhead) {
    if (lane == 0) {
      if (shown) atomicOr(&sWords[0], shown);
      if (unseen) atomicOr(&sWords[1], unseen);
      if (prefix) atomicOr(&sWords[2], prefix);
    }
    __syncthreads();
    if (look && lse0 >= -5e9f) idle = ~sWords[0];
    unseen = sWords[1];
    prefix = sWords[2];
  }
  // First unit of key block j (of a part's units there may be none).
  auto first_unit = [&](int j) {
    if (!kAhead) return 0;
    const uint32_t before = (1u << j) - 1u;
    return ((unseen & before) | ((prefix >> j) & 1u)) ? 0 : max(0, 2 * j - q_base / 64);
  };
  auto passed_over = [&](int j) {
    return ((idle >> j) & 1u) != 0u || (kAhead && kParts && first_unit(j) >= units);
  };
  const uint32_t tmem_base = *tmem_slot;

  if (warp == kTmaWarp) {
    if (lane == 0) {
      bool ok = true;
      int n = 0, u = 0;      // key blocks and units walked
      int loaded = 0, stored = 0;      // key blocks whose K and V were requested, whose gradients were stored
      int j_load = 0, j_store = 0;     // the next ones
      auto skip = [&](int j) {
        while (j < nkb && passed_over(j)) ++j;
        return j;
      };
      // the gradients of the oldest key block that is still on the chip, from where its K and V were
      auto store_kv = [&]() {
        const int st = stored & 1;
        if (!mbar_wait(&bar_staged[st], (stored >> 1) & 1, abort_flag)) return false;
        j_store = skip(j_store);
        ++stored;
        if (kParts) return true;  // (they have been added to memory)
        tma_store_4d(&tmDK, smem + HeadSmem::kK + st * HeadSmem::kPanel, 0, h, j_store * 128, b);
        tma_store_4d(&tmDV, smem + HeadSmem::kV + st * HeadSmem::kPanel, 0, h, j_store * 128, b);
        bulk_commit();
        ++j_store;
        return true;
      };
      auto load_kv = [&]() {
        j_load = skip(j_load);
        if (j_load >= nkb) return true;
        const int st = loaded & 1;
        if (loaded >= 2) {
          if (!store_kv()) return false;
          bulk_store_wait_read();
        }
        mbar_expect_tx(&bar_kv[st], 2 * HeadSmem::kPanel);
        tma_load_4d(smem + HeadSmem::kK + st * HeadSmem::kPanel, &tmK, &bar_kv[st], 0, h, j_load * 128, b);
        tma_load_4d(smem + HeadSmem::kV + st * HeadSmem::kPanel, &tmV, &bar_kv[st], 0, h, j_load * 128, b);
        ++loaded;
        ++j_load;
        return true;
      };
      for (int j = 0; j < nkb && ok; ++j) {
        if (passed_over(j)) continue;
        if (loaded == n) ok = load_kv();
        const int first = first_unit(j);
        for (int w = first; w < units && ok; ++w, ++u) {
          const int st = u % kRing;
          if (u >= kRing) ok = mbar_wait(&bar_qfree[st], (u / kRing - 1) & 1, abort_flag);
          if (!ok) break;
          mbar_expect_tx(&bar_q[st], 2 * HeadSmem::kHalf);
          tma_load_4d(smem + HeadSmem::kQ + st * HeadSmem::kHalf, &tmQ, &bar_q[st], 0, h, q_base + w * 64, b);
          tma_load_4d(smem + HeadSmem::kDO + st * HeadSmem::kHalf, &tmDO, &bar_q[st], 0, h, q_base + w * 64, b);
          // the next key block, once the operands of this one's first units are under way (its place holds
          // the gradients of the block before until they are stored)
          if (w == min(first + 2, units - 1)) ok = load_kv();
        }
        // What the CTA after this one on the SM (about hp.ahead heads further) starts with goes to L2 now:
        // all SMs load their 320 KB at about the same time, and wait for it.
        if (!kParts && n == 0) {
          const long long head = static_cast<long long>(b) * p.H + h + hp.ahead;
          const int hn = static_cast<int>(head % p.H), bn = static_cast<int>(head / p.H);
          if (bn < p.B) {
            for (int i = 0; i < p.Lq; i += 64) {
              tma_prefetch_4d(&tmO, 0, hn, i, bn);
              tma_prefetch_4d(&tmDO, 0, hn, i, bn);
              tma_prefetch_4d(&tmQ, 0, hn, i, bn);
            }
            tma_prefetch_4d(&tmK, 0, hn, 0, bn);
            tma_prefetch_4d(&tmV, 0, hn, 0, bn);
          }
        }
        ++n;
      }
      while (ok && stored < loaded) ok = store_kv();
      if (ok) ok = mbar_wait(bar_dq, 0, abort_flag);
      if (ok) {
        for (int i = 0; i < lq_pad / 128; ++i)
          tma_store_4d(&tmDQ, smem + HeadSmem::kDS + i * HeadSmem::kPanel, 0, h, q_base + i * 128, b);
        bulk_commit();
      }
      bulk_store_wait_all();
      if (!ok) {
        report_status(p.status, kStatusTimeoutProducer, kKernelId, blockIdx.x, blockIdx.y);
        *abort_flag = 1;
      }
    }
  } else if (warp == kMmaWarp) {
    // The whole warp walks the units and one lane issues: with everything uniform the descriptors stay in
    // uniform registers and an addition apart (in a branch of one lane an MMA took 90 to 120 cycles to
    // issue, twice what it takes to run).
    const bool leader = elect_one();
    bool ok = true;
    const uint32_t idesc_s = make_idesc_bf16(128, 64, 0, 0);   // [keys x queries], K = d
    const uint32_t idesc_kd = make_idesc_bf16(128, 64, 0, 1);  // [keys x d], K = queries
    const uint32_t idesc_qd = make_idesc_bf16(128, 64, 1, 1);  // [queries x d], K = keys
    constexpr uint32_t kP16 = HeadSmem::kPanel >> 4, kH16 = HeadSmem::kHalf >> 4;
    // operands with the contraction contiguous (K S-steps 32 bytes apart), and those read across it
    const uint64_t row_major = make_smem_desc_sw128(smem_u32(smem), 16, 1024);
    const uint64_t col_major = make_smem_desc_sw128(smem_u32(smem), HeadSmem::kPanel, 1024);
    uint32_t started = 0u;  // query blocks whose dQ holds something
    // dV += P^T dO, dK += dS^T Q, and after the last unit of a query block dQ += dS K (whose A operand is
    // the dS^T tiles read with the queries contiguous; the panel of a unit that does not exist adds to
    // rows that nothing reads).
    auto issue_grads = [&](int u, int ring, int kv, int w, bool first, int pair) {
      const uint64_t qd = col_major + (HeadSmem::kQ >> 4) + static_cast<uint32_t>(ring) * kH16;
      const uint64_t dod = col_major + (HeadSmem::kDO >> 4) + static_cast<uint32_t>(ring) * kH16;
      const uint64_t pd = row_major + (HeadSmem::kP >> 4) + static_cast<uint32_t>(u & 1) * kP16;
      const uint64_t dsd = row_major + (HeadSmem::kDS >> 4) + static_cast<uint32_t>(pair * 2 + (w & 1)) * kP16;
      const bool whole = (w & 1) || w == units - 1;
      const int i = w >> 1;
      if (leader) {
#pragma unroll
        for (int s = 0; s < 4; ++s)
          umma_bf16(tmem_base + cDV, pd + 2 * s, dod + 128 * s, idesc_kd, !first || s != 0);
#pragma unroll
        for (int s = 0; s < 4; ++s)
          umma_bf16(tmem_base + cDK, dsd + 2 * s, qd + 128 * s, idesc_kd, !first || s != 0);
        umma_commit(&bar_qfree[ring]);
        if (whole) {
          const uint64_t kd = col_major + (HeadSmem::kK >> 4) + static_cast<uint32_t>(kv) * kP16;
          const uint64_t da = col_major + (HeadSmem::kDS >> 4) + static_cast<uint32_t>(pair * 2) * kP16;
          const bool add = (started >> i) & 1u;
#pragma unroll
          for (int s = 0; s < 8; ++s)
            umma_bf16(tmem_base + cDQ + i * 64, da + 128 * s, kd + 128 * s, idesc_qd, add || s != 0);
        }
        umma_commit(&bar_g[u & 1]);
      }
      if (whole) started |= 1u << i;
    };
    int n = 0, u = 0, pair = 0, ring = 0, ring_phase = 0;
    int prev_ring = 0, prev_kv = 0, prev_w = 0, prev_pair = 0;
    bool prev_first = false;
    for (int j = 0; j < nkb && ok; ++j) {
      if (passed_over(j)) continue;
      const int kv = n & 1;
      ok = mbar_wait(&bar_kv[kv], (n >> 1) & 1, abort_flag);
      const int first = first_unit(j);
      for (int w = first; w < units && ok; ++w) {
        ok = mbar_wait(&bar_q[ring], ring_phase, abort_flag);
        if (ok && u > 0) ok = mbar_wait(bar_sfree, (u - 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint64_t kd = row_major + (HeadSmem::kK >> 4) + static_cast<uint32_t>(kv) * kP16;
        const uint64_t vd = row_major + (HeadSmem::kV >> 4) + static_cast<uint32_t>(kv) * kP16;
        const uint64_t qd = row_major + (HeadSmem::kQ >> 4) + static_cast<uint32_t>(ring) * kH16;
        const uint64_t dod = row_major + (HeadSmem::kDO >> 4) + static_cast<uint32_t>(ring) * kH16;
        if (leader) {
#pragma unroll
          for (int s = 0; s < 4; ++s) umma_bf16(tmem_base + cS, kd + 2 * s, qd + 2 * s, idesc_s, s != 0);
#pragma unroll
          for (int s = 0; s < 4; ++s) umma_bf16(tmem_base + cDP, vd + 2 * s, dod + 2 * s, idesc_s, s != 0);
          umma_commit(bar_s);
        }
        if (u > 0) {
          ok = mbar_wait(&bar_p[(u - 1) & 1], ((u - 1) >> 1) & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          issue_grads(u - 1, prev_ring, prev_kv, prev_w, prev_first, prev_pair);
        }
        prev_ring = ring;
        prev_kv = kv;
        prev_w = w;
        prev_first = w == first;
        prev_pair = pair;
        if ((w & 1) || w == units - 1) pair ^= 1;
        if (++ring == kRing) {
          ring = 0;
          ring_phase ^= 1;
        }
        ++u;
      }
      ++n;
    }
    if (ok && u > 0) {
      ok = mbar_wait(&bar_p[(u - 1) & 1], ((u - 1) >> 1) & 1, abort_flag);
      if (ok) {
        tc_fence_after();
        issue_grads(u - 1, prev_ring, prev_kv, prev_w, prev_first, prev_pair);
      }
    }
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) {
      if (lane == 0) report_status(p.status, kStatusTimeoutMma, kKernelId, blockIdx.x, blockIdx.y);
      *abort_flag = 1;
    }
  } else {
    // ------------------------------ softmax / gradient warps ------------------------------
    const int quarter = warp & 3, part = warp >> 2;  // 32 keys, 16 queries of each unit
    const int r = quarter * 32 + lane;               // key row of the tile == TMEM lane
    const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    const bool has_bias = p.rel_bias != nullptr;
    const bool want_drel = p.d_rel_bias != nullptr;
    bool ok = true;

    if (threadIdx.x < lq_pad) {
      sLse[threadIdx.x] = -lse * kLog2e;
      sQseg[threadIdx.x] = code;
    }
    // words[3], bit g: queries 16 g .. 16 g + 15 all exist, and none of them has all its keys hidden
    const uint32_t good = __ballot_sync(0xffffffffu, threadIdx.x < lq && lse * kLog2e >= -5e9f);
    // words[4], bit g: they have one code
    const uint32_t alike = __ballot_sync(0xffffffffu, code == __shfl_sync(0xffffffffu, code, lane & 16));
    auto both_halves = [&](uint32_t bits) {
      return ((bits & 0xffffu) == 0xffffu ? 1u << (2 * warp) : 0u) | ((bits >> 16) == 0xffffu ? 2u << (2 * warp) : 0u);
    };
    if (lane == 0) {
      atomicOr(&sWords[3], both_halves(good));
      atomicOr(&sWords[4], both_halves(alike));
    }
    if (has_bias) {
      const float* tab = p.rel_bias + static_cast<long long>(h) * p.num_buckets;
      if (threadIdx.x < kBuckets) sBucket[threadIdx.x] = 0.f;
#pragma unroll
      for (int c = 0; c < kRelRounds; ++c) {
        const int t = threadIdx.x + c * kSoftmaxThreads;
        if (t - lane < kMaxRel + 32) {  // (whole warps)
          const int up = __shfl_up_sync(0xffffffffu, bucket[c], 1);
          const uint32_t change = __ballot_sync(0xffffffffu, bucket[c] != (lane == 0 ? left[c] : up));
          if (lane == 0) sChange[t >> 5] = change;
          if (t < kMaxRel) {
            sRel[t] = bucket[c] >= 0 ? __ldg(tab + bucket[c]) : 0.f;
            sDRel[t] = 0.f;
            sBucketAt[t] = static_cast<uint8_t>(bucket[c]);
          }
        }
      }
    }
    for (int q0 = threadIdx.x >> 3; q0 < lq_pad; q0 += 4 * kRows) {
      if (q0 >= 4 * kRows) request_rows(q0);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const __nv_bfloat162* px = reinterpret_cast<const __nv_bfloat162*>(&xo[c]);
        const __nv_bfloat162* py = reinterpret_cast<const __nv_bfloat162*>(&xd[c]);
        float s = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 fx = __bfloat1622float2(px[e]), fy = __bfloat1622float2(py[e]);
          s += fx.x * fy.x + fx.y * fy.y;
        }
        s += __shfl_xor_sync(0xffffffffu, s, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        const int q = q0 + c * kRows;
        if (sub == 0 && q < lq_pad) sDelta[q] = -s;
      }
    }
    softmax_bar_sync();
    if (has_bias && threadIdx.x < kMaxRel / 16) {  // no change of bucket at t - 14 .. t + 31
      const int t = threadIdx.x * 16 - 14;
      bool flat = false;
      if (t > 0 && t + 45 < rels) {
        const uint32_t a = sChange[t >> 5], c = sChange[(t >> 5) + 1], d = sChange[(t >> 5) + 2];
        flat = (__funnelshift_r(a, c, t & 31) | (__funnelshift_r(c, d, t & 31) & 0x3fffu)) == 0u;
      }
      sFlat[threadIdx.x] = flat ? sBucketAt[t + 14] : kMixed;
    }
    softmax_bar_sync();
    const uint32_t counting = sWords[3], one_code = sWords[4];

    // 16 columns of a row of an accumulator, in bf16, into a panel that a tensor copy stores
    auto stage = [&](uint32_t col, uint8_t* panel, bool zero) {
      uint32_t v[16];
      tmem_ld16(t_row + col + part * 16, v);
      tmem_ld_wait();
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const uint32_t* x = v + 8 * g;
        uint4 out;
        out.x = pack_bf16x2(__uint_as_float(x[0]), __uint_as_float(x[1]));
        out.y = pack_bf16x2(__uint_as_float(x[2]), __uint_as_float(x[3]));
        out.z = pack_bf16x2(__uint_as_float(x[4]), __uint_as_float(x[5]));
        out.w = pack_bf16x2(__uint_as_float(x[6]), __uint_as_float(x[7]));
        if (zero) out = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4*>(panel + r * 128 + (((part * 2 + g) ^ (r & 7)) << 4)) = out;
      }
    };
    // kParts: 16 columns of a row are added to memory. Four lanes exchange their 16-byte pieces, so that an
    // instruction adds 64 contiguous bytes of 8 rows.
    auto add_rows = [&](uint32_t col, float* to, int j) {
      uint32_t v[16];
      tmem_ld16(t_row + col + part * 16, v);
      tmem_ld_wait();
      transpose_pieces(v, lane);
      const int k = j * 128 + quarter * 32 + (lane & ~3);
      float* dst = to + ((static_cast<long long>(b) * p.Lk + k) * p.H + h) * 64 + part * 16 + (lane & 3) * 4;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (k + i < p.Lk)
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + i * static_cast<long long>(p.H) * 64),
                       "f"(__uint_as_float(v[4 * i])), "f"(__uint_as_float(v[4 * i + 1])),
                       "f"(__uint_as_float(v[4 * i + 2])), "f"(__uint_as_float(v[4 * i + 3]))
                       : "memory");
    };
    // dK and dV of the n-th key block walked, block j, into the place of its K and V (or to memory)
    auto stage_keys = [&](int n, int j) {
      if (kParts) {
        add_rows(cDK, hp.dK32, j);
        add_rows(cDV, hp.dV32, j);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_staged[n & 1]);
        return;
      }
      stage(cDK, smem + HeadSmem::kK + (n & 1) * HeadSmem::kPanel, false);
      stage(cDV, smem + HeadSmem::kV + (n & 1) * HeadSmem::kPanel, false);
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_staged[n & 1]);
    };
    const bool prefix_lm = p.causal == 2;
    const int seg_mask = prefix_lm ? 0x3fffffff : -1;
    const bool simple_mask = !p.causal && p.kv_seg == nullptr;
    const float inv_lk = 1.f / static_cast<float>(p.Lk);
    const uint64_t log2e2 = pair_of(kLog2e, kLog2e);
    // A block of 32 keys x 16 queries whose relative positions share one bucket takes its bias as one
    // number and leaves its gradient as one sum per thread, kept until another bucket comes.
    float flat_sum = 0.f;
    int flat_bucket = kOutside;
    auto flush_flat = [&]() {
      const float s = warp_sum(flat_sum);
      if (lane == 0 && flat_bucket < kBuckets) atomicAdd(sBucket + flat_bucket, s);
      flat_sum = 0.f;
    };
    auto next_block = [&](int j) {  // the first key block from j on that is walked
      while (j < nkb && passed_over(j)) {
        for (int i = threadIdx.x; !kParts && i < 128 * 8; i += kSoftmaxThreads) {
          const int k = j * 128 + i / 8;
          if (k < p.Lk) {
            const long long off = b * p.dk_sb + static_cast<long long>(k) * p.dk_sl + h * p.dk_sh + i % 8 * 8;
            *reinterpret_cast<uint4*>(p.dK + off) = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4*>(p.dV + off) = make_uint4(0u, 0u, 0u, 0u);
          }
        }
        ++j;
      }
      return j;
    };
    // this thread's key of a block: whether it counts, and its code
    auto request_key = [&](int j, bool& vis, int& code) {
      const int k = j * 128 + r;
      const long long at = static_cast<long long>(b) * p.Lk + k;
      vis = k < p.Lk && (p.key_mask == nullptr || p.key_mask[at] != 0);
      code = (k < p.Lk && p.kv_seg) ? p.kv_seg[at] : 0;
    };
    int u = 0, pair = 0, n = 0;  // units walked, key blocks walked
    int j = next_block(0), w = 0, next_j = nkb, last_j = 0;
    bool kvis = false, next_kvis = false;
    int kcode = 0, next_kcode = 0;
    uint32_t sv[16], dpv[16];
    auto request_scores = [&](int unit) {
      if (!mbar_wait_relaxed(bar_s, unit & 1, abort_flag)) return false;
      tc_fence_after();
      tmem_ld16(t_row + cS + part * 16, sv);
      tmem_ld16(t_row + cDP + part * 16, dpv);
      return true;
    };
    bool all_keys = false;  // of this warp's quarter of the block, all keys count
    auto enter_block = [&]() {
      w = first_unit(j);
      kvis = next_kvis;
      kcode = next_kcode;
      all_keys = __all_sync(0xffffffffu, kvis);
      next_j = next_block(j + 1);
      if (next_j < nkb) request_key(next_j, next_kvis, next_kcode);
    };
    if (j < nkb) {
      request_key(j, next_kvis, next_kcode);
      enter_block();
    }
    while (j < nkb && ok) {
      const int k = j * 128 + r;
      const int first = first_unit(j);
      const int q0 = w * 64 + part * 16;  // this thread's 16 queries
      // which of them see this key
      uint32_t mv = kvis ? 0xffffu : 0u;
      bool all_seen = all_keys;
      if (!simple_mask) {
        // of causal attention the first of them come before the key
        const int hidden = p.causal ? k - p.causal_off - q_base - q0 : 0;
        const uint32_t behind = hidden <= 0 ? 0xffffu : (hidden >= 16 ? 0u : 0xffffu << hidden);
        if (p.kv_seg == nullptr) {
          mv &= behind;
        } else {
          const int kseg = kcode & seg_mask;
          const bool k_pre = prefix_lm && ((kcode >> 30) & 1);
          if ((one_code >> (q0 >> 4)) & 1u) {
            const int code = sQseg[q0];
            mv &= kseg == (code & seg_mask) ? ((k_pre && ((code >> 30) & 1)) ? 0xffffu : behind) : 0u;
          } else {
            uint32_t m = 0u;
#pragma unroll 4
            for (int x = 0; x < 16; ++x) {
              const int code = sQseg[q0 + x];
              const bool v = kseg == (code & seg_mask) && (((behind >> x) & 1u) || (k_pre && ((code >> 30) & 1)));
              m |= (v ? 1u : 0u) << x;
            }
            mv &= m;
          }
        }
        all_seen = __all_sync(0xffffffffu, (mv & 0xffffu) == 0xffffu);
      }
      const bool fast = all_seen && ((counting >> (q0 >> 4)) & 1u);
      // relative positions k - q of the warp's block: table indexes t0 - 15 .. t0 + 31
      const int t0 = j * 128 + quarter * 32 - q0 + lq_pad;
      const int flat = has_bias ? sFlat[t0 >> 4] : kOutside;

      ok = request_scores(u);
      if (!ok) break;
      tmem_wait_into(sv, dpv);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_sfree);

      float ds[16];
      uint32_t pp[8], pd[8];  // P and dS as the MMAs read them
      const float* rel = sRel + t0 + lane;  // rel[-x]
      if (fast) {
        const float one = has_bias ? sRel[t0] : 0.f;
        const uint64_t b0 = pair_of(one, one);
        // kEach: every score has a bias of its own
        auto visible = [&](auto each) {
          constexpr bool kEach = decltype(each)::value;
#pragma unroll
          for (int g = 0; g < 4; ++g) {  // 16-byte broadcast loads of the per-query values
            const ulonglong2 l2 = reinterpret_cast<const ulonglong2*>(sLse + q0)[g];
            const ulonglong2 d2 = reinterpret_cast<const ulonglong2*>(sDelta + q0)[g];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int x = 4 * g + 2 * e;
              uint64_t s = pair_of(__uint_as_float(sv[x]), __uint_as_float(sv[x + 1]));
              s = add2(s, kEach ? pair_of(rel[-x], rel[-x - 1]) : b0);
              s = fma2(s, log2e2, e ? l2.y : l2.x);
              const float p0 = exp2f(low_of(s)), p1 = exp2f(high_of(s));
              uint64_t dp = pair_of(__uint_as_float(dpv[x]), __uint_as_float(dpv[x + 1]));
              dp = mul2(pair_of(p0, p1), add2(dp, e ? d2.y : d2.x));
              ds[x] = low_of(dp);
              ds[x + 1] = high_of(dp);
              pp[x >> 1] = pack_bf16x2(p0, p1);
              pd[x >> 1] = pack_bf16x2(ds[x], ds[x + 1]);
            }
          }
        };
        if (flat == kMixed)
          visible(std::true_type());
        else
          visible(std::false_type());
      } else {
#pragma unroll
        for (int x = 0; x < 16; x += 2) {
          float e2[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int xx = x + c;
            float s = __uint_as_float(sv[xx]);
            if (has_bias) s += rel[-xx];
            s = ((mv >> xx) & 1u) ? s : kMaskValue;
            const float nl = sLse[q0 + xx];
            float e = exp2f(fmaf(s, kLog2e, nl));
            // A row with every key masked has lse = -1e10 + log(Lk), which fp32 rounds to -1e10:
            // its probabilities are uniform over the Lk keys.
            if (nl > 5e9f) e = inv_lk;
            if (k >= p.Lk || q0 + xx >= lq) e = 0.f;
            e2[c] = e;
            ds[xx] = e * (__uint_as_float(dpv[xx]) + sDelta[q0 + xx]);
          }
          pp[x >> 1] = pack_bf16x2(e2[0], e2[1]);
          pd[x >> 1] = pack_bf16x2(ds[x], ds[x + 1]);
        }
      }
      // the products of unit u - 2 read these panels last (and dQ of the query block before the last)
      if (u >= 2) {
        ok = mbar_wait_relaxed(&bar_g[u & 1], ((u >> 1) - 1) & 1, abort_flag);
        if (!ok) break;
      }
      uint8_t* pt = smem + HeadSmem::kP + (u & 1) * HeadSmem::kPanel + r * 128;
      uint8_t* dst = smem + HeadSmem::kDS + (pair * 2 + (w & 1)) * HeadSmem::kPanel + r * 128;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const int at = ((part * 2 + g) ^ (r & 7)) << 4;
        *reinterpret_cast<uint4*>(pt + at) = make_uint4(pp[4 * g], pp[4 * g + 1], pp[4 * g + 2], pp[4 * g + 3]);
        *reinterpret_cast<uint4*>(dst + at) = make_uint4(pd[4 * g], pd[4 * g + 1], pd[4 * g + 2], pd[4 * g + 3]);
      }
      // dK and dV of the key block before: complete with the products of unit u - 1, read before those
      // of this unit may start
      if (w == first && n > 0) {
        ok = mbar_wait_relaxed(&bar_g[(u - 1) & 1], ((u - 1) >> 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        stage_keys(n - 1, last_j);
      }
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_p[u & 1]);

      if ((w & 1) || w == units - 1) pair ^= 1;
      ++u;
      if (++w == units) {
        last_j = j;
        j = next_j;
        ++n;
        if (j < nkb) enter_block();
      }
      if (want_drel) {
        if (flat != kMixed) {
          if (flat != flat_bucket) {
            flush_flat();
            flat_bucket = flat;
          }
          uint64_t s = pair_of(ds[0], ds[1]);
#pragma unroll
          for (int x = 2; x < 16; x += 2) s = add2(s, pair_of(ds[x], ds[x + 1]));
          flat_sum += low_of(s) + high_of(s);
        } else {
          // dS[key r][query c] belongs to position r - c. Lane L collects the diagonals L and L - 32 of
          // the warp's block: at column x it fetches the value of lane (L + x) mod 32.
          float diag_pos[2] = {0.f, 0.f}, diag_neg[2] = {0.f, 0.f};
#pragma unroll
          for (int x = 0; x < 16; ++x) {
            const float v = __shfl_sync(0xffffffffu, ds[x], lane + x);  // (modulo 32)
            if (lane + x < 32) {
              diag_pos[x & 1] += v;
            } else {
              diag_neg[x & 1] += v;
            }
          }
          atomicAdd(sDRel + t0 + lane, diag_pos[0] + diag_pos[1]);
          if (lane > 16) atomicAdd(sDRel + t0 + lane - 32, diag_neg[0] + diag_neg[1]);
        }
      }
    }
    if (ok && u > 0) {
      ok = mbar_wait_relaxed(&bar_g[(u - 1) & 1], ((u - 1) >> 1) & 1, abort_flag);
      if (ok) {
        tc_fence_after();
        stage_keys(n - 1, last_j);
      }
    }
    if (ok) {
      for (int i = 0; i < lq_pad / 128; ++i)
        stage(cDQ + i * 64, smem + HeadSmem::kDS + i * HeadSmem::kPanel, u == 0);
      tc_fence_before();
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_dq);
      if (want_drel) {
        flush_flat();
        softmax_bar_sync();
        // The relative positions are folded into their buckets here. Neighbouring positions share
        // buckets: each run of equal buckets in a warp is summed by shuffles and added once.
        float* out = p.d_rel_bias + static_cast<long long>(h) * p.num_buckets;
        for (int t = threadIdx.x; t < rels; t += kSoftmaxThreads) {  // whole warps
          float g = sDRel[t];
          const int bucket = sBucketAt[t];
          const int prev = __shfl_up_sync(0xffffffffu, bucket, 1);
          const bool head = lane == 0 || prev != bucket;
          const uint32_t heads = __ballot_sync(0xffffffffu, head);
          const uint32_t later = lane == 31 ? 0u : heads >> (lane + 1);
          const int run_end = later ? lane + __ffs(later) : 32;  // first lane of the next run
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float v = __shfl_down_sync(0xffffffffu, g, o);
            if (lane + o < run_end) g += v;
          }
          if (head && bucket < kBuckets && g != 0.f) atomicAdd(sBucket + bucket, g);
        }
        softmax_bar_sync();
        for (int t = threadIdx.x; t < p.num_buckets; t += kSoftmaxThreads)
          if (sBucket[t] != 0.f) atomicAdd(out + t, sBucket[t]);
      }
    } else if (lane == 0) {
      report_status(p.status, kStatusTimeoutEpilogue, kKernelId, blockIdx.x, blockIdx.y);
      *abort_flag = 1;
    }
  }
  if (*abort_flag && threadIdx.x == 0)
    for (int it = 0; it < 2000; ++it) __nanosleep(1000);
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <bool kAhead, bool kParts>
int launch_head(const CUtensorMap* tq, const CUtensorMap* tk, const CUtensorMap* tv, const CUtensorMap* tdo,
                const CUtensorMap* tdq, const CUtensorMap* tdk, const CUtensorMap* tdv, const CUtensorMap* to,
                const HeadParams& hp, cudaStream_t st) {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_bwd_head_kernel<kAhead, kParts>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, HeadSmem<kParts>::kTotal);
    if (e != cudaSuccess) return set_error("attention_bwd_head attr: %s", cudaGetErrorString(e));
    attr_set[dev] = true;
  }
  const dim3 grid(hp.a.H, hp.a.B, (hp.a.Lq + kMaxQ - 1) / kMaxQ);
  attn_bwd_head_kernel<kAhead, kParts><<<grid, kThreads, HeadSmem<kParts>::kTotal, st>>>(*tq, *tk, *tv, *tdo, *tdq,
                                                                                         *tdk, *tdv, *to, hp);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("attention_bwd_head: %s", cudaGetErrorString(e));
  return 0;
}
}  // namespace
}  // namespace t5x

using namespace t5x;

// Whether t5x_attention_bwd_head takes these sizes and is the faster of the two backward kernels: 0, or 1 as it
// stands, or 2 with fp32 buffers for dK and dV.
T5X_API int t5x_attention_bwd_head_covers(int B, int H, int Lq, int Lk, int D, int num_buckets) {
  if (D != 64 || B <= 0 || B > 65535 || H <= 0 || Lq <= 0 || Lq > 8 * kMaxQ || Lk <= 0 || Lk > kMaxKeys) return 0;
  const int nkb = (Lk + 127) / 128, nq = (Lq + 127) / 128, parts = (Lq + kMaxQ - 1) / kMaxQ;
  if (num_buckets > 0 && (num_buckets > kBuckets || (nkb + (nq < 4 ? nq : 4)) * 128 >
                                                        (parts > 1 ? kMaxRelOf<true> : kMaxRelOf<false>)))
    return 0;
  // Thousands of cycles, measured: 14 for a CTA and 3 for each of its 128 x 64 units, 2.2 without a bias (of parts 2.9
  // and 2.7); the other kernel, with a CTA per key block, 14 and 7.2 for each 128 x 128 tile, 5.2 without a bias;
  // some 10 for its three further launches or for those of parts; clearing and casting dQ (there) or the dK and dV of
  // parts (here), ten bytes an element at 3.4 MB a thousand cycles. Up to a head per SM the last part, which has
  // fewer units, makes room for a whole one. (us, other / this, with a bias and without: 512 x 512, 48 heads 53 / 55
  // and 41 / 43, 96 heads 78 / 55, 60 / 43; 1024 x 1024, 48 heads 124 / 116, 91 / 106, 148 heads 333 / 250, 247 /
  // 231, 300 heads 694 / 601, 513 / 555; 600 x 600, 144 heads 152 / 125, 122 / 113; 1100 x 300, 6 heads 50 / 54,
  // 42 / 45.)
  const bool bias = num_buckets > 0;
  const long long sms = num_sms(), heads = static_cast<long long>(B) * H;
  const double cast = heads * 640.0 / 3.4e6;
  auto cta = [&](int queries) {
    return 14 + (parts > 1 ? (bias ? 2.9 : 2.7) : (bias ? 3 : 2.2)) * nkb * ((queries + 63) / 64);
  };
  const double whole = cta(Lq < kMaxQ ? Lq : kMaxQ);
  double here = static_cast<double>((heads * parts + sms - 1) / sms) * whole;
  if (heads <= sms) here = std::min(here, (parts - 1) * whole + cta(Lq - (parts - 1) * kMaxQ));
  if (parts > 1) here += 10 + 2 * Lk * cast;
  const double other =
      static_cast<double>((heads * nkb + sms - 1) / sms) * (14 + (bias ? 7.2 : 5.2) * nq) + 10 + Lq * cast;
  if (here > other) return 0;
  return parts > 1 ? 2 : 1;
}

// q [B,Lq,H,64], k/v [B,Lk,H,64], o and d_o like q, bf16 with element strides (sb, sl, sh), innermost
// contiguous; dq, dk and dv (the strides of dk) are written whole, in bf16; of more than 512 queries, dk32 and dv32
// (fp32, [B,Lk,H,64], cleared) are added to instead of dk and dv. The rest as t5x_attention_bwd.
T5X_API int t5x_attention_bwd_head(const void* q, const void* k, const void* v, const void* o, const void* d_o,
                                   const void* lse, void* dq, void* dk, void* dv, void* dk32, void* dv32, int B,
                                   int H, int Lq, int Lk, long long q_sb, long long q_sl, long long q_sh,
                                   long long k_sb, long long k_sl, long long k_sh, long long v_sb,
                                   long long v_sl, long long v_sh, long long o_sb, long long o_sl, long long o_sh,
                                   long long do_sb, long long do_sl, long long do_sh, long long dq_sb,
                                   long long dq_sl, long long dq_sh, long long dk_sb, long long dk_sl,
                                   long long dk_sh, const void* rel_bias, const void* rel_bucket,
                                   void* d_rel_bias, int num_buckets, int nrel, int rel_off,
                                   const void* key_mask, const void* q_seg, const void* kv_seg, int causal,
                                   int causal_off, void* stream) {
  if (B <= 0 || H <= 0 || Lq <= 0 || Lk <= 0) return 0;
  const int nkb = (Lk + 127) / 128, nq = (Lq + 127) / 128;
  const bool parts = Lq > kMaxQ;
  if (Lq > 8 * kMaxQ || Lk > kMaxKeys || B > 65535)
    return set_error("attention_bwd_head: %d examples of %d queries and %d keys are not covered", B, Lq, Lk);
  if (rel_bias != nullptr && (num_buckets > kBuckets || (nkb + (nq < 4 ? nq : 4)) * 128 >
                                                            (parts ? kMaxRelOf<true> : kMaxRelOf<false>)))
    return set_error("attention_bwd_head: %d buckets over %d + %d positions are not covered", num_buckets, Lq, Lk);
  if (parts && (dk32 == nullptr || dv32 == nullptr || !aligned_to(16, {dk32, dv32})))
    return set_error("attention_bwd_head: more than %d queries need fp32 buffers for dK and dV", kMaxQ);
  if ((do_sb | do_sl | do_sh | o_sb | o_sl | o_sh | dq_sb | dq_sl | dq_sh | dk_sb | dk_sl | dk_sh) & 7)
    return set_error("attention_bwd_head: dO / O / dQ / dK strides must be multiples of 8 elements");
  if (!aligned_to(16, {o, d_o, dq, dk, dv}))
    return set_error("attention_bwd_head: O, dO and the gradients must be 16-byte aligned");
  CUtensorMap tq, tk, tv, tdo, tdq, tdk, tdv, to;
  if (!bhld_map(&tq, q, B, Lq, H, q_sb, q_sl, q_sh, 64, 64) || !bhld_map(&tk, k, B, Lk, H, k_sb, k_sl, k_sh) ||
      !bhld_map(&tv, v, B, Lk, H, v_sb, v_sl, v_sh) || !bhld_map(&tdo, d_o, B, Lq, H, do_sb, do_sl, do_sh, 64, 64) ||
      !bhld_map(&to, o, B, Lq, H, o_sb, o_sl, o_sh, 64, 64) ||
      !bhld_map(&tdq, dq, B, Lq, H, dq_sb, dq_sl, dq_sh) || !bhld_map(&tdk, dk, B, Lk, H, dk_sb, dk_sl, dk_sh) ||
      !bhld_map(&tdv, dv, B, Lk, H, dk_sb, dk_sl, dk_sh))
    return -1;
  HeadParams hp = {};
  AttnParams& p = hp.a;
  p.B = B; p.H = H; p.Lq = Lq; p.Lk = Lk;
  p.rel_bias = static_cast<const float*>(rel_bias);
  p.rel_bucket = static_cast<const int*>(rel_bucket);
  p.num_buckets = num_buckets;
  p.d_rel_bias = rel_bias != nullptr ? static_cast<float*>(d_rel_bias) : nullptr;
  p.nrel = nrel; p.rel_off = rel_off;
  p.key_mask = static_cast<const uint8_t*>(key_mask);
  p.q_seg = static_cast<const int*>(q_seg);
  p.kv_seg = static_cast<const int*>(kv_seg);
  p.causal = causal; p.causal_off = causal_off;
  p.lse = const_cast<float*>(static_cast<const float*>(lse));
  p.dK = static_cast<__nv_bfloat16*>(dk);
  p.dV = static_cast<__nv_bfloat16*>(dv);
  p.dk_sb = dk_sb; p.dk_sl = dk_sl; p.dk_sh = dk_sh;
  p.status = device_status_buffer();
  hp.O = static_cast<const __nv_bfloat16*>(o);
  hp.dO = static_cast<const __nv_bfloat16*>(d_o);
  hp.o_sb = o_sb; hp.o_sl = o_sl; hp.o_sh = o_sh;
  hp.do_sb = do_sb; hp.do_sl = do_sl; hp.do_sh = do_sh;
  hp.ahead = num_sms();
  hp.dK32 = static_cast<float*>(dk32);
  hp.dV32 = static_cast<float*>(dv32);
  const bool ahead = causal && Lq == Lk && causal_off == 0 && Lq > 128;
  const auto launch = parts ? (ahead ? launch_head<true, true> : launch_head<false, true>)
                            : (ahead ? launch_head<true, false> : launch_head<false, false>);
  return launch(&tq, &tk, &tv, &tdo, &tdq, &tdk, &tdv, &to, hp, static_cast<cudaStream_t>(stream));
}
