// Declarations shared by the attention kernels: forward, attention_fwd_rows_sm100.cu (64 channels, up to 2048
// keys), attention_fwd_few_sm100.cu (the same for few heads and up to 512) and attention_fwd_sm100.cu (any
// length, 64 or 128 channels); backward, attention_bwd_head_sm100.cu (64
// channels, where there are heads enough) and attention_sm100.cu.
#pragma once
#include "common.cuh"

namespace t5x {

constexpr int kAttnD = 64;
constexpr int kSoftmaxWarps = 16;
constexpr int kSoftmaxThreads = kSoftmaxWarps * 32;
constexpr int kAttnThreads = kSoftmaxThreads + 32;  // + 1 warp: TMA + MMA issue, TMEM owner
constexpr int kCtrlWarp = kSoftmaxWarps;
constexpr int kKernelIdAttnFwd = 2;
constexpr int kKernelIdAttnBwd = 3;
constexpr float kMaskValue = -1e10f;
constexpr float kLog2e = 1.4426950408889634f;

struct AttnParams {
  int B, H, Lq, Lk;
  const float* rel_bias;     // [H, num_buckets] or null: the T5 bucket table
  const int* rel_bucket;     // [nrel]: bucket of the relative position (k - q) = t - rel_off
  int nrel, rel_off, num_buckets;
  const uint8_t* key_mask;  // [B, Lk] (1 = attend) or null
  const int* q_seg;         // [B, Lq] or null
  const int* kv_seg;        // [B, Lk] or null
  int causal, causal_off;
  __nv_bfloat16* O;         // forward output [B, Lq, H, D]
  long long o_sb, o_sl, o_sh;
  float* lse;               // [B, H, Lq]
  // backward
  const float* delta;       // [B, H, Lq] rowsum(dO * O)
  float* dQ;                // fp32 [B, Lq, H, D] (contiguous), accumulated atomically
  __nv_bfloat16* dK;        // [B, Lk, H, D]
  __nv_bfloat16* dV;
  long long dk_sb, dk_sl, dk_sh;
  float* d_rel_bias;        // [H, num_buckets] (added to) or null
  int* status;
};

// The bias of head h at relative index t = (k - q) + rel_off (0 outside the table).
__device__ __forceinline__ float rel_bias_at(const AttnParams& p, const float* head_table, int t) {
  return (t >= 0 && t < p.nrel) ? __ldg(head_table + __ldg(p.rel_bucket + t)) : 0.f;
}

__device__ __forceinline__ void softmax_bar_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kSoftmaxThreads) : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&p);
}

// Key blocks that the streaming forward kernel walks. Blocks that a mask hides whole from all of a
// tile's queries would contribute exact zeros (the scores of visible keys being far above the -1e10 of
// hidden ones), unless a query sees no key at all: its row is uniform over all keys, and all count.
//   kLookMask    Nothing but a key mask hides keys (the padding of a batch): up to the last visible key.
//                us before / so, 8 x 32 heads of 128 features x 1024 x 1024: 60 to 100 % of the keys visible
//                643 / 562; all visible 643 / 643.
//   kLookCausal  A causal or prefix-LM mask of self-attention with a key mask or segments: up to a tile's
//                last query (and the last prefix key, if the tile has queries inside the prefix), as long
//                as each of its queries sees itself. To look that up costs a CTA some 3 us, so only from
//                more than kAheadKeys keys on (causal with a key mask, 8 x 32 heads of 128 x 1024 655 / 472;
//                but without that bound 8 x 32 x 256 72 / 77).
//   kLookNone    Everything else, in a variant of its own: the look-up at run time cost it 2 to 5 % (8 x 32
//                heads of 128 x 256, causal, 61.4 / 64.3).
enum KeyLook : int { kLookNone = 0, kLookMask = 1, kLookCausal = 2 };
__host__ __device__ __forceinline__ bool key_mask_alone(const AttnParams& p) {
  return p.key_mask != nullptr && !p.causal && p.kv_seg == nullptr;
}
constexpr int kAheadKeys = 512;
inline KeyLook key_look(const AttnParams& p) {
  if (key_mask_alone(p)) return kLookMask;
  // (causal alone: the last query gives the number of blocks, see the kernel)
  const bool self = p.causal && p.Lq == p.Lk && p.causal_off == 0 && p.Lk > kAheadKeys;
  return self && (p.key_mask != nullptr || p.kv_seg != nullptr) ? kLookCausal : kLookNone;
}
__device__ __forceinline__ bool sees_itself(const AttnParams& p, int b, int q) {
  const long long at = static_cast<long long>(b) * p.Lk + q;
  const int mask = p.causal == 2 ? 0x3fffffff : -1;
  return (p.key_mask == nullptr || p.key_mask[at] != 0) &&
         (p.kv_seg == nullptr || (p.q_seg != nullptr && ((p.q_seg[at] ^ p.kv_seg[at]) & mask) == 0));
}
__device__ __forceinline__ bool in_prefix(const AttnParams& p, int b, int k) {
  return p.causal == 2 && p.kv_seg != nullptr && ((p.kv_seg[static_cast<long long>(b) * p.Lk + k] >> 30) & 1);
}
constexpr int kAllKeys = 0x7fffffff;
// A thread's first 16 bytes of the key mask, requested as the kernel starts, so that they arrive while the
// barriers and the tensor memory are set up.
struct MaskAhead {
  uint4 bytes;
  bool vec;  // the example's mask may be read 16 bytes at a time
};
__device__ __forceinline__ MaskAhead request_key_mask(const AttnParams& p, int b) {
  MaskAhead m = {make_uint4(0u, 0u, 0u, 0u), false};
  const uint8_t* row = p.key_mask + static_cast<long long>(b) * p.Lk;
  m.vec = p.Lk % 16 == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0;
  if (m.vec && static_cast<int>(threadIdx.x) * 16 < p.Lk)
    m.bytes = reinterpret_cast<const uint4*>(row)[threadIdx.x];
  return m;
}
__device__ __forceinline__ int last_nonzero_byte(const uint4& u) {  // 0 .. 15, -1: none
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
  int at = -1;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (w[i] != 0u) at = 4 * i + (31 - __clz(w[i])) / 8;
  return at;
}
// `find_*` leave two words per warp: the last key that counts, and whether the tile has prefix queries. A
// __syncthreads later `visible_key_blocks` gives the number of blocks.
__device__ __forceinline__ void leave_words(int last, int pre, int* words) {
  last = __reduce_max_sync(0xffffffffu, last);
  pre = __reduce_max_sync(0xffffffffu, pre);
  if ((threadIdx.x & 31) == 0) {
    words[(threadIdx.x >> 5) * 2] = last;
    words[(threadIdx.x >> 5) * 2 + 1] = pre;
  }
}
__device__ __forceinline__ void find_in_mask(const AttnParams& p, const MaskAhead& ahead, int b, int* words) {
  const uint8_t* row = p.key_mask + static_cast<long long>(b) * p.Lk;
  int last = -1;
  if (ahead.vec) {
    uint4 u = ahead.bytes;
    for (int k = threadIdx.x * 16; k < p.Lk; k += blockDim.x * 16) {
      if (k != static_cast<int>(threadIdx.x) * 16) u = *reinterpret_cast<const uint4*>(row + k);
      const int at = last_nonzero_byte(u);
      if (at >= 0) last = k + at;
    }
  } else {
    for (int k = threadIdx.x; k < p.Lk; k += blockDim.x)
      if (row[k]) last = k;
  }
  leave_words(last, 0, words);
}
__device__ __forceinline__ void find_ahead(const AttnParams& p, int b, int q_base, int q_end, int* words) {
  int last = -1, pre = 0;
  for (int k = threadIdx.x; k < p.Lk; k += blockDim.x) {
    if (in_prefix(p, b, k)) {
      last = max(last, k);
      if (k >= q_base && k < q_end) pre = 1;
    }
    if (k >= q_base && k < q_end && !sees_itself(p, b, k)) last = kAllKeys;
  }
  leave_words(last, pre, words);
}
template <int kLook>
__device__ __forceinline__ int visible_key_blocks(const AttnParams& p, int q_end, const int* words, int warps) {
  const int all = (p.Lk + 127) / 128;
  int last = -1, pre = 0;
  for (int w = 0; w < warps; ++w) {
    last = max(last, words[2 * w]);
    pre |= words[2 * w + 1];
  }
  if (kLook == kLookMask) return last < 0 ? all : last / 128 + 1;
  if (last == kAllKeys) return all;
  return min(all, max(q_end - 1, pre ? last : -1) / 128 + 1);
}

// Writes 8 consecutive bf16 (one 16-byte chunk) of row r, chunk c (0..7) of a [128 x 64] K-major
// 128B-swizzled tile.
__device__ __forceinline__ void store_swizzled_chunk(uint8_t* tile, int r, int c, const float* v) {
  uint4 u;
  u.x = pack_bf16x2(v[0], v[1]);
  u.y = pack_bf16x2(v[2], v[3]);
  u.z = pack_bf16x2(v[4], v[5]);
  u.w = pack_bf16x2(v[6], v[7]);
  *reinterpret_cast<uint4*>(tile + r * 128 + ((c ^ (r & 7)) << 4)) = u;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

// 16 fp32 values -> 16 bf16 written as two 16-byte stores.
__device__ __forceinline__ void store16_bf16(__nv_bfloat16* dst, const uint32_t (&v)[16], float scale) {
  uint4 u0, u1;
  u0.x = pack_bf16x2(__uint_as_float(v[0]) * scale, __uint_as_float(v[1]) * scale);
  u0.y = pack_bf16x2(__uint_as_float(v[2]) * scale, __uint_as_float(v[3]) * scale);
  u0.z = pack_bf16x2(__uint_as_float(v[4]) * scale, __uint_as_float(v[5]) * scale);
  u0.w = pack_bf16x2(__uint_as_float(v[6]) * scale, __uint_as_float(v[7]) * scale);
  u1.x = pack_bf16x2(__uint_as_float(v[8]) * scale, __uint_as_float(v[9]) * scale);
  u1.y = pack_bf16x2(__uint_as_float(v[10]) * scale, __uint_as_float(v[11]) * scale);
  u1.z = pack_bf16x2(__uint_as_float(v[12]) * scale, __uint_as_float(v[13]) * scale);
  u1.w = pack_bf16x2(__uint_as_float(v[14]) * scale, __uint_as_float(v[15]) * scale);
  reinterpret_cast<uint4*>(dst)[0] = u0;
  reinterpret_cast<uint4*>(dst)[1] = u1;
}


// Two fp32 values in one register pair and the arithmetic on both at once (each rounded as by itself).
__device__ __forceinline__ uint64_t pair_of(float a, float b) {
  return static_cast<uint64_t>(__float_as_uint(a)) | (static_cast<uint64_t>(__float_as_uint(b)) << 32);
}
__device__ __forceinline__ float low_of(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float high_of(uint64_t v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
      :
      : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}

// The 4 x 4 transpose of 16-byte pieces among four adjacent lanes: lane j brings pieces 0..3 of its
// row and leaves with piece j of the four rows, in order of the lanes.
__device__ __forceinline__ void transpose_pieces(uint32_t* v, int lane) {
  const bool odd = lane & 1, high = lane & 2;
#pragma unroll
  for (int c = 0; c < 16; c += 8)
#pragma unroll
    for (int e = 0; e < 4; ++e) {  // pieces c / 4 and c / 4 + 1 with the neighbour
      const uint32_t a = v[c + e], b = v[c + 4 + e];
      const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
      v[c + e] = odd ? got : a;
      v[c + 4 + e] = odd ? b : got;
    }
#pragma unroll
  for (int c = 0; c < 8; ++c) {  // the pairs with the lane two away
    const uint32_t a = v[c], b = v[c + 8];
    const uint32_t got = __shfl_xor_sync(0xffffffffu, high ? a : b, 2);
    v[c] = high ? got : a;
    v[c + 8] = high ? b : got;
  }
}

// Tensor map over a [B, L, H, D] bf16 tensor with element strides (sb, sl, sh): boxes of
// 64 channels x 128 (or `rows`) positions of one head (one 128-byte-swizzled shared-memory panel).
inline bool bhld_map(CUtensorMap* map, const void* ptr, int B, int L, int H, long long sb, long long sl,
                     long long sh, int D = kAttnD, uint32_t rows = 128) {
  uint64_t dims[4] = {static_cast<uint64_t>(D), static_cast<uint64_t>(H),
                      static_cast<uint64_t>(L), static_cast<uint64_t>(B)};
  uint64_t strides[3] = {static_cast<uint64_t>(sh) * 2, static_cast<uint64_t>(sl) * 2,
                         static_cast<uint64_t>(sb) * 2};
  uint32_t box[4] = {64, 1, rows, 1};
  return get_tensor_map(map, ptr, 2, 4, dims, strides, box, 1);
}

}  // namespace t5x
