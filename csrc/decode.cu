// Attention kernels of the autoregressive decode step (one new token per row).
//
// decode_self_attention: each (batch, beam) row attends over that beam's key/value history.
// The cache is written once per step and never reordered: row (b, j) stores the key/value it
// computed at position t in cache[b][j][t], and `ancestry[b][j][t]` names the slot that holds
// beam j's key/value for position t (beam search rewrites the small ancestry table when beams
// are reselected, instead of gathering every layer's cache). Fused in one launch: the cache
// write of the new key/value, the T5 relative-position bias (a [heads, max_len] row prepared
// once per step), the softmax and the value sum. One warp per (row, head).
//
// decode_cross_attention: the `beams` rows of one example attend over that example's encoder
// keys/values, stored once per example. One CTA per (example, head): every key / value row is
// read once and used for all beams.
//
// Memory layout of the work, both kernels (head_dim = 64, bf16): 8 adjacent lanes read one
// 128-byte key or value row with one 16-byte load each, so a warp instruction fetches four
// rows; partial dot products are combined with three shuffles, partial value sums with two.
#include "common.cuh"
#include "t5x_b200.h"

namespace t5x {

constexpr int kDecHeadDim = 64;
constexpr int kDecWarps = 4;
constexpr int kDecMaxLen = 1024;  // probabilities of one row are staged in shared memory

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* p2 = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 t = __bfloat1622float2(p2[e]);
    f[2 * e] = t.x;
    f[2 * e + 1] = t.y;
  }
}
__device__ __forceinline__ float sum_over_row_lanes(float x) {  // the 8 lanes of one row
  x += __shfl_xor_sync(0xffffffffu, x, 1);
  x += __shfl_xor_sync(0xffffffffu, x, 2);
  x += __shfl_xor_sync(0xffffffffu, x, 4);
  return x;
}
__device__ __forceinline__ float sum_over_row_groups(float x) {  // the 4 row groups of a warp
  x += __shfl_xor_sync(0xffffffffu, x, 8);
  x += __shfl_xor_sync(0xffffffffu, x, 16);
  return x;
}

// kFirst: positions per lane group whose key and value are held in registers (see below). kChained:
// inside a chain of launches, where the inputs come from kernels that may still be running; by itself
// otherwise, where everything is read at once and through L1. (One body with the choice at run time
// cost the form by itself 7 %: us, one body / two, 256 rows x 32 heads at position 64 of 129 49.2 / 45.9,
// at 127 79.9 / 73.7, 64 x 32 at 100 30.7 / 28.7; beam search of XL, 24 layers, 128 steps 589 / 579 ms.)
template <int kFirst, bool kChained>
__global__ void __launch_bounds__(kDecWarps * 32)
    decode_self_attention_kernel(const __nv_bfloat16* __restrict__ q,      // [rows, H, 64]
                                 const __nv_bfloat16* __restrict__ k_new,  // [rows, H, 64]
                                 const __nv_bfloat16* __restrict__ v_new,
                                 __nv_bfloat16* __restrict__ cache_k,  // [B, beams, H, L, 64]
                                 __nv_bfloat16* __restrict__ cache_v,
                                 const int* __restrict__ ancestry,     // [B, beams, L]
                                 const float* __restrict__ bias_row,   // [H, L] or null
                                 const int* __restrict__ cur_index,    // device scalar
                                 __nv_bfloat16* __restrict__ out,      // [rows, H, 64]
                                 long long in_ld,  // row stride of q / k_new / v_new (elements)
                                 int rows, int beams, int H, int L) {
  __shared__ float sprob[kDecWarps][kDecMaxLen];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int item = blockIdx.x * kDecWarps + warp;  // (row, head)
  if (kChained) chain_release();
  if (item >= rows * H) {
    if (kChained) chain_wait();
    return;
  }
  const int row = item / H, h = item - row * H;
  const int b = row / beams;
  const int g = lane >> 3, part = lane & 7;
  const long long rh = static_cast<long long>(row) * in_ld + h * kDecHeadDim;  // inputs
  const long long oh = (static_cast<long long>(row) * H + h) * kDecHeadDim;   // output
  // cache layout [B, beams, H, L, 64]: the history of one (slot, head) is contiguous
  const long long tstride = kDecHeadDim;
  const long long slot_stride = static_cast<long long>(H) * L * kDecHeadDim;
  const long long batch_base = static_cast<long long>(b) * beams * slot_stride +
                               static_cast<long long>(h) * L * kDecHeadDim;
  const int* anc = ancestry + static_cast<long long>(row) * L;

  // With few (row, head) items the kernel is a chain of dependent loads, so with kFirst = 8 it is kept
  // to two links: the position, the slots of the first 32 positions and (not chained) this step's
  // vectors together, then the keys AND values of those positions. Chained, both links come ahead of
  // the wait for the preceding kernel: the history is from before this chain of launches, which
  // decode_begin starts; q / k / v and the bias come from it. Later positions are streamed below, and
  // with kFirst = 0 all are.
  constexpr int kU = 4;  // positions in flight per lane group in the streams
  constexpr int kHeld = kFirst > 0 ? kFirst : 1;
  auto input = [&](const __nv_bfloat16* x) {  // 8 dims per lane
    const uint4* at = reinterpret_cast<const uint4*>(x + rh) + part;
    return kChained ? ld_chained(at) : *at;
  };
  auto bias_at = [&](int t) {  // (by itself the lines stay in L1 for the many rows of a head)
    const float* at = bias_row + static_cast<long long>(h) * L + t;
    return kChained ? ld_chained(at) : *at;
  };
  int slot[kHeld];
#pragma unroll
  for (int u = 0; u < kFirst; ++u) {
    const int t = u * 4 + g;
    slot[u] = t < L ? anc[t] : 0;
  }
  const int cur = min(max(*cur_index, 0), L - 1);
  // 1. this step's query / key / value; append key / value at position `cur` of the row's own slot
  uint4 qu, kn, vn;
  if (!kChained) qu = input(q), kn = input(k_new), vn = input(v_new);
  uint4 kf4[kHeld], vf4[kHeld];
  float bf[kHeld];
#pragma unroll
  for (int u = 0; u < kFirst; ++u) {
    const int t = u * 4 + g;
    if (!kChained) {
      kf4[u] = kn;
      vf4[u] = vn;
      bf[u] = 0.f;
    }
    if (t < cur) {
      const long long at = batch_base + slot[u] * slot_stride + t * tstride;
      kf4[u] = reinterpret_cast<const uint4*>(cache_k + at)[part];
      vf4[u] = reinterpret_cast<const uint4*>(cache_v + at)[part];
    }
    if (!kChained && bias_row != nullptr && t <= cur) bf[u] = bias_at(t);
  }
  if (kChained) {
    chain_wait();
    qu = input(q), kn = input(k_new), vn = input(v_new);
#pragma unroll
    for (int u = 0; u < kFirst; ++u) {
      const int t = u * 4 + g;
      if (t >= cur) {
        kf4[u] = kn;
        vf4[u] = vn;
      }
      bf[u] = 0.f;
      if (bias_row != nullptr && t <= cur) bf[u] = bias_at(t);
    }
  }
  if (g == 0) {
    const long long dst = batch_base + (row - b * beams) * slot_stride + cur * tstride;
    reinterpret_cast<uint4*>(cache_k + dst)[part] = kn;
    reinterpret_cast<uint4*>(cache_v + dst)[part] = vn;
  }
  float qf[8];
  unpack8(qu, qf);
  auto dot = [&](const uint4& u) {
    float kf[8];
    unpack8(u, kf);
    float s = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) s = fmaf(qf[e], kf[e], s);
    return sum_over_row_lanes(s);
  };

  // 2. scores over positions 0..cur (no 1/sqrt(d): T5 folds it into the query init)
  float mx = -INFINITY;
#pragma unroll
  for (int u = 0; u < kFirst; ++u) {
    const int t = u * 4 + g;
    const float s = dot(kf4[u]) + bf[u];
    if (t <= cur) {
      if (part == 0) sprob[warp][t] = s;
      mx = fmaxf(mx, s);
    }
  }
  for (int t0 = 4 * kFirst; t0 <= cur; t0 += 4 * kU) {
    uint4 ku[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int t = t0 + u * 4 + g;
      ku[u] = kn;
      if (t < cur)
        ku[u] = reinterpret_cast<const uint4*>(cache_k + batch_base + anc[t] * slot_stride +
                                               t * tstride)[part];
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int t = t0 + u * 4 + g;
      float s = dot(ku[u]);
      if (t <= cur) {
        if (bias_row != nullptr) s += bias_at(t);
        if (part == 0) sprob[warp][t] = s;
        mx = fmaxf(mx, s);
      }
    }
  }
  mx = warp_max(mx);
  __syncwarp();
  float sum = 0.f;
  for (int t = lane; t <= cur; t += 32) {
    const float e = __expf(sprob[warp][t] - mx);
    sprob[warp][t] = e;
    sum += e;
  }
  sum = warp_sum(sum);
  __syncwarp();

  // 3. out = sum_t p_t * V[t]; lane accumulates its 8 dims over its row group's positions
  float acc[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = 0.f;
#pragma unroll
  for (int u = 0; u < kFirst; ++u) {
    const int t = u * 4 + g;
    if (t <= cur) {
      const float pt = sprob[warp][t];
      float vf[8];
      unpack8(vf4[u], vf);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = fmaf(pt, vf[e], acc[e]);
    }
  }
  for (int t0 = 4 * kFirst; t0 <= cur; t0 += 4 * kU) {
    uint4 vu[kU];
    float pt[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int t = t0 + u * 4 + g;
      pt[u] = 0.f;
      vu[u] = vn;
      if (t <= cur) {
        pt[u] = sprob[warp][t];
        if (t < cur)
          vu[u] = reinterpret_cast<const uint4*>(cache_v + batch_base + anc[t] * slot_stride +
                                                 t * tstride)[part];
      }
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      float vf[8];
      unpack8(vu[u], vf);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] = fmaf(pt[u], vf[e], acc[e]);
    }
  }
  const float inv = 1.f / sum;
#pragma unroll
  for (int e = 0; e < 8; ++e) acc[e] = sum_over_row_groups(acc[e]) * inv;
  if (g == 0) {
    uint4 o;
    __nv_bfloat162 p0 = __floats2bfloat162_rn(acc[0], acc[1]);
    __nv_bfloat162 p1 = __floats2bfloat162_rn(acc[2], acc[3]);
    __nv_bfloat162 p2 = __floats2bfloat162_rn(acc[4], acc[5]);
    __nv_bfloat162 p3 = __floats2bfloat162_rn(acc[6], acc[7]);
    o.x = *reinterpret_cast<uint32_t*>(&p0);
    o.y = *reinterpret_cast<uint32_t*>(&p1);
    o.z = *reinterpret_cast<uint32_t*>(&p2);
    o.w = *reinterpret_cast<uint32_t*>(&p3);
    reinterpret_cast<uint4*>(out + oh)[part] = o;
  }
}

// First kernel of a decode step: looks up the embedding row of every live row's token at the
// current position and lays out the T5 bias of that position, bias_row[h][t] =
// table[h][bucket_of_distance[cur - t]] for t <= cur (bucket 0 beyond it, as for any key not
// before its query). One block per row, then one per head. As tensor operations this was some
// sixteen launches of 2 us each per step. It is launched the ordinary way, so that a step starts a
// chain of its own: what earlier steps and the beam kernels wrote (position, ancestry, caches) is
// complete and visible before any kernel of the step runs, and those may read it ahead of their wait.
constexpr int kBeginThreads = 128;
__global__ void __launch_bounds__(kBeginThreads)
    decode_begin_kernel(const long long* __restrict__ live_seqs,  // [rows, L]
                        const int* __restrict__ cur_index, const __nv_bfloat16* __restrict__ emb,
                        __nv_bfloat16* __restrict__ x, const float* __restrict__ table,
                        const int* __restrict__ bucket_of_distance, float* __restrict__ bias_row,
                        int rows, int L, int d, int vocab, int num_buckets) {
  chain_release();
  const int cur = min(max(*cur_index, 0), L - 1);
  if (static_cast<int>(blockIdx.x) < rows) {
    const int row = blockIdx.x;
    const long long id = live_seqs[static_cast<long long>(row) * L + cur];
    const long long tok = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    const uint4* src = reinterpret_cast<const uint4*>(emb + tok * d);
    uint4* dst = reinterpret_cast<uint4*>(x + static_cast<long long>(row) * d);
    for (int v = threadIdx.x; v < d / 8; v += kBeginThreads) dst[v] = src[v];
    return;
  }
  const int h = blockIdx.x - rows;
  for (int t = threadIdx.x; t < L; t += kBeginThreads)
    bias_row[static_cast<long long>(h) * L + t] =
        table[static_cast<long long>(h) * num_buckets + bucket_of_distance[max(cur - t, 0)]];
}

// Encoder keys and values [B, Lk, H, 64] in the layout of the tensor-core cross attention: keys
// [B, H, Lp, 64], values transposed [B, H, 64, Lp], zero beyond Lk. One CTA per 64 keys of a
// head; both sides move whole 128-byte rows, the values through shared memory. As tensor
// operations this was two fills and two strided copies of 0.22 ms each per layer at 64 x 512
// positions x 32 heads, against 0.08 ms for the bytes.
constexpr int kLayoutThreads = 256;
__global__ void __launch_bounds__(kLayoutThreads)
    decode_cross_layout_kernel(const __nv_bfloat16* __restrict__ k,
                               const __nv_bfloat16* __restrict__ v, __nv_bfloat16* __restrict__ kp,
                               __nv_bfloat16* __restrict__ vt, int Lk, int Lp, int H) {
  // [key][channel], the 16-byte pieces of a row permuted by key / 8: neither side has conflicts
  __shared__ __align__(16) __nv_bfloat16 tile[64][64];
  const int parts = (Lp + 63) / 64;
  const int bh = blockIdx.x / parts, t0 = (blockIdx.x - bh * parts) * 64;
  const int b = bh / H, h = bh - b * H;
  const int piece = threadIdx.x & 7;
  for (int r = threadIdx.x >> 3; r < 64; r += kLayoutThreads / 8) {
    const int key = t0 + r;
    uint4 ku = make_uint4(0u, 0u, 0u, 0u), vu = ku;
    if (key < Lk) {
      const long long at = ((static_cast<long long>(b) * Lk + key) * H + h) * 8 + piece;
      ku = reinterpret_cast<const uint4*>(k)[at];
      vu = reinterpret_cast<const uint4*>(v)[at];
    }
    if (key < Lp) reinterpret_cast<uint4*>(kp)[(static_cast<long long>(bh) * Lp + key) * 8 + piece] = ku;
    *reinterpret_cast<uint4*>(&tile[r][(piece ^ (r >> 3)) * 8]) = vu;
  }
  __syncthreads();
  // Lp is a multiple of 32: a row of the transposed tile is four or eight pieces of eight keys
  if (t0 + piece * 8 >= Lp) return;
  for (int c = threadIdx.x >> 3; c < 64; c += kLayoutThreads / 8) {
    __align__(16) __nv_bfloat16 o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = tile[piece * 8 + j][((c >> 3) ^ piece) * 8 + (c & 7)];
    *reinterpret_cast<uint4*>(vt + (static_cast<long long>(bh) * 64 + c) * Lp + t0 + piece * 8) =
        *reinterpret_cast<const uint4*>(o);
  }
}

constexpr int kCrossWarps = 8;
constexpr int kCrossThreads = kCrossWarps * 32;
constexpr int kCrossMaxKeys = 1024;

template <int BEAMS>
__global__ void __launch_bounds__(kCrossThreads, BEAMS <= 4 ? 4 : 2)
    decode_cross_attention_kernel(const __nv_bfloat16* __restrict__ q,  // [B*beams, H, 64]
                                  const __nv_bfloat16* __restrict__ k,  // [B, H, Lk, 64]
                                  const __nv_bfloat16* __restrict__ v,
                                  const uint8_t* __restrict__ key_mask,  // [B, Lk] or null
                                  __nv_bfloat16* __restrict__ out,       // [B*beams, H, 64]
                                  long long q_ld, int H, int Lk) {
  __shared__ float sp[BEAMS][kCrossMaxKeys];
  __shared__ float sred[BEAMS][kCrossWarps];
  // per-warp partial outputs reuse the probability buffer once every warp is done with it
  float (*sout)[BEAMS][kDecHeadDim] = reinterpret_cast<float (*)[BEAMS][kDecHeadDim]>(&sp[0][0]);
  static_assert(kCrossWarps * kDecHeadDim <= kCrossMaxKeys, "sout must fit in sp");
  const int b = blockIdx.x / H, h = blockIdx.x - b * H;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 3, part = lane & 7;
  constexpr int kRowsPerIter = kCrossWarps * 4;
  float qf[BEAMS][8];
#pragma unroll
  for (int j = 0; j < BEAMS; ++j) {
    const uint4 qu = reinterpret_cast<const uint4*>(
        q + (static_cast<long long>(b) * BEAMS + j) * q_ld + h * kDecHeadDim)[part];
    unpack8(qu, qf[j]);
  }
  // key / value layout [B, H, Lk, 64]: one (example, head) is a contiguous 128 * Lk bytes
  const long long kv_stride = kDecHeadDim;
  const long long kv_base = (static_cast<long long>(b) * H + h) * Lk * kDecHeadDim;
  const uint8_t* km = key_mask == nullptr ? nullptr : key_mask + static_cast<long long>(b) * Lk;

  // scores
  float mx[BEAMS];
#pragma unroll
  for (int j = 0; j < BEAMS; ++j) mx[j] = -INFINITY;
  constexpr int kU = 4;  // key rows in flight per lane group
  for (int t0 = 0; t0 < Lk; t0 += kU * kRowsPerIter) {
    uint4 ku[kU];
    int tt[kU];
    bool valid[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      tt[u] = t0 + u * kRowsPerIter + warp * 4 + g;
      valid[u] = tt[u] < Lk && (km == nullptr || km[tt[u]] != 0);
      ku[u] = make_uint4(0, 0, 0, 0);
      if (valid[u]) ku[u] = reinterpret_cast<const uint4*>(k + kv_base + tt[u] * kv_stride)[part];
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      float kf[8];
      unpack8(ku[u], kf);
#pragma unroll
      for (int j = 0; j < BEAMS; ++j) {
        float s = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) s = fmaf(qf[j][e], kf[e], s);
        float sv = sum_over_row_lanes(s);
        if (tt[u] < Lk) {
          if (!valid[u]) sv = -1e10f;  // additive mask value of the reference
          if (part == 0) sp[j][tt[u]] = sv;
          mx[j] = fmaxf(mx[j], sv);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < BEAMS; ++j) {
    const float m = warp_max(mx[j]);
    if (lane == 0) sred[j][warp] = m;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < BEAMS; ++j) {
    float m = sred[j][0];
#pragma unroll
    for (int w = 1; w < kCrossWarps; ++w) m = fmaxf(m, sred[j][w]);
    mx[j] = m;
  }
  __syncthreads();
  float sum[BEAMS];
#pragma unroll
  for (int j = 0; j < BEAMS; ++j) sum[j] = 0.f;
  for (int t = tid; t < Lk; t += kCrossThreads) {
#pragma unroll
    for (int j = 0; j < BEAMS; ++j) {
      const float e = __expf(sp[j][t] - mx[j]);
      sp[j][t] = e;
      sum[j] += e;
    }
  }
#pragma unroll
  for (int j = 0; j < BEAMS; ++j) {
    const float sj = warp_sum(sum[j]);
    if (lane == 0) sred[j][warp] = sj;
  }
  __syncthreads();

  // values
  float acc[BEAMS][8];
#pragma unroll
  for (int j = 0; j < BEAMS; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[j][e] = 0.f;
  for (int t0 = 0; t0 < Lk; t0 += kU * kRowsPerIter) {
    uint4 vu[kU];
    int tt[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      tt[u] = t0 + u * kRowsPerIter + warp * 4 + g;
      vu[u] = make_uint4(0, 0, 0, 0);
      if (tt[u] < Lk) vu[u] = reinterpret_cast<const uint4*>(v + kv_base + tt[u] * kv_stride)[part];
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (tt[u] < Lk) {
        float vf[8];
        unpack8(vu[u], vf);
#pragma unroll
        for (int j = 0; j < BEAMS; ++j) {
          const float pt = sp[j][tt[u]];
#pragma unroll
          for (int e = 0; e < 8; ++e) acc[j][e] = fmaf(pt, vf[e], acc[j][e]);
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < BEAMS; ++j)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float tot = sum_over_row_groups(acc[j][e]);
      if (g == 0) sout[warp][j][part * 8 + e] = tot;
    }
  __syncthreads();
  for (int i = tid; i < BEAMS * kDecHeadDim; i += kCrossThreads) {
    const int j = i / kDecHeadDim, d = i - j * kDecHeadDim;
    float tot = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kCrossWarps; ++w) {
      tot += sout[w][j][d];
      den += sred[j][w];
    }
    out[((static_cast<long long>(b) * BEAMS + j) * H + h) * kDecHeadDim + d] =
        __float2bfloat16(tot / den);
  }
}

}  // namespace t5x

using namespace t5x;

// k, v [B, Lk, H, 64] bf16 contiguous; kp [B, H, Lp, 64], vt [B, H, 64, Lp], Lp a multiple of 32.
T5X_API int t5x_decode_cross_layout(const void* k, const void* v, void* kp, void* vt, int B, int Lk,
                                    int H, int Lp, void* stream) {
  using namespace t5x;
  if (B <= 0 || Lp <= 0 || H <= 0) return 0;
  const long long blocks = static_cast<long long>((Lp + 63) / 64) * H * B;
  if (Lp % 32 || Lp < Lk || blocks > 0x7fffffff)
    return set_error("decode_cross_layout: B=%d H=%d Lk=%d Lp=%d is not covered", B, H, Lk, Lp);
  if ((reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(kp) | reinterpret_cast<uintptr_t>(vt)) & 15)
    return set_error("decode_cross_layout: tensors must start on 16-byte boundaries");
  decode_cross_layout_kernel<<<static_cast<unsigned>(blocks), kLayoutThreads, 0,
                               static_cast<cudaStream_t>(stream)>>>(
      static_cast<const __nv_bfloat16*>(k), static_cast<const __nv_bfloat16*>(v),
      static_cast<__nv_bfloat16*>(kp), static_cast<__nv_bfloat16*>(vt), Lk, Lp, H);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("decode_cross_layout: %s", cudaGetErrorString(e));
  return 0;
}

// live_seqs [rows, L] int64, cur_index device int32, emb [vocab, d] bf16 (d % 8 == 0, 16-byte
// aligned), x [rows, d] bf16; table [H, num_buckets] fp32, bucket_of_distance [L] int32 in
// [0, num_buckets), bias_row [H, L] fp32.
T5X_API int t5x_decode_begin(const void* live_seqs, const void* cur_index, const void* emb, void* x,
                             const void* table, const void* bucket_of_distance, void* bias_row,
                             int rows, int H, int L, int d, int vocab, int num_buckets,
                             void* stream) {
  using namespace t5x;
  if (rows <= 0 || L <= 0) return 0;
  if (d % 8 || ((reinterpret_cast<uintptr_t>(emb) | reinterpret_cast<uintptr_t>(x)) & 15))
    return set_error("decode_begin: embedding rows must be 16-byte aligned (d=%d)", d);
  decode_begin_kernel<<<rows + H, kBeginThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const long long*>(live_seqs), static_cast<const int*>(cur_index),
      static_cast<const __nv_bfloat16*>(emb), static_cast<__nv_bfloat16*>(x),
      static_cast<const float*>(table), static_cast<const int*>(bucket_of_distance),
      static_cast<float*>(bias_row), rows, L, d, vocab, num_buckets);
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("decode_begin: %s", cudaGetErrorString(e));
  return 0;
}

// q, k_new, v_new: [rows, heads, 64] bf16 with row stride `in_ld` elements (views into one
// fused projection are fine; 16-byte aligned), out: [rows, heads, 64] contiguous; rows =
// batch * beams; cache_k / cache_v: [batch, beams, heads, max_len, 64] bf16; ancestry:
// [batch, beams, max_len] int32; bias_row: [heads, max_len] fp32 or null; cur_index: device
// int32 (position being decoded).
T5X_API int t5x_decode_self_attention(const void* q, const void* k_new, const void* v_new,
                                      void* cache_k, void* cache_v, const void* ancestry,
                                      const void* bias_row, const void* cur_index, void* out,
                                      long long in_ld, int rows, int beams, int heads,
                                      int head_dim, int max_len, void* stream) {
  if (rows <= 0) return 0;
  if (head_dim != kDecHeadDim) return set_error("decode_self_attention: head_dim must be 64");
  if (max_len > kDecMaxLen) return set_error("decode_self_attention: max_len > %d", kDecMaxLen);
  if (beams <= 0 || rows % beams) return set_error("decode_self_attention: rows %% beams != 0");
  if (in_ld % 8) return set_error("decode_self_attention: input row stride must be a multiple of 8");
  const int items = rows * heads;
  // Up to 16 warps an SM the loads' latency counts, beyond that the warps hide it and the 118
  // registers of the wide form (128 in a chain) cost occupancy. us, wide / narrow: 4 rows x 12 heads at
  // position 40 5.5 / 7.2, 64 x 32 10.4 / 12.2, 256 rows x 32 heads over 64 steps 28.2 / 22.5.
  const bool wide = items <= 16 * num_sms();
  auto kernel = chained_launches()
                    ? (wide ? decode_self_attention_kernel<8, true> : decode_self_attention_kernel<0, true>)
                    : (wide ? decode_self_attention_kernel<8, false> : decode_self_attention_kernel<0, false>);
  cudaError_t e = launch_chained(
      kernel, dim3((items + kDecWarps - 1) / kDecWarps), dim3(kDecWarps * 32),
      0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(q),
      static_cast<const __nv_bfloat16*>(k_new), static_cast<const __nv_bfloat16*>(v_new),
      static_cast<__nv_bfloat16*>(cache_k), static_cast<__nv_bfloat16*>(cache_v),
      static_cast<const int*>(ancestry), static_cast<const float*>(bias_row),
      static_cast<const int*>(cur_index), static_cast<__nv_bfloat16*>(out), in_ld, rows, beams,
      heads, max_len);
  count_launches(1);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("decode_self_attention: %s", cudaGetErrorString(e));
  return 0;
}

// q: [batch * beams, heads, 64] bf16 with row stride q_ld; k, v: [batch, heads, Lk, 64] bf16
// contiguous; key_mask: [batch, Lk] uint8 (0 = padding) or null; out: [batch * beams, heads, 64].
// beams must be 1, 2, 4 or 8.
T5X_API int t5x_decode_cross_attention(const void* q, const void* k, const void* v,
                                       const void* key_mask, void* out, long long q_ld, int batch,
                                       int beams, int heads, int head_dim, int Lk, void* stream) {
  if (batch <= 0) return 0;
  if (head_dim != kDecHeadDim) return set_error("decode_cross_attention: head_dim must be 64");
  if (Lk < 1 || Lk > kCrossMaxKeys)
    return set_error("decode_cross_attention: Lk must be in [1, %d]", kCrossMaxKeys);
  if (q_ld % 8) return set_error("decode_cross_attention: q row stride must be a multiple of 8");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid(batch * heads);
  auto qp = static_cast<const __nv_bfloat16*>(q);
  auto kp = static_cast<const __nv_bfloat16*>(k);
  auto vp = static_cast<const __nv_bfloat16*>(v);
  auto mp = static_cast<const uint8_t*>(key_mask);
  auto op = static_cast<__nv_bfloat16*>(out);
  switch (beams) {
    case 1:
      decode_cross_attention_kernel<1><<<grid, kCrossThreads, 0, st>>>(qp, kp, vp, mp, op, q_ld, heads, Lk);
      break;
    case 2:
      decode_cross_attention_kernel<2><<<grid, kCrossThreads, 0, st>>>(qp, kp, vp, mp, op, q_ld, heads, Lk);
      break;
    case 4:
      decode_cross_attention_kernel<4><<<grid, kCrossThreads, 0, st>>>(qp, kp, vp, mp, op, q_ld, heads, Lk);
      break;
    case 8:
      decode_cross_attention_kernel<8><<<grid, kCrossThreads, 0, st>>>(qp, kp, vp, mp, op, q_ld, heads, Lk);
      break;
    default:
      return set_error("decode_cross_attention: beams must be 1, 2, 4 or 8 (got %d)", beams);
  }
  count_launches(1);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return set_error("decode_cross_attention: %s", cudaGetErrorString(e));
  return 0;
}
