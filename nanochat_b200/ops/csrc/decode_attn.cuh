// Device parts of single-token attention at head dim 128, shared by the kernels that attend: where a token lies in the
// cache, the rotary + norm of a query or key, and a CTA's share of a row's keys with an online softmax.
//
// A key is served by half a warp: a lane holds eight dims (one 16-byte load of K, one of V), so a warp's load covers two
// whole 256-byte rows and a dot product costs four shuffles for two keys. Four keys per half warp are requested ahead of
// the four being used (8 loads of 16 bytes in flight per lane), which is what covers the latency of the page lookups and
// of HBM; a key per thread instead (32 rows per load instruction, nothing in flight behind it) took twice as long.
#pragma once

#include "decode.h"
#include "ptx.cuh"

namespace nc {

constexpr float kDecodeEps = 1.1920929e-07f;   // fp32 machine epsilon, as F.rms_norm(eps=None)
constexpr int kAttnWarps = 8;                  // warps that share the keys of one (row, head, split)
constexpr int kKeysAhead = 4;                  // keys of a half warp per batch
constexpr int kTableCache = 128;               // page-table entries a CTA keeps in shared memory

// Where token t of a row lives in one layer's K (or V) store: contiguous rows (table == nullptr; `base` is the row's
// offset), or pages of 2^page_shift tokens named by the row's table (c_bat is then the pitch of a page).
struct KvRow {
  const int* table;
  int page_shift;
  long long base, c_bat, c_tok;
  __device__ __forceinline__ long long at(int t) const {
    if (table == nullptr) return base + (long long)t * c_tok;
    return table[t >> page_shift] * c_bat + (long long)(t & ((1 << page_shift) - 1)) * c_tok;
  }
};

__device__ __forceinline__ KvRow kv_row(const KvPages& pages, int b, long long c_bat, long long c_tok) {
  return {pages.table == nullptr ? nullptr : pages.table + (long long)b * pages.max_pages, pages.page_shift, b * c_bat, c_bat, c_tok};
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const float2 a = unpack_bf16(v.x), b = unpack_bf16(v.y), c = unpack_bf16(v.z), d = unpack_bf16(v.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
}
// Sum over the 16 lanes of a half warp; every lane gets it. All 32 lanes take part.
__device__ __forceinline__ float half_sum(float v) {
#pragma unroll
  for (int w = 8; w > 0; w >>= 1) v += __shfl_xor_sync(0xffffffffu, v, w);
  return v;
}

// Rotary at one position, RMS norm and the gain of 1.2 on a head spread over a half warp (lane hl: dims 8 hl .. 8 hl + 7);
// rounded to bf16 as the cache and the tensor cores take it. cos / sin: the position's 64 entries.
__device__ __forceinline__ uint4 rope_norm_half(const uint4& raw, const __nv_bfloat16* cos_p, const __nv_bfloat16* sin_p, int hl) {
  float x[8], c[8], s[8], y[8], ss = 0.f;
  unpack8(raw, x);
  unpack8(*reinterpret_cast<const uint4*>(cos_p + (hl & 7) * 8), c);
  unpack8(*reinterpret_cast<const uint4*>(sin_p + (hl & 7) * 8), s);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float o = __shfl_xor_sync(0xffffffffu, x[i], 8);          // the partner dim, 64 away
    y[i] = hl < 8 ? x[i] * c[i] + o * s[i] : x[i] * c[i] - o * s[i];
    ss += y[i] * y[i];
  }
  const float r = rsqrtf(half_sum(ss) * (1.f / 128.f) + kDecodeEps) * 1.2f;
#pragma unroll
  for (int i = 0; i < 8; ++i) y[i] *= r;
  return pack8(y);
}

struct KeyBatch {
  uint4 k[kKeysAhead], v[kKeysAhead];
};
// Keys j0 + half + 16 u of one row; places past `end` read the last key instead (their weight is zero).
__device__ __forceinline__ void load_keys(KeyBatch& b, const __nv_bfloat16* kb, const __nv_bfloat16* vb, const KvRow& row, int j0, int end) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < kKeysAhead; ++u) {
    const int j = min(j0 + (lane >> 4) + 2 * kAttnWarps * u, end - 1);
    const long long o = row.at(j) + (lane & 15) * 8;
    b.k[u] = __ldcg(reinterpret_cast<const uint4*>(kb + o));
    b.v[u] = __ldcg(reinterpret_cast<const uint4*>(vb + o));
  }
}

// Online softmax of one half warp.
struct HalfSoftmax {
  float m = -1.0e30f, l = 0.f, o[8] = {};

  __device__ __forceinline__ void add(const KeyBatch& b, const float (&q)[8], float scale_log2, int j0, int end) {
    const int half = (threadIdx.x & 31) >> 4;
    float s[kKeysAhead], top = m;
#pragma unroll
    for (int u = 0; u < kKeysAhead; ++u) {
      float k[8], d = 0.f;
      unpack8(b.k[u], k);
#pragma unroll
      for (int i = 0; i < 8; ++i) d += q[i] * k[i];
      s[u] = half_sum(d) * scale_log2;
      if (j0 + half + 2 * kAttnWarps * u >= end) s[u] = -1.0e30f;
      top = fmaxf(top, s[u]);
    }
    const float alpha = exp2f(m - top);
    m = top;
    l *= alpha;
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] *= alpha;
#pragma unroll
    for (int u = 0; u < kKeysAhead; ++u) {
      const float p = j0 + half + 2 * kAttnWarps * u < end ? exp2f(s[u] - top) : 0.f;
      float v[8];
      unpack8(b.v[u], v);
      l += p;
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] += p * v[i];
    }
  }
};

struct AttnShared {
  float m[2 * kAttnWarps], l[2 * kAttnWarps], o[2 * kAttnWarps][128];
};

// All keys [begin, end) of a row by the CTA's first kAttnWarps warps; `b` holds this warp's first batch already
// (load_keys at begin + 2 warp), so that the caller can request it before it has the query.
__device__ __forceinline__ void attend_keys(HalfSoftmax& st, KeyBatch& b, const float (&q)[8], const __nv_bfloat16* kb, const __nv_bfloat16* vb,
                                            const KvRow& row, int begin, int end, float scale_log2) {
  const int first = begin + 2 * (threadIdx.x >> 5);
  constexpr int STEP = 2 * kAttnWarps * kKeysAhead;
  for (int j = first; j < end; j += STEP) {
    KeyBatch next;
    if (j + STEP < end) load_keys(next, kb, vb, row, j + STEP, end);
    st.add(b, q, scale_log2, j, end);
    b = next;
  }
}

// Every half warp leaves its part; after the caller's barrier merge_halves gives dim d of the CTA's sum.
__device__ __forceinline__ void leave_half(AttnShared& sh, const HalfSoftmax& st) {
  const int hw = threadIdx.x >> 4, hl = threadIdx.x & 15;
  if (hl == 0) { sh.m[hw] = st.m; sh.l[hw] = st.l; }
  *reinterpret_cast<float4*>(&sh.o[hw][hl * 8]) = make_float4(st.o[0], st.o[1], st.o[2], st.o[3]);
  *reinterpret_cast<float4*>(&sh.o[hw][hl * 8 + 4]) = make_float4(st.o[4], st.o[5], st.o[6], st.o[7]);
}
__device__ __forceinline__ void merge_halves(const AttnShared& sh, int d, float& m, float& l, float& o) {
  m = -1.0e30f; l = 0.f; o = 0.f;
#pragma unroll
  for (int i = 0; i < 2 * kAttnWarps; ++i) m = fmaxf(m, sh.m[i]);
#pragma unroll
  for (int i = 0; i < 2 * kAttnWarps; ++i) {
    const float f = exp2f(sh.m[i] - m);
    l += f * sh.l[i];
    o += f * sh.o[i][d];
  }
}

}  // namespace nc
