// Attention of a decode step with everything around it: rotary and norm of the step's queries and keys, value embeddings,
// append to the cache, softmax over each row's keys.
//
// Rows that continue one prompt name the same pages for it, and reading those once per row made the kernel a bandwidth
// problem (d26, 64 rows of 520 tokens: 221 MB of cache reads a layer, 36.5 us). A cluster of C CTAs therefore serves one head
// of G <= 8 rows: the pages that all its rows name go to its warps sixteen keys at a time, as matrix products with the G rows
// (mma.sync: a handful of rows does not fill a tcgen05 tile, and the operands come straight from global memory); what a row
// has for itself is spread over the half warps that belong to the row. Probabilities enter the product as two bf16, the upper
// eight rows of the tile carrying what rounding the lower eight left, so that they keep 16 bits of fraction.
// The parts meet in the shared memory of the CTA that owns the row (st.async counted on an mbarrier) instead of going through
// global memory and an arrival counter. How many leading pages are shared is found by comparing the page tables, so any table
// is right, whoever made it. Positions, tables and older keys are read before the wait on the projections.
#include "decode.h"
#include "decode_attn.cuh"
#include "host_utils.cuh"
#include "ptx.cuh"

namespace nc {

namespace {

constexpr int THREADS = kAttnWarps * 32;
constexpr int HALVES = 2 * kAttnWarps;         // half warps of a CTA
constexpr int REGISTERS_FOR = THREADS + 64;    // threads the registers are divided by: a linear layer's CTA stays beside this one

struct Args {
  const __nv_bfloat16* qkv; long long ld;
  __nv_bfloat16 *k_cache, *v_cache; long long c_bat, c_tok;
  const int* seqlens;
  int B, H, Hkv, window, t_max;
  float scale_log2;
  const __nv_bfloat16 *cos_t, *sin_t;
  const __nv_bfloat16* xn; long long ld_xn; const float* wg;            // value-embedding gate; xn == nullptr: none
  const __nv_bfloat16* ve; long long ld_ve; const long long* idx;
  __nv_bfloat16* y; long long ldy;
  KvPages pages;
  int* status;
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_async(uint32_t addr, float v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
               ::"r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}

__device__ __forceinline__ void st_async4(uint32_t addr, const float4& v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(addr), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)),
               "r"(bar) : "memory");
}
__device__ __forceinline__ void store_row(const Args& a, int b, int h, int d, const float4& O, float L) {
  const float r = L > 0.f ? 1.f / L : 0.f;
  *reinterpret_cast<uint2*>(a.y + b * a.ldy + h * 128 + d) = make_uint2(pack_bf16(O.x * r, O.y * r), pack_bf16(O.z * r, O.w * r));
}

// Keys j0, j0 + stride, ... of a row, one per half warp and place; places past `end` read the last key (weight zero).
template <int U>
struct Keys {
  uint4 k[U], v[U];
  __device__ __forceinline__ void load(const __nv_bfloat16* kb, const __nv_bfloat16* vb, const KvRow& row, int j0, int stride, int end) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long o = row.at(min(j0 + u * stride, end - 1)) + (threadIdx.x & 15) * 8;
      k[u] = __ldcg(reinterpret_cast<const uint4*>(kb + o));
      v[u] = __ldcg(reinterpret_cast<const uint4*>(vb + o));
    }
  }
};

// Online softmax of a half warp for one row: a lane holds dims 8 hl .. 8 hl + 7 of the sum.
struct OwnSoftmax {
  float m = -1.0e30f, l = 0.f, o[8] = {};

  // keys j0 + u * stride; those from `end` on do not count
  template <int U>
  __device__ __forceinline__ void add(const Keys<U>& b, const float (&q)[8], float scale_log2, int j0, int stride, int end) {
    float p[U], top = m;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float k[8], d = 0.f;
      unpack8(b.k[u], k);
#pragma unroll
      for (int i = 0; i < 8; ++i) d += q[i] * k[i];
      p[u] = half_sum(d) * scale_log2;
      if (j0 + u * stride >= end) p[u] = -1.0e30f;
      top = fmaxf(top, p[u]);
    }
    const float alpha = exp2f(m - top);
    m = top;
    l *= alpha;
#pragma unroll
    for (int i = 0; i < 8; ++i) o[i] *= alpha;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      p[u] = j0 + u * stride >= end ? 0.f : exp2f(p[u] - top);
      float v[8];
      unpack8(b.v[u], v);
      l += p[u];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i] += p[u] * v[i];
    }
  }
};

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Sixteen keys for eight rows by one warp. With g = lane / 4, q = lane % 4:
//   scores (row g, keys 8 t + 2 q + e): the sum over dims takes any order, so lane (g, q) feeds dims 32 i + 8 q .. + 7 of key
//   8 t + g as they come from one 16-byte load, and of row g's query by the same rule;
//   sums (row g, dims 64 f + 8 (2 q + e) + t): tile t of half f takes the t-th dim of each lane's 16 bytes of V, and a lane
//   loads keys 2 q, 2 q + 1, 2 q + 8, 2 q + 9, which pairs them as the product wants them.
struct SharedKeys {
  uint4 k[2][4], v[2][4];
  __device__ __forceinline__ void load_k(const __nv_bfloat16* kb, const KvRow& row, int j0, int end) {
    const int g = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const __nv_bfloat16* p = kb + row.at(min(j0 + 8 * t + g, end - 1)) + q * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) k[t][i] = __ldcg(reinterpret_cast<const uint4*>(p + 32 * i));
    }
  }
  __device__ __forceinline__ void load_v(const __nv_bfloat16* vb, const KvRow& row, int j0, int end) {
    const int g = (threadIdx.x & 31) >> 2, q = threadIdx.x & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat16* p = vb + row.at(min(j0 + 2 * q + (i & 1) + 8 * (i >> 1), end - 1)) + g * 8;
#pragma unroll
      for (int f = 0; f < 2; ++f) v[f][i] = __ldcg(reinterpret_cast<const uint4*>(p + 64 * f));
    }
  }
};

struct SharedSoftmax {
  float m = -1.0e30f, l = 0.f, o[16][4] = {};     // m: row g's, l: this lane's share of row g's; o[.][2 + e]: the rounding remainders'

  __device__ __forceinline__ void scores(float (&s)[2][4], const SharedKeys& b, const __nv_bfloat16* q_row) const {
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[t][e] = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 q = *reinterpret_cast<const uint4*>(q_row + 32 * i + (threadIdx.x & 3) * 8);
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        mma_16816(s[t], q.x, 0u, q.y, 0u, b.k[t][i].x, b.k[t][i].y);
        mma_16816(s[t], q.z, 0u, q.w, 0u, b.k[t][i].z, b.k[t][i].w);
      }
    }
  }
  // keys j0 .. j0 + 15; those outside [lo, end) do not count (lo: row g's)
  __device__ __forceinline__ void weigh(float (&s)[2][4], float scale_log2, int j0, int lo, int end) {
    float top = m;
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = j0 + 8 * t + 2 * (threadIdx.x & 3) + e;
        s[t][e] = j < lo || j >= end ? -1.0e30f : s[t][e] * scale_log2;
        top = fmaxf(top, s[t][e]);
      }
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
    const float alpha = exp2f(m - top);
    m = top;
    l *= alpha;
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int j = j0 + 8 * t + 2 * (threadIdx.x & 3) + e;
        s[t][e] = j < lo || j >= end ? 0.f : exp2f(s[t][e] - top);
        l += s[t][e];
      }
    if (__any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll
      for (int t = 0; t < 16; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[t][e] *= alpha;
    }
  }
  __device__ __forceinline__ void sums(const float (&p)[2][4], const SharedKeys& b) {
    uint32_t hi[2], lo[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      hi[t] = pack_bf16(p[t][0], p[t][1]);
      const float2 h = unpack_bf16(hi[t]);
      lo[t] = pack_bf16(p[t][0] - h.x, p[t][1] - h.y);
    }
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const uint4 &a = b.v[f][0], &c = b.v[f][1], &d = b.v[f][2], &e = b.v[f][3];
      const uint32_t va[4] = {a.x, a.y, a.z, a.w}, vc[4] = {c.x, c.y, c.z, c.w}, vd[4] = {d.x, d.y, d.z, d.w}, ve[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const uint32_t sel = t & 1 ? 0x7632 : 0x5410;
        mma_16816(o[f * 8 + t], hi[0], lo[0], hi[1], lo[1], __byte_perm(va[t >> 1], vc[t >> 1], sel), __byte_perm(vd[t >> 1], ve[t >> 1], sel));
      }
    }
  }
};

// grid (C, H, ceil(B / G)), clusters of C CTAs.
// Bound by the chain position -> page -> key (before the wait, when there is room to start early) and q -> scores -> parts ->
// row behind it. Step of d26 after 512 tokens with one CTA per (row, head, split) and a merge through global memory / now: 1 row
// 757 / 732 us, 8 rows 1153 / 998, 64 rows 2165 / 1658.
template <int G>
__global__ void __launch_bounds__(REGISTERS_FOR) decode_qkv_attn_kernel(const Args a) {
  constexpr int AHEAD = 4;
  constexpr bool SHARE = G > 1;
  static_assert(G == 1 || G == 8, "rows of the matrix products");
  __shared__ int s_pos[G], s_shared;
  __shared__ int s_table[G][kTableCache];
  __shared__ __align__(16) __nv_bfloat16 s_q[G][128];
  __shared__ __align__(16) float s_o[SHARE ? kAttnWarps : 1][G][128], p_o[kAttnWarps][128];     // shared keys: [warp][row]; own: [warp]
  __shared__ float s_m[kAttnWarps][G], s_l[kAttnWarps][G], p_m[kAttnWarps], p_l[kAttnWarps];
  __shared__ float f_s[G][kAttnWarps], f_p[G][kAttnWarps], t_m[G], t_l[G];
  __shared__ __align__(16) float r_o[8][128];               // parts of this CTA's rows: [row][CTA], at most 8
  __shared__ float r_m[8], r_l[8];
  __shared__ uint64_t parts_full;
  __shared__ int abort_word;
  const int C = gridDim.x, c = blockIdx.x, h = blockIdx.y, r0 = blockIdx.z * G, group = a.H / a.Hkv, hkv = h / group;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hl = lane & 15, half = lane >> 4;
  const int mine = (G - c + C - 1) / C;                     // rows c, c + C, ... of the group are this CTA's (none from G on)
  if (tid == 0) {
    mbar_init(&parts_full, 1);
    abort_word = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(&parts_full, max(mine, 0) * C * (128 + 2) * 4);
    s_shared = a.pages.max_pages;
  }
  // a position outside the cache (or no such row): -1
  if (tid < G) {
    const int pos = r0 + tid < a.B ? a.seqlens[r0 + tid] : -1;
    s_pos[tid] = pos >= 0 && pos < a.t_max ? pos : -1;
  }
  const bool cached = a.pages.table != nullptr && a.pages.max_pages <= kTableCache;
  const int* table = a.pages.table;
  if (cached) {
    for (int i = tid; i < G * a.pages.max_pages; i += THREADS) {
      const int g = i / a.pages.max_pages, p = i - g * a.pages.max_pages;
      s_table[g][p] = r0 + g < a.B ? table[(long long)(r0 + g) * a.pages.max_pages + p] : 0;
    }
  }
  __syncthreads();
  auto row_of = [&](int g) {
    KvRow row = kv_row(a.pages, r0 + g, a.c_bat, a.c_tok);
    if (cached) row.table = s_table[g];
    return row;
  };
  // tokens below sh_end lie in pages that all rows of the group name
  int rows = 0, first = 0, least = 0x7fffffff;
#pragma unroll
  for (int g = G - 1; g >= 0; --g)
    if (s_pos[g] >= 0) { ++rows; first = g; least = min(least, s_pos[g]); }
  int sh_end = 0;
  if (G > 1 && table != nullptr && rows > 1) {              // the same for all threads
    const KvRow base = row_of(first);
    const int full = min(least >> a.pages.page_shift, a.pages.max_pages);
    for (int p = tid; p < full; p += THREADS) {
      bool same = true;
      for (int g = first + 1; g < G; ++g)
        if (s_pos[g] >= 0) same = same && row_of(g).table[p] == base.table[p];
      if (!same) atomicMin(&s_shared, p);
    }
    __syncthreads();
    sh_end = min(full, s_shared) << a.pages.page_shift;
  }
  auto low = [&](int pos) { return a.window < 0 ? 0 : max(0, pos - a.window); };
  const __nv_bfloat16 *kb = a.k_cache + hkv * 128, *vb = a.v_cache + hkv * 128;
  // shared keys, from the lowest row's window on: sixteen at a time, the warps of the cluster taking turns
  const int sh_step = C * kAttnWarps * 16, sh_first = (rows > 0 ? low(least) : 0) + (c * kAttnWarps + warp) * 16;
  const KvRow shared_row = row_of(first);
  SharedKeys shared;
  if (SHARE && sh_first < sh_end) {
    shared.load_k(kb, shared_row, sh_first, sh_end);
    shared.load_v(vb, shared_row, sh_first, sh_end);
  }
  // own keys: the half warps of the cluster are divided among the rows there are (their number rounded up to a power of two);
  // row gp's [p_lo, pos), every per_row-th one
  const int there = min(G, a.B - r0), row_shift = there > 1 ? 32 - __clz(there - 1) : 0;
  const int per_row = (C * HALVES) >> row_shift, slot = c * HALVES + 2 * warp, gp = slot / per_row, sub = slot - gp * per_row;
  const int pos = s_pos[gp], p_lo = pos >= 0 ? max(low(pos), sh_end) : 0, p_first = p_lo + sub;
  const KvRow own_row = row_of(gp);
  Keys<AHEAD> own;
  if (p_first < pos) own.load(kb, vb, own_row, p_first + half, per_row, pos);
  if (C > 1) cluster_sync_all();                            // the barriers that the others count on are ready
  pdl_wait();
  pdl_trigger();
  if (tid < G && c == 0 && h == 0 && r0 + tid < a.B && s_pos[tid] < 0 && a.status)        // a full cache: the row is left alone
    atomicCAS(a.status, 0, (ST_BAD_ARG << 24) | 0xdec0de);

  // queries of all rows, a half warp each
  if (2 * warp < G) {
    const int g = min(2 * warp + half, G - 1), qpos = max(s_pos[g], 0);
    const int src = min(r0 + g, a.B - 1);
    const uint4 q = rope_norm_half(*reinterpret_cast<const uint4*>(a.qkv + src * a.ld + h * 128 + hl * 8), a.cos_t + (long long)qpos * 64,
                                   a.sin_t + (long long)qpos * 64, hl);
    *reinterpret_cast<uint4*>(&s_q[g][hl * 8]) = q;
  }
  // the new key of row gp, by the last of its warps
  uint4 kn = make_uint4(0, 0, 0, 0), vn = kn;
  const bool newest = pos >= 0 && sub == per_row - 2;
  if (newest) {
    const __nv_bfloat16* proj = a.qkv + (r0 + gp) * a.ld;
    kn = rope_norm_half(*reinterpret_cast<const uint4*>(proj + (a.H + hkv) * 128 + hl * 8), a.cos_t + (long long)pos * 64,
                        a.sin_t + (long long)pos * 64, hl);
    vn = *reinterpret_cast<const uint4*>(proj + (a.H + a.Hkv + hkv) * 128 + hl * 8);
    if (a.xn != nullptr) {
      float gate = hl < 12 ? __bfloat162float(a.xn[(r0 + gp) * a.ld_xn + hl]) * a.wg[hkv * 12 + hl] : 0.f;
      gate = 3.f / (1.f + __expf(-half_sum(gate)));
      float v[8], e[8];
      unpack8(vn, v);
      unpack8(*reinterpret_cast<const uint4*>(a.ve + a.idx[r0 + gp] * a.ld_ve + hkv * 128 + hl * 8), e);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] += gate * e[i];
      vn = pack8(v);
    }
    if (half == 0 && h % group == 0) {
      const long long o = own_row.at(pos) + hkv * 128 + hl * 8;
      *reinterpret_cast<uint4*>(a.k_cache + o) = kn;
      *reinterpret_cast<uint4*>(a.v_cache + o) = vn;
    }
  }
  __syncthreads();

  {
    OwnSoftmax st;
    float q[8];
    unpack8(*reinterpret_cast<const uint4*>(&s_q[gp][hl * 8]), q);
    if (newest) {
      Keys<1> b;
      b.k[0] = kn; b.v[0] = vn;
      st.add<1>(b, q, a.scale_log2, half, 1, 1);            // the other half of the warp starts empty
    }
    for (int j = p_first; j < pos; j += AHEAD * per_row) {
      Keys<AHEAD> next;
      if (j + AHEAD * per_row < pos) next.load(kb, vb, own_row, j + AHEAD * per_row + half, per_row, pos);
      st.add<AHEAD>(own, q, a.scale_log2, j + half, per_row, pos);
      own = next;
    }
    // the two halves of the warp
    const float om = __shfl_xor_sync(0xffffffffu, st.m, 16), top = fmaxf(st.m, om), f = exp2f(st.m - top);
    st.l *= f;
    st.l += __shfl_xor_sync(0xffffffffu, st.l, 16);
    if (lane == 0) { p_m[warp] = top; p_l[warp] = st.l; }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      st.o[i] *= f;
      st.o[i] += __shfl_xor_sync(0xffffffffu, st.o[i], 16);
    }
    if (half == 0) *reinterpret_cast<float4*>(&p_o[warp][hl * 8]) = make_float4(st.o[0], st.o[1], st.o[2], st.o[3]);
    else *reinterpret_cast<float4*>(&p_o[warp][hl * 8 + 4]) = make_float4(st.o[4], st.o[5], st.o[6], st.o[7]);
  }
  if (SHARE && sh_end > 0) {
    SharedSoftmax st;
    const int g = lane >> 2, q4 = lane & 3;
    const int row_lo = s_pos[g % G] >= 0 ? low(s_pos[g % G]) : 0x7fffffff;
    for (int j = sh_first; j < sh_end; j += sh_step) {
      float s[2][4];
      st.scores(s, shared, s_q[g % G]);
      if (j + sh_step < sh_end) shared.load_k(kb, shared_row, j + sh_step, sh_end);
      st.weigh(s, a.scale_log2, j, row_lo, sh_end);
      st.sums(s, shared);
      if (j + sh_step < sh_end) shared.load_v(vb, shared_row, j + sh_step, sh_end);
    }
    st.l += __shfl_xor_sync(0xffffffffu, st.l, 1);
    st.l += __shfl_xor_sync(0xffffffffu, st.l, 2);
    if (q4 == 0) { s_m[warp][g % G] = st.m; s_l[warp][g % G] = st.l; }
#pragma unroll
    for (int f = 0; f < 2; ++f)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float* dst = &s_o[SHARE ? warp : 0][g % G][64 * f + 8 * (2 * q4 + e)];
#pragma unroll
        for (int t = 0; t < 8; t += 4)
          *reinterpret_cast<float4*>(dst + t) =
              make_float4(st.o[f * 8 + t][e] + st.o[f * 8 + t][2 + e], st.o[f * 8 + t + 1][e] + st.o[f * 8 + t + 1][2 + e],
                          st.o[f * 8 + t + 2][e] + st.o[f * 8 + t + 2][2 + e], st.o[f * 8 + t + 3][e] + st.o[f * 8 + t + 3][2 + e]);
      }
  }
  __syncthreads();
  // the warps of the CTA: what each part counts for in its row, then a thread per row and four dims
  if (tid < G * kAttnWarps) {
    const int g = tid / kAttnWarps, w = tid % kAttnWarps;
    const unsigned lanes = G * kAttnWarps >= 32 ? 0xffffffffu : (1u << (G * kAttnWarps)) - 1;
    const bool its = (c * HALVES + 2 * w) / per_row == g, sh = SHARE && sh_end > 0;
    const float ms = sh ? s_m[w][g] : -1.0e30f, mp = its ? p_m[w] : -1.0e30f;
    float top = fmaxf(ms, mp);
#pragma unroll
    for (int x = 1; x < kAttnWarps; x <<= 1) top = fmaxf(top, __shfl_xor_sync(lanes, top, x));
    const float fs = exp2f(ms - top), fp = exp2f(mp - top);
    float L = (sh ? fs * s_l[w][g] : 0.f) + (its ? fp * p_l[w] : 0.f);
#pragma unroll
    for (int x = 1; x < kAttnWarps; x <<= 1) L += __shfl_xor_sync(lanes, L, x);
    f_s[g][w] = fs;
    f_p[g][w] = fp;
    if (w == 0) { t_m[g] = top; t_l[g] = L; }
  }
  __syncthreads();
  const uint32_t bar = smem_u32(&parts_full);
  const int g = warp, d = lane * 4;
  if (g < G) {
    float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
    auto plus = [&](float f, const float* x) {
      const float4 v = *reinterpret_cast<const float4*>(x);
      O.x += f * v.x; O.y += f * v.y; O.z += f * v.z; O.w += f * v.w;
    };
    if (SHARE && sh_end > 0) {
#pragma unroll
      for (int w = 0; w < kAttnWarps; ++w) plus(f_s[g][w], &s_o[SHARE ? w : 0][g][d]);
    }
    const int w0 = max(0, (g * per_row - c * HALVES) / 2), w1 = min(kAttnWarps, ((g + 1) * per_row - c * HALVES) / 2);
#pragma unroll 4
    for (int w = w0; w < w1; ++w) plus(f_p[g][w], &p_o[w][d]);
    if (C == 1) {
      if (s_pos[g] >= 0) store_row(a, r0 + g, h, d, O, t_l[g]);
    } else {
      const int owner = g % C, part = (g / C) * C + c;
      st_async4(map_to_cta(smem_u32(&r_o[part][d]), owner), O, map_to_cta(bar, owner));
      if (lane == 0) {
        st_async(map_to_cta(smem_u32(&r_m[part]), owner), t_m[g], map_to_cta(bar, owner));
        st_async(map_to_cta(smem_u32(&r_l[part]), owner), t_l[g], map_to_cta(bar, owner));
      }
    }
  }
  if (C == 1) return;
  __syncwarp();
  cluster_arrive();                                         // this warp has sent its share
  if (warp < mine && mbar_wait(&parts_full, 0, &abort_word, a.status, ST_WAIT_PEER, 0xa77e)) {
    const int own_g = c + warp * C;
    if (s_pos[own_g] >= 0) {
      const float m = lane < C ? r_m[warp * C + lane] : -1.0e30f;
      float top = m;
#pragma unroll
      for (int x = 1; x < 8; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
      const float f = lane < C ? exp2f(m - top) : 0.f;
      float L = lane < C ? f * r_l[warp * C + lane] : 0.f;
#pragma unroll
      for (int x = 1; x < 8; x <<= 1) L += __shfl_xor_sync(0xffffffffu, L, x);
      L = __shfl_sync(0xffffffffu, L, 0);
      float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float w = __shfl_sync(0xffffffffu, f, r);
        if (r >= C) break;
        const float4 v = *reinterpret_cast<const float4*>(&r_o[warp * C + r][d]);
        O.x += w * v.x; O.y += w * v.y; O.z += w * v.z; O.w += w * v.w;
      }
      store_row(a, r0 + own_g, h, d, O, L);
    }
  }
  __syncwarp();
  cluster_wait();                                           // nothing more will be written here by the others
}

}  // namespace

cudaError_t decode_qkv_attn(const void* qkv, long long ld, void* k_cache, void* v_cache, long long c_bat, long long c_tok,
                            const int* seqlens, int B, int H, int Hkv, int window, float scale, const void* cos_t,
                            const void* sin_t, const void* xn, long long ld_xn, const float* wg, const void* ve,
                            long long ld_ve, const long long* idx, int t_max, int* status, void* y, long long ldy,
                            const KvPages& pages, cudaStream_t s) {
  if (B < 1 || H % Hkv != 0 || ((ld | c_tok | c_bat | ld_ve | ldy) & 7)) return cudaErrorInvalidValue;
  if (pages.table != nullptr && (pages.page_shift < 0 || pages.page_shift > 16 || pages.max_pages <= 0 ||
                                 t_max > (pages.max_pages << pages.page_shift)))
    return cudaErrorInvalidValue;
  Args a;
  a.qkv = reinterpret_cast<const __nv_bfloat16*>(qkv); a.ld = ld;
  a.k_cache = reinterpret_cast<__nv_bfloat16*>(k_cache); a.v_cache = reinterpret_cast<__nv_bfloat16*>(v_cache);
  a.c_bat = c_bat; a.c_tok = c_tok; a.seqlens = seqlens;
  a.B = B; a.H = H; a.Hkv = Hkv; a.window = window; a.t_max = t_max; a.scale_log2 = scale * 1.4426950408889634f;
  a.cos_t = reinterpret_cast<const __nv_bfloat16*>(cos_t); a.sin_t = reinterpret_cast<const __nv_bfloat16*>(sin_t);
  a.xn = reinterpret_cast<const __nv_bfloat16*>(xn); a.ld_xn = ld_xn; a.wg = wg;
  a.ve = reinterpret_cast<const __nv_bfloat16*>(ve); a.ld_ve = ld_ve; a.idx = idx;
  a.y = reinterpret_cast<__nv_bfloat16*>(y); a.ldy = ldy; a.pages = pages; a.status = status;
  // Contiguous rows share nothing, and up to four rows are quicker each by itself (d26, 512 tokens, per step: 2 rows 903 against
  // 942 us, 4 rows 995 / 980; d12, 4 rows 331 / 360; 8 rows 998 with shared pages, 1058 without).
  const int G = pages.table == nullptr || B <= 4 ? 1 : 8;
  const int clusters = H * ((B + G - 1) / G);
  // CTAs of a cluster: one CTA per SM at most (twice that: 16 rows of d26 1347 us for 1126), up to eight for a row by itself
  // (d26, 1 row: 798 us with four, 732 with eight); four where rows share, since a cluster of eight finds room later beside the
  // kernel in front (d4, 64 rows: 219 us with eight, 183 with four; d12, 20 rows: 426 / 372).
  const int most = G == 1 ? 8 : 4;
  int C = 1;
  while (C < most && 2 * C * clusters <= sm_count()) C *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C, H, (B + G - 1) / G); cfg.blockDim = dim3(THREADS); cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = C; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
  cfg.attrs = at; cfg.numAttrs = 2;
  return G == 1 ? cudaLaunchKernelEx(&cfg, decode_qkv_attn_kernel<1>, a) : cudaLaunchKernelEx(&cfg, decode_qkv_attn_kernel<8>, a);
}

}  // namespace nc
