// Linear layers of up to 64 rows (decode steps, short prompts) on the 5th-generation tensor cores:
//
//   y[b, n] = epi( sum_k x'[b, k] W[n, k] ) + aux[b, n],   x' = x or rmsnorm(x)
//
// A step reads every weight once, so the kernel is built around weight bytes in flight and a short chain behind the wait on
// the kernel in front. The weights are the 128-row operand of the MMA (tcgen05, M = 128 outputs), the step's rows the narrow
// one (N = 16, 32 or 64): 16 KB of weights per 2 to 8 KB of activations. The CTAs of a cluster share the reduction of a tile,
// so that even the 13 tiles of a 1664-wide output put 104 SMs to work; each pushes its part of a row to the CTA that sums it
// (st.async, four rows per packet, counted on an mbarrier), and the row statistic of the norm rides along
// (rmsnorm(x) . w = rstd * (x . w)).
//
// A CTA requests as many weight tiles as its ring holds before it waits for the kernel in front (programmatic dependent
// launch). The ring stays below half of an SM's shared memory, so that the next kernel's CTAs move in beside this one's.
//
// What bounds it, d26 on a B200: a layer's four products take 4.4 (QKV), 3.0, 5.0 and 8.1 us behind their waits for 2.5, 0.8,
// 3.3 and 3.3 us of weight bytes; the rest is the chain TMA - MMA - push - store and, where K per CTA exceeds the ring (MLP
// down: 13 blocks of 64 over 5 stages), the latency of its refills. Per step of d26, 512 tokens back: 8 rows 2046 us with a
// fp32 matrix-vector kernel, 1153 now; 64 rows 3060 us with 128-row tiles of activations and no split, 2165 now.
#include "decode.h"
#include "host_utils.cuh"
#include "ptx.cuh"

namespace nc {

namespace {

constexpr int BM = 128;                    // outputs of a tile
constexpr int BK = 64;                     // one 128-byte swizzle row of bf16
constexpr int W_BYTES = BM * 128;
constexpr int MAX_SPLIT = 8;               // CTAs of a portable cluster
constexpr int THREADS = 192;               // TMA warp, MMA warp, four epilogue warps
constexpr float kEps = 1.1920929e-07f;     // fp32 machine epsilon, as F.rms_norm(eps=None)

template <int R>
struct Cfg {
  static constexpr int STAGE = W_BYTES + R * 128;
  static constexpr int GROUPS = R / 4 < MAX_SPLIT ? MAX_SPLIT : R / 4;    // most parts a CTA receives, each four rows of a tile
  static constexpr int PARTS = GROUPS * BM * 16;
  static constexpr int STAGES = (112 * 1024 - PARTS) / STAGE;
  static constexpr int TMEM_COLS = R < 32 ? 32 : R;
  static constexpr int SMEM = STAGES * STAGE + PARTS + 1024;
  static_assert(SMEM <= 113 * 1024, "two CTAs of an SM");
};

struct Args {
  int B, N, K, splits, norm_input, act, mul_aux, head_cols;
  const __nv_bfloat16* aux; long long ldaux;
  __nv_bfloat16* out; long long ldo;
  RowsMix mix;
  const __nv_bfloat16* x; long long ldx;
  __nv_bfloat16* xn_head; long long ldxn;
  float* logits; long long ldl; float softcap;
  int* status;
};

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Into a CTA's shared memory, counted on a barrier of that CTA.
__device__ __forceinline__ void st_async(uint32_t addr, float v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
               ::"r"(addr), "r"(__float_as_uint(v)), "r"(bar) : "memory");
}
__device__ __forceinline__ void st_async4(uint32_t addr, const uint32_t* v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
               ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(bar) : "memory");
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16(v)); }

template <int R>
__global__ void __launch_bounds__(THREADS)
rows_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Args a) {
  using C = Cfg<R>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[C::STAGES], empty[C::STAGES], acc_full, parts_full;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ __align__(16) float s_ss[4 * C::GROUPS];      // like `parts`, one value per row
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  volatile int* abort_flag = &abort_word;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = a.splits, rank = blockIdx.x % S, tile = blockIdx.x / S, n0 = tile * BM;
  const int blocks = (a.K + BK - 1) / BK;
  // Four rows at a time are summed by the CTA that owns them: rows 4 g .. 4 g + 3 by CTA g % S, as the g / S-th of `mine`.
  const int groups = (a.B + 3) / 4, shift = 31 - __clz(S), per = (groups + S - 1) >> shift, mine = (groups - rank + S - 1) >> shift;
  float4* parts = reinterpret_cast<float4*>(ring + C::STAGES * C::STAGE);     // [CTA of the cluster][group of this CTA][output]
  const int kb0 = rank * blocks / S, nkb = (rank + 1) * blocks / S - kb0;

  if (tid == 0) {
    for (int s = 0; s < C::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1 + (a.norm_input ? 4 : 0)); }
    mbar_init(&acc_full, 1);
    mbar_init(&parts_full, 1);
    abort_word = 0;
    fence_mbar_init();
    mbar_arrive_expect_tx(&parts_full, S * mine * (BM * 16 + (a.norm_input ? 16 : 0)));
    // the weights do not depend on the kernel in front
    const int ahead = min(C::STAGES, nkb);
    for (int i = 0; i < ahead; ++i) {
      mbar_arrive_expect_tx(&full[i], C::STAGE);
      tma_load_2d(ring + i * C::STAGE, &tmW, &full[i], (kb0 + i) * BK, n0);
    }
    tma_prefetch_desc(&tmX);
    pdl_trigger();
  }
  if (warp == 1) { tmem_alloc(&tmem_slot, C::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  if (S > 1) cluster_sync_all();                             // the barriers that the others count on are ready
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      const int ahead = min(C::STAGES, nkb);
      for (int i = 0; i < ahead; ++i) tma_load_2d(ring + i * C::STAGE + W_BYTES, &tmX, &full[i], (kb0 + i) * BK, 0);
      for (int i = ahead; i < nkb; ++i) {
        const int s = i % C::STAGES;
        if (!mbar_wait(&empty[s], ((i / C::STAGES) & 1) ^ 1, abort_flag, a.status, ST_WAIT_EMPTY, tile)) break;
        mbar_arrive_expect_tx(&full[s], C::STAGE);
        tma_load_2d(ring + s * C::STAGE, &tmW, &full[s], (kb0 + i) * BK, n0);
        tma_load_2d(ring + s * C::STAGE + W_BYTES, &tmX, &full[s], (kb0 + i) * BK, 0);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(BM, R, false, false);
      bool ok = true;
      for (int i = 0; i < nkb; ++i) {
        const int s = i % C::STAGES;
        if (!mbar_wait(&full[s], (i / C::STAGES) & 1, abort_flag, a.status, ST_WAIT_FULL, tile)) { ok = false; break; }
        tc_fence_after();
        const uint32_t w_addr = smem_u32(ring + s * C::STAGE), x_addr = w_addr + W_BYTES;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k)
          mma_f16(tmem, umma_desc_sw128(w_addr + k * 32, 16, 1024), umma_desc_sw128(x_addr + k * 32, 16, 1024), idesc, (i | k) != 0);
        mma_commit(&empty[s]);
      }
      if (ok) mma_commit(&acc_full);
    }
  } else {
    const int t = tid - 64, quad = warp & 3;
    bool ok = true;
    if (a.norm_input) {
      // sums of squares of the rows over this CTA's share of K: eight lanes read a row's 128 bytes (swizzling only
      // permutes them)
      float ss[R / 16];
#pragma unroll
      for (int j = 0; j < R / 16; ++j) ss[j] = 0.f;
      for (int i = 0; i < nkb; ++i) {
        const int s = i % C::STAGES;
        if (!mbar_wait(&full[s], (i / C::STAGES) & 1, abort_flag, a.status, ST_WAIT_FULL, tile)) { ok = false; break; }
        const uint8_t* x = ring + s * C::STAGE + W_BYTES + (t >> 3) * 128 + (t & 7) * 16;
#pragma unroll
        for (int j = 0; j < R / 16; ++j) {
          const uint4 v = *reinterpret_cast<const uint4*>(x + j * 16 * 128);
          const float2 p = unpack_bf16(v.x), q = unpack_bf16(v.y), r = unpack_bf16(v.z), u = unpack_bf16(v.w);
          ss[j] += p.x * p.x + p.y * p.y + q.x * q.x + q.y * q.y + r.x * r.x + r.y * r.y + u.x * u.x + u.y * u.y;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[s]);
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < R / 16; ++j) {
#pragma unroll
        for (int w = 4; w > 0; w >>= 1) ss[j] += __shfl_xor_sync(0xffffffffu, ss[j], w);
        const int b = (t >> 3) + 16 * j, g = b >> 2, owner = g & (S - 1);
        if (ok && (t & 7) == 0 && g < groups)
          st_async(map_to_cta(smem_u32(&s_ss[(rank * per + (g >> shift)) * 4 + (b & 3)]), owner), ss[j],
                   map_to_cta(smem_u32(&parts_full), owner));
      }
    }
    if (ok) ok = mbar_wait(&acc_full, 0, abort_flag, a.status, ST_WAIT_TMEM_FULL, tile);
    __syncwarp();
    const int m = quad * 32 + lane, n = n0 + m;
    const bool live = n < a.N, mix = a.mix.xm != nullptr, head = a.xn_head != nullptr && n < a.head_cols;
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after();
      const uint32_t part = smem_u32(parts) + (rank * per * BM + m) * 16, bar = smem_u32(&parts_full);
#pragma unroll
      for (int c = 0; c < R / 16; ++c) {
        if (c * 4 >= groups) break;
        uint32_t v[16];
        tmem_ld16(tmem + (static_cast<uint32_t>(quad * 32) << 16) + c * 16, v);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int g = c * 4 + j, owner = g & (S - 1);
          if (g < groups) st_async4(map_to_cta(part + (g >> shift) * (BM * 16), owner), v + 4 * j, map_to_cta(bar, owner));
        }
      }
      tc_fence_before();
    }
    __syncwarp();
    if (S > 1) cluster_arrive();                             // this warp has sent its share
    const float lam_r = mix ? a.mix.lam_r[a.mix.layer] : 0.f, lam_0 = mix ? a.mix.lam_0[a.mix.layer] : 0.f;
    if (mine > 0 && mbar_wait(&parts_full, 0, abort_flag, a.status, ST_WAIT_PEER, tile) && live) {
      for (int i = 0; i < mine; ++i) {
        const int b0 = (rank + (i << shift)) * 4;
        float y[4] = {0.f, 0.f, 0.f, 0.f}, q[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int r = 0; r < MAX_SPLIT; ++r) {
          if (r >= S) break;
          const float4 p = parts[(r * per + i) * BM + m];
          y[0] += p.x; y[1] += p.y; y[2] += p.z; y[3] += p.w;
          if (a.norm_input) {
            const float4 s4 = *reinterpret_cast<const float4*>(&s_ss[(r * per + i) * 4]);
            q[0] += s4.x; q[1] += s4.y; q[2] += s4.z; q[3] += s4.w;
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int b = b0 + u;
          if (b >= a.B) break;
          float v = y[u];
          if (a.norm_input) {
            const float rstd = rsqrtf(q[u] / a.K + kEps);
            v *= rstd;
            if (head) a.xn_head[b * a.ldxn + n] = __float2bfloat16(__bfloat162float(a.x[b * a.ldx + n]) * rstd);
          }
          if (a.act != ROWS_LINEAR) v = fmaxf(v, 0.f);
          if (a.act == ROWS_RELU2) v *= v;
          if (a.aux != nullptr) {
            const float x = __bfloat162float(a.aux[b * a.ldaux + n]);
            v = a.mul_aux ? v * x : v + x;
          }
          if (a.out != nullptr) a.out[b * a.ldo + n] = __float2bfloat16(v);
          if (mix) {
            const float x0 = __bfloat162float(a.mix.x0[b * a.mix.ldx0 + n]);
            a.mix.xm[b * a.mix.ldxm + n] = __float2bfloat16(lam_r * round_bf16(v) + lam_0 * x0);
          }
          if (a.logits != nullptr) a.logits[b * a.ldl + n] = a.softcap > 0.f ? a.softcap * tanhf(v / a.softcap) : v;
        }
      }
    }
  }
  __syncwarp();
  if (S > 1) {
    if (warp < 2) cluster_arrive();
    cluster_wait();                                          // nothing more will be written here by the others
  }
  __syncthreads();
  if (*abort_flag) {
    // give copies that are still in flight time to land before shared memory is released
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, C::TMEM_COLS); }
}

template <int R>
cudaError_t launch(const CUtensorMap& tmW, const CUtensorMap& tmX, const Args& a, bool overlap, cudaStream_t s) {
  static PerDeviceOnce configured;
  cudaError_t e = configured.once([] {
    return cudaFuncSetAttribute(rows_gemm_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<R>::SMEM);
  });
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((a.N + BM - 1) / BM * a.splits); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = Cfg<R>::SMEM; cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = a.splits; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at; cfg.numAttrs = overlap ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, rows_gemm_kernel<R>, tmW, tmX, a);
}

}  // namespace

cudaError_t rows_gemm(const RowsGemm& g, cudaStream_t s) {
  if (g.B < 1 || g.B > kRowsGemmMax || g.N < 1 || g.K < 8 || ((g.K | g.ldx | g.ldw) & 7) ||
      ((reinterpret_cast<uintptr_t>(g.x) | reinterpret_cast<uintptr_t>(g.W)) & 15))
    return cudaErrorInvalidValue;
  const int R = g.B <= 16 ? 16 : g.B <= 32 ? 32 : 64;
  const int tiles = (g.N + BM - 1) / BM, blocks = (g.K + BK - 1) / BK;
  // As many CTAs per tile as it takes to give every SM one. Half as many for the wide products (one wave with the kernel in
  // front still resident) made the d26 step of 1 to 64 rows 4 to 7 % slower: longer refill chains.
  int splits = 1;
  while (splits < MAX_SPLIT && tiles * splits < sm_count() && 2 * splits <= blocks) splits *= 2;
  Args a = {};
  a.B = g.B; a.N = g.N; a.K = g.K; a.splits = splits; a.norm_input = g.norm_input; a.act = g.act; a.mul_aux = g.mul_aux;
  a.aux = reinterpret_cast<const __nv_bfloat16*>(g.aux); a.ldaux = g.ldaux;
  a.out = reinterpret_cast<__nv_bfloat16*>(g.out); a.ldo = g.ldo;
  a.mix = g.mix;
  a.x = reinterpret_cast<const __nv_bfloat16*>(g.x); a.ldx = g.ldx;
  a.xn_head = reinterpret_cast<__nv_bfloat16*>(g.xn_head); a.ldxn = g.ldxn; a.head_cols = g.head_cols;
  a.logits = g.logits; a.ldl = g.ldl; a.softcap = g.softcap;
  a.status = g.status;
  CUtensorMap tmW, tmX;
  const uint64_t wd[2] = {(uint64_t)g.K, (uint64_t)g.N}, xd[2] = {(uint64_t)g.K, (uint64_t)g.B};
  const uint64_t ws[1] = {(uint64_t)g.ldw * 2}, xs[1] = {(uint64_t)g.ldx * 2};
  const uint32_t wb[2] = {BK, BM}, xb[2] = {BK, (uint32_t)R};
  if (!make_tmap(&tmW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, g.W, wd, ws, wb) ||
      !make_tmap(&tmX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, g.x, xd, xs, xb))
    return cudaErrorInvalidValue;
  const bool o = g.overlap != 0;
  return R == 16 ? launch<16>(tmW, tmX, a, o, s) : R == 32 ? launch<32>(tmW, tmX, a, o, s) : launch<64>(tmW, tmX, a, o, s);
}

}  // namespace nc
