// GPT's layers over a prompt, for inference: the kernels of the training forward launched from one call. From Python a layer
// cost about 170 us of host time (tensor bookkeeping around eleven launches), which set the time of every prompt below some
// 1500 tokens: d12, 45 tokens 2.13 ms for 1.1 ms of kernels, now 1.36; d26, 20 tokens 4.43 / 2.66, 2000 tokens 7.18 / 6.79. Keys and values go to the cache in one copy of their common span
// (two strided tensor copies before: 15.4 us a layer at 2000 x 1664, 13 MB). Prompts of up to 64 tokens run the decode step's
// products, with norms and the next layer's mix inside them.
#include "prefill.h"

#include "attention.h"
#include "decode.h"
#include "fused.h"
#include "gemm.h"
#include "host_utils.cuh"

namespace nc {

namespace {

// [k heads | v heads] of every token's projections to the cache: one 16-byte piece per thread.
__global__ void __launch_bounds__(256)
kv_sink_kernel(const uint4* __restrict__ kv, long long ld, int T, int pieces, uint4* __restrict__ k, uint4* __restrict__ v,
               long long bat, long long tok, long long total) {
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const long long m = i / (2 * pieces);
    const int p = (int)(i - m * 2 * pieces);
    const long long to = (m / T) * bat + (m % T) * tok;
    const uint4 x = kv[m * ld + p];
    if (p < pieces) k[to + p] = x; else v[to + p - pieces] = x;
  }
}

#define TRY(expr) do { cudaError_t e_ = (expr); if (e_ != cudaSuccess) return e_; } while (0)

}  // namespace

cudaError_t gpt_prefill(const Prefill& p, const PrefillLayer* layers, cudaStream_t s) {
  const int M = p.B * p.T, C = p.C, nq = p.H * 128, nkv = p.Hkv * 128, width = nq + 2 * nkv;
  if (M < 1 || (C & 7) || p.H % p.Hkv != 0) return cudaErrorInvalidValue;
  const bool few = M <= kRowsGemmMax;
  char* const qkv = reinterpret_cast<char*>(p.qkv);
  // out = act(x W^T) + aux; with few rows also the norm of x, and the next layer's mix in place of a plain result
  auto linear = [&](const void* x, int K, const void* W, int N, void* out, long long ldo, const void* aux, bool relu2, bool norm, const RowsMix& mix,
                    void* xn_head) -> cudaError_t {
    if (few) {
      RowsGemm g{};
      g.x = x; g.ldx = K; g.W = W; g.ldw = K; g.B = M; g.N = N; g.K = K;
      g.norm_input = norm; g.act = relu2 ? ROWS_RELU2 : ROWS_LINEAR; g.overlap = 1;
      g.aux = aux; g.ldaux = N; g.out = out; g.ldo = ldo; g.mix = mix;
      g.xn_head = xn_head; g.ldxn = C; g.head_cols = xn_head != nullptr ? 16 : 0;
      g.status = p.status;
      return rows_gemm(g, s);
    }
    GemmDesc d{};
    d.A = x; d.lda = K; d.B = W; d.ldb = K; d.C = out; d.ldc = ldo; d.aux = aux; d.ldaux = N;
    d.M = M; d.N = N; d.K = K; d.batch = 1; d.alpha = 1.f; d.beta = aux != nullptr ? 1.f : 0.f; d.epi = relu2 ? EPI_RELU2 : EPI_LINEAR;
    return gemm_bf16(d, p.status, s);
  };
  const void* x = p.x0;
  for (int i = 0; i < p.layers; ++i) {
    const PrefillLayer& l = layers[i];
    const bool last = i + 1 == p.layers, keep = last || i == p.backout_layer;
    if (!few || i == 0) TRY(mixnorm_fwd(x, p.x0, p.lam_r, p.lam_0, i, p.xm, p.xn, nullptr, M, C, s));
    const void* in = few ? p.xm : p.xn;
    void* head = few && l.ve != nullptr ? p.xn : nullptr;
    const char *wq = reinterpret_cast<const char*>(l.wq), *wk = reinterpret_cast<const char*>(l.wk), *wv = reinterpret_cast<const char*>(l.wv);
    if (wk == wq + 2ll * nq * C && wv == wk + 2ll * nkv * C) {                 // one matrix
      TRY(linear(in, C, wq, width, qkv, width, nullptr, false, true, {}, head));
    } else {
      TRY(linear(in, C, wq, nq, qkv, width, nullptr, false, true, {}, head));
      TRY(linear(in, C, wk, nkv, qkv + 2ll * nq, width, nullptr, false, true, {}, nullptr));
      TRY(linear(in, C, wv, nkv, qkv + 2ll * (nq + nkv), width, nullptr, false, true, {}, nullptr));
    }
    TRY(qkv_post_fwd(qkv, width, p.H, p.Hkv, p.cos_t, p.sin_t, p.T, p.rstd, l.ve != nullptr ? p.xn : nullptr, C, l.wg, l.ve, p.idx, M, s));
    {
      const long long total = 2ll * M * nkv / 8;
      const int grid = (int)((total + 255) / 256 < 8ll * sm_count() ? (total + 255) / 256 : 8ll * sm_count());
      kv_sink_kernel<<<grid, 256, 0, s>>>(reinterpret_cast<const uint4*>(qkv + 2ll * nq), width / 8, p.T, nkv / 8, reinterpret_cast<uint4*>(l.k_sink),
                                          reinterpret_cast<uint4*>(l.v_sink), p.sink_bat / 8, p.sink_tok / 8, total);
      TRY(cudaGetLastError());
    }
    AttnDesc a{};
    a.B = p.B; a.Tq = a.Tk = p.T; a.H = p.H; a.Hkv = p.Hkv; a.D = 128;
    a.q = qkv; a.k = qkv + 2ll * nq; a.v = qkv + 2ll * (nq + nkv); a.o = p.y; a.lse = p.lse;
    a.q_tok = a.k_tok = a.v_tok = width; a.o_tok = nq;
    a.q_bat = a.k_bat = a.v_bat = (long long)p.T * width; a.o_bat = (long long)p.T * nq;
    a.q_head = a.k_head = a.v_head = a.o_head = 128;
    a.window = l.window >= 0 && l.window < p.T ? l.window : -1;
    a.scale = p.scale;
    TRY(attention_fwd(a, p.status, s));
    TRY(linear(p.y, nq, l.wo, C, p.xa, C, p.xm, false, false, {}, nullptr));
    if (!few) TRY(norm_fwd(p.xa, p.xn, nullptr, M, C, s));
    TRY(linear(few ? p.xa : p.xn, C, l.wfc, p.ff, p.h, p.ff, nullptr, true, true, {}, nullptr));
    void* out = i == p.backout_layer ? p.x_backout : p.x[i & 1];
    RowsMix mix;
    if (few && !last)
      mix = {p.lam_r, p.lam_0, i + 1, reinterpret_cast<const __nv_bfloat16*>(p.x0), C, reinterpret_cast<__nv_bfloat16*>(p.xm), C};
    TRY(linear(p.h, p.ff, l.wpr, C, !few || keep ? out : nullptr, C, p.xa, false, false, mix, nullptr));
    x = out;
  }
  return cudaSuccess;
}

}  // namespace nc
