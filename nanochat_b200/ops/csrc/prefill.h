// Host interface of GPT's prompt pass (prefill.cu). All tensors bf16 unless noted, rows dense; head dim 128.
#pragma once

#include <cuda_runtime.h>

namespace nc {

// Weights (outputs x inputs), value-embedding gate (Hkv x 12 fp32) and table (null: none), where the layer's keys and values go,
// and tokens a query looks back over.
struct PrefillLayer {
  const void *wq, *wk, *wv, *wo, *wfc, *wpr;
  const float* wg; const void* ve;
  void *k_sink, *v_sink;
  int window;
};
// x0: (B * T, C) embedded tokens. After the call the last layer's output is in x_backout when that is the backout layer, else in
// x[(layers - 1) & 1]; x_backout holds the backout layer's. Workspaces: xm, xn, xa, x[2], x_backout (B * T, C); y (.., H * 128);
// qkv (.., (H + 2 Hkv) * 128); h (.., ff); rstd (.., H + Hkv) and lse (B, H, T) fp32. cos, sin: (T, 64). Sinks: token t of row b
// at b * sink_bat + t * sink_tok elements.
struct Prefill {
  int B, T, C, H, Hkv, ff, layers, backout_layer;
  const void* x0; const long long* idx; const void *cos_t, *sin_t;
  const float *lam_r, *lam_0;
  float scale;
  long long sink_bat, sink_tok;
  void *xm, *xn, *xa, *x[2], *x_backout, *y, *qkv, *h;
  float *rstd, *lse;
  int* status;
};
cudaError_t gpt_prefill(const Prefill& p, const PrefillLayer* layers, cudaStream_t s);

}  // namespace nc
