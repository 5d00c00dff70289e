// Activations of the GEMM epilogues.
#pragma once
#include "common.cuh"

namespace pg {

// activation of the bf16 epilogue (GemmArgs::act_gelu): 1 = gelu(tanh), 2 = relu(x)^2, 6 = gelu(erf)
PG_DEVINL float epilogue_act(float x, int act) {
  if (act == 2) { const float r = fmaxf(x, 0.f); return r * r; }
  if (act == 6) return pg::gelu_erf(x);
  return gelu_tanh_fast(x);
}

// gated unit of the GEGLU epilogue (GemmArgs::act_gelu in that mode): 0 / 1 gelu_tanh(g) * u; 3 silu(g) * u; 5 relu(g) * u;
// 4 clamped: g' = min(g, c), u' = clamp(u, -c, c), g' * sigmoid(alpha * g') * (u' + 1) with c = GemmArgs::scale
PG_DEVINL float glu_act(float g, float u, int kind, float limit, float alpha) {
  if (kind == 3) return g / (1.0f + __expf(-g)) * u;
  if (kind == 4) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + __expf(-alpha * g)) * (u + 1.0f);
  }
  if (kind == 5) return fmaxf(g, 0.f) * u;
  return gelu_tanh_fast(g) * u;
}

// f(ActConst<...>) for the activation of a call: chosen once per run of elements.  A test per element made the epilogue, not the main loop, pace the products with a
// gated unit or a gelu: gate || up of 16640 tokens, 32768 x 2048: 2296 us (973 TFLOP/s), now 1500 (1489).
template <int N>
struct ActConst { static constexpr int value = N; };
template <typename Fn>
PG_DEVINL void with_act(int act, Fn&& f) {
  switch (act) {
    case 0: f(ActConst<0>{}); break;
    case 2: f(ActConst<2>{}); break;
    case 6: f(ActConst<6>{}); break;
    default: f(ActConst<1>{});
  }
}
template <typename Fn>
PG_DEVINL void with_glu(int kind, Fn&& f) {
  switch (kind) {
    case 3: f(ActConst<3>{}); break;
    case 4: f(ActConst<4>{}); break;
    case 5: f(ActConst<5>{}); break;
    default: f(ActConst<1>{});
  }
}

}  // namespace pg
