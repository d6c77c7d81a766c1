// Activations by code, 32-bit (norm_act.cu, gemm_grouped.cu)
#pragma once
#include "common.cuh"

enum : int { ACT_SILU = 0, ACT_GELU = 1, ACT_GELU_TANH = 2, ACT_RELU = 3, ACT_GELU_NEW = 4, ACT_GELU_FAST = 5,
             ACT_QUICK_GELU = 6, ACT_RELU2 = 7 };

template <int ACT> VB_DEVICE float act_fn(float x) {
  if (ACT == ACT_SILU) return x / (1.f + __expf(-x));
  if (ACT == ACT_GELU) return 0.5f * x * (1.f + erff(x * 0.70710678118654752f));
  if (ACT == ACT_GELU_TANH || ACT == ACT_GELU_NEW)
    return 0.5f * x * (1.f + tanhf(0.7978845608028654f * (x + 0.044715f * x * x * x)));
  if (ACT == ACT_GELU_FAST) return 0.5f * x * (1.f + tanhf(x * 0.7978845608f * (1.f + 0.044715f * x * x)));
  if (ACT == ACT_QUICK_GELU) return x / (1.f + __expf(-1.702f * x));
  if (ACT == ACT_RELU2) { float r = fmaxf(x, 0.f); return r * r; }
  return fmaxf(x, 0.f);
}
