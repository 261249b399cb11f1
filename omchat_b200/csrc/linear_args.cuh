// What describes a product of omc_linear to its kernels, and its activations.
#pragma once
#include "seq_common.cuh"

namespace omc {

struct LinearArgs {
  const void* X;
  const void* W;
  void* Y;
  long long ldx, sx, ldw, sw, ldy, sy, group_stride;
  const int32_t* tile_group;
  int M, N, K;
  float alpha;
  int act;
  const void* bias;  // [N] of the weights' dtype, added before the activation (NULL: none); batch item b reads bias + b * sbias
  long long sbias;
  const void* gate;  // [M, .] of gate_dt: outputs are multiplied by sigmoid(gate[m * ldg + b * sg + n]) (NULL: none)
  int gate_dt;
  long long ldg, sg;
};

__device__ __forceinline__ float apply_act(float z, int act) {
  if (act == OMC_ACT_RELU2) {
    z = fmaxf(z, 0.f);
    return z * z;
  }
  if (act == OMC_ACT_GELU_TANH) return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
  if (act == OMC_ACT_GELU_ERF) return 0.5f * z * (1.f + erff(z * 0.70710678118654752f));
  return z;
}

}  // namespace omc
