// Activations of the GEMM epilogues on an array, next to the forms with a division and tanhf.
#include "../../mscclpp_b200/csrc/kernels/activation.cuh"

using namespace mscclpp;

extern "C" __global__ void activations(const float* x, float* out, int n, int kind) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float v = x[i];
    if (kind == 0) out[i] = silu(v);
    else if (kind == 1) out[i] = geluTanh(v);
    else if (kind == 2) out[i] = v / (1.f + __expf(-v));
    else out[i] = 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));
  }
}
