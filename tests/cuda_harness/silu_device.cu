// Device-side harness over the surrogate network's activations (silu8 of
// adaptive-gimp_b200/csrc/mlp.cu).  Test infrastructure only.
#include "../../adaptive-gimp_b200/csrc/mlp.cu"

// the plain expressions that silu8 stands for: the sigmoid's quotient (out:
// num / (1 + exp(-z)), num = z or 1) and, with deriv, SiLU's derivative of it
__global__ void k_silu(const float* z, float* fast, float* plain, long long n8, int deriv) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float v[8], a[8];
    for (int j = 0; j < 8; ++j) v[j] = z[8 * i + j];
    if (deriv)
      agimp::mlp::silu8<true>(v, a);
    else
      agimp::mlp::silu8<false>(v, a);
    for (int j = 0; j < 8; ++j) {
      float q = __fdiv_rn(deriv ? 1.f : v[j], 1.f + __expf(-v[j]));
      if (deriv) q = q * (1.f + v[j] * (1.f - q));
      fast[8 * i + j] = a[j];
      plain[8 * i + j] = q;
    }
  }
}

// z, fast, plain: device arrays of n floats, n a multiple of 8
extern "C" int h_silu(const float* z, float* fast, float* plain, long long n, int deriv) {
  k_silu<<<592, 256>>>(z, fast, plain, n / 8, deriv);
  return (int)cudaDeviceSynchronize();
}
