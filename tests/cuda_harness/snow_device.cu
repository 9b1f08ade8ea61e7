// Device-side harness over the 3D snow return map near rotations
// (snow_clamp_near of adaptive-gimp_b200/csrc/common.cuh), whose device build
// uses the hardware's reciprocal root and quotient.  Test infrastructure only.
#include "../../adaptive-gimp_b200/csrc/common.cuh"

__global__ void k_snow(float* F, float* jp, int* ok, float lo, float hi, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float f[9], j = jp[i];
    for (int k = 0; k < 9; ++k) f[k] = F[9 * i + k];
    ok[i] = agimp::snow_clamp_near(f, j, lo, hi) ? 1 : 0;
    for (int k = 0; k < 9; ++k) F[9 * i + k] = f[k];
    jp[i] = j;
  }
}

// F [n][9], jp [n], ok [n]: device arrays
extern "C" int h_snow_near(float* F, float* jp, int* ok, float lo, float hi, int n) {
  k_snow<<<(n + 127) / 128, 128>>>(F, jp, ok, lo, hi, n);
  return (int)cudaDeviceSynchronize();
}
