// Host-side harness over the 3D snow return map near rotations
// (adaptive-gimp_b200/csrc/common.cuh).  Test infrastructure only.
#include "../../adaptive-gimp_b200/csrc/common.cuh"

extern "C" void h_snow_near(float* F, float* jp, int* ok, float lo, float hi, int n) {
  for (int i = 0; i < n; ++i) ok[i] = agimp::snow_clamp_near(F + 9 * i, jp[i], lo, hi) ? 1 : 0;
}
