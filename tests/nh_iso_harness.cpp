// The isochoric Neo-Hookean energy compiled for the host (tests/test_devmath_nh_iso.py).
#include "../bartels_gb300/csrc/devmath.cuh"

extern "C" void nh_iso(int n, const double *H, const double *pv, double *psi) {
  for (int i = 0; i < n; ++i) psi[i] = bartels::psi_model_disp<double>(bartels::MODEL_NH_ISO, H + 9 * i, pv);
}
