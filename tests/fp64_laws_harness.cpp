// The FP64 pieces of the energy and stress kernels compiled for the host
// (tests/test_devmath_fp64_laws.py).
#include "../bartels_gb300/csrc/devmath.cuh"

extern "C" {
void jlog(int n, const double *j, double *out) {
  for (int i = 0; i < n; ++i) out[i] = bartels::j_minus_log1p(j[i]);
}
void corot(int n, const double *F, const double *pv, double *psi, double *P, int *polar) {
  double R[9];
  for (int i = 0; i < n; ++i) {
    psi[i] = bartels::psi_model<double>(bartels::MODEL_COROT, F + 9 * i, pv);
    bartels::pk1_model<double>(bartels::MODEL_COROT, F + 9 * i, pv, P + 9 * i);
    polar[i] = bartels::polar_rot<2>(F + 9 * i, R);
  }
}
}
