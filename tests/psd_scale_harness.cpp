// The PSD projection's slow path in FP32 compiled for the host (tests/test_devmath_psd_scale.py).
#include "../bartels_gb300/csrc/devmath.cuh"

// blocks of nodes 1 .. 3 of the projected matrix (packed 9x9) and the thin QR's Q (4 x 3)
extern "C" void psd_nodes(const float *F, const float *pv, const float *dphi9, float tol, float *K, float *Q) {
  float phi[4][3], R[9];
  for (int d = 0; d < 3; ++d) {
    phi[0][d] = 0.f;
    for (int a = 1; a < 4; ++a) {
      phi[a][d] = dphi9[3 * (a - 1) + d];
      phi[0][d] -= phi[a][d];
    }
  }
  bartels::psd_eig_K(bartels::LawStVK<float>(F, pv), phi, tol, K);
  bartels::qr_phi(phi, reinterpret_cast<float(*)[3]>(Q), R);
}
