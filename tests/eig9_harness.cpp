// The kernels' 9x9 eigen-solver compiled for the host (tests/test_devmath_eig9.py).
#include "../bartels_gb300/csrc/devmath.cuh"

template <class T>
static void run(int n, const T *A, T *d, T *Z) {
  for (int t = 0; t < n; ++t) {
    T M[45];
    for (int i = 0; i < 9; ++i)
      for (int j = 0; j <= i; ++j) M[bartels::p9(i, j)] = A[81 * t + i + 9 * j];
    bartels::eig9p(M, d + 9 * t, Z + 81 * t);
  }
}
extern "C" void eig9_f32(int n, const float *A, float *d, float *Z) { run(n, A, d, Z); }
extern "C" void eig9_f64(int n, const double *A, double *d, double *Z) { run(n, A, d, Z); }
