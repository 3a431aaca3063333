// The assembly launch's rule compiled for the host (tests/test_hess_shape.py).
#include "../bartels_gb300/csrc/hess_shape.h"

extern "C" void shape(long long vertices, long long chunks, long long sms, int cheap, int tuned, int *out) {
  const bartels::HessShape s = bartels::hess_shape(vertices, chunks, sms, cheap != 0, tuned);
  out[0] = s.chunk;
  out[1] = s.lanes;
}
