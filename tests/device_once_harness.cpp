// The per-device flag compiled for the host (tests/test_device_once.py).
#include "../bartels_gb300/csrc/device_once.h"

#include <thread>
#include <vector>

extern "C" {
// whether device d is pending after devices 0 .. n-1 of `set` have been set
int pending_after(int n, const int *set, int d) {
  bartels::DeviceOnce f;
  for (int i = 0; i < n; ++i) f.set(set[i]);
  return f.pending(d);
}
// devices 0 .. 63, set from one thread each; those still pending
int pending_after_threads() {
  bartels::DeviceOnce f;
  std::vector<std::thread> t;
  for (int d = 0; d < 64; ++d) t.emplace_back([&f, d] { f.set(d); });
  for (auto &x : t) x.join();
  int left = 0;
  for (int d = 0; d < 64; ++d) left += f.pending(d);
  return left;
}
}
