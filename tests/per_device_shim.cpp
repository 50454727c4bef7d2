// C entry of PerDevice for tests/test_per_device.py.
#include <stdexcept>
#include <thread>
#include <vector>

#include "../votca_gb300/csrc/per_device.hpp"

static vgb::PerDevice g_once;

// Runs on the given device; *count += 1 when the work is done.  Returns 1 when it threw.
extern "C" int per_device_run(int device, int fail, int *count) {
  try {
    g_once.run(device, [&] {
      if (fail) throw std::runtime_error("work");
      ++*count;
    });
  } catch (const std::runtime_error &) {
    return 1;
  }
  return 0;
}

// The same from many threads at once.
extern "C" void per_device_threads(int device, int n, int *count) {
  std::vector<std::thread> t;
  for (int i = 0; i < n; ++i) t.emplace_back([=] { per_device_run(device, 0, count); });
  for (auto &x : t) x.join();
}
