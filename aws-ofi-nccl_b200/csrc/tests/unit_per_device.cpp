// What is set up once per device: every device of the process gets its turn, a failure is no success, and devices beyond the table are
// set up every time.
#include <thread>
#include <vector>
#include "../kernels/per_device.h"
#include "test_util.h"
int main() {
  b200::OncePerDevice once;
  std::vector<int> calls(128, 0);
  auto set = [&](int device, int rc = 0) { return once.run(device, [&] { ++calls[device + 1]; return rc; }); };
  for (int round = 0; round < 3; ++round)
    for (int device : {0, 1, 15, 16, 63}) CHECK_EQ(set(device), 0);   // the second device's turn does not depend on the first's
  for (int device : {0, 1, 15, 16, 63}) CHECK_EQ(calls[device + 1], 1);
  CHECK_EQ(set(2, 700), 700);   // tried again until it works
  CHECK_EQ(set(2), 0);
  CHECK_EQ(set(2, 700), 0);
  CHECK_EQ(calls[3], 2);
  for (int i = 0; i < 2; ++i) {
    CHECK_EQ(set(64), 0);
    CHECK_EQ(set(-1), 0);
  }
  CHECK_EQ(calls[65], 2);
  CHECK_EQ(calls[0], 2);
  b200::OncePerDevice other;   // each kernel has a table of its own
  CHECK_EQ(other.run(0, [] { return 5; }), 5);
  std::atomic<int> runs{0};
  std::vector<std::thread> threads;
  for (int i = 0; i < 8; ++i)
    threads.emplace_back([&] {
      for (int device = 0; device < 64; ++device) other.run(device, [&] { ++runs; return 0; });
    });
  for (auto& t : threads) t.join();
  CHECK(runs >= 64 && runs <= 8 * 64);
  const int before = runs;
  for (int device = 0; device < 64; ++device) CHECK_EQ(other.run(device, [&] { ++runs; return 0; }), 0);
  CHECK_EQ(runs.load(), before);
  TEST_MAIN_END();
}
