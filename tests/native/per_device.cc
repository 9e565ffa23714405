// Once on every device, also from several threads, and again after a failure.
#include "../../csrc/core/per_device.h"

#include <cstdio>
#include <thread>
#include <vector>

int main() {
  amem::OncePerDevice once;
  int calls = 0;
  auto well = [&] { ++calls; return 0; };
  for (int dev : {0, 0, 1, 0, 1, 63, 63}) once(dev, well);
  if (calls != 3) return std::printf("%d calls for three devices\n", calls), 1;
  if (once(2, [] { return 7; }) != 7 || once(2, well) != 0 || once(2, well) != 0 || calls != 4) return std::printf("after a failure: %d calls\n", calls), 1;
  once(64, well);
  once(64, well);
  once(-1, well);
  if (calls != 7) return std::printf("devices without a bit: %d calls\n", calls), 1;
  amem::OncePerDevice shared;
  std::atomic<int> made{0};
  std::vector<std::thread> threads;
  for (int i = 0; i < 8; ++i) threads.emplace_back([&, i] { for (int j = 0; j < 1000; ++j) shared(i % 4, [&] { made.fetch_add(1); return 0; }); });
  for (auto& t : threads) t.join();
  if (made < 4 || made > 8) return std::printf("%d times on four devices from eight threads\n", made.load()), 1;
  return 0;
}
