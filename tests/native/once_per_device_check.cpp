/* OncePerDevice (plume_b200/csrc/once_per_device.cuh, compiled here as it is): set up once on every device, again after a
 * failure, once among threads that meet. Prints what was wrong, nothing when all is right. */
#include <stdio.h>

#include <atomic>
#include <chrono>
#include <thread>
#include <vector>

#include "once_per_device.cuh"

int main() {
  plume::OncePerDevice once;
  for (int device : {0, 1, 7, 63}) {
    int calls = 0;
    for (int n = 0; n < 3; ++n)
      if (once.run(device, [&] { return ++calls, 0; }) != 0) printf("device %d: status\n", device);
    if (calls != 1) printf("device %d: set up %d times\n", device, calls);
  }
  int calls = 0;
  for (int n = 0; n < 3; ++n) {
    const int status = once.run(2, [&] { return ++calls < 2 ? -3 : 0; });
    if (status != (n == 0 ? -3 : 0)) printf("call %d after a failure: status %d\n", n, status);
  }
  if (calls != 2) printf("after a failure: set up %d times\n", calls);
  calls = 0;
  for (int n = 0; n < 3; ++n) once.run(64, [&] { return ++calls, 0; });
  if (calls != 3) printf("device 64: set up %d times\n", calls);
  std::atomic<int> at_work{0}, ready{0}, early{0};
  std::vector<std::thread> threads;
  for (int n = 0; n < 8; ++n)
    threads.emplace_back([&] {
      once.run(3, [&] {
        ++at_work;
        std::this_thread::sleep_for(std::chrono::milliseconds(20));
        ready = 1;
        return 0;
      });
      if (!ready) ++early;
    });
  for (std::thread& t : threads) t.join();
  if (at_work != 1 || early != 0) printf("threads: set up %d times, %d went ahead\n", at_work.load(), early.load());
  return 0;
}
