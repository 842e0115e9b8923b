// OncePerDevice from eight threads at once (built with the thread sanitizer): nobody goes on before the work was done,
// a failure is tried again, a device beyond the marks does the work each time.
#include "../../systemds_b200/csrc/cla_once.h"
#include <cstdio>
#include <thread>
#include <vector>

int main() {
  static cla::OncePerDevice once;
  static std::atomic<int> ready[4], calls[4], bad{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; t++)
    threads.emplace_back([] {
      for (int i = 0; i < 4000; i++) {
        const int d = i % 4;
        if (once(d, [&]() -> int64_t { calls[d]++; ready[d] = 1; return 0; }) < 0) bad++;
        if (!ready[d]) bad++;
      }
    });
  for (auto& t : threads) t.join();
  for (int d = 0; d < 4; d++)
    if (calls[d] < 1 || calls[d] > 8) bad++;
  int n = 0;
  auto fails = [&]() -> int64_t { return ++n == 1 ? -5 : 0; };
  if (once(9, fails) != -5 || once(9, fails) != 0 || once(9, fails) != 0 || n != 2) bad++;
  n = 1;
  if (once(64, fails) != 0 || once(64, fails) != 0 || n != 3) bad++;
  printf("%s\n", bad ? "MISMATCH" : "ok");
  return bad ? 1 : 0;
}
