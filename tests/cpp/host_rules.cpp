// Host-side rules of the engine, run without a device:
//   host_rules step   the counters follow the steps that were made
//   host_rules grid   threads that launch a kernel form first, together
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

#include "resident_grid.h"
#include "step_record.h"

namespace {

// Steps as a segment runs them: forces, the step's kernel, and its finishing
// launch anywhere between that kernel and the next one: before the next
// step's forces, or after they have set the error word.
int step() {
  for (int bad = 0; bad <= 6; ++bad) {    // the step whose forces fail (6: none)
    for (int late = 0; late < 2; ++late) {  // the finishing launch runs late
      apo::StepRecord rec{0u};
      unsigned err = 0;
      long long moved = 0, counted = 0;
      bool pending = false;
      for (int k = 0; k < 6; ++k) {
        if (pending && !late) counted += apo::take_step(rec);
        if (k == bad) err = 16;  // the forces of step k
        if (pending && late) counted += apo::take_step(rec);
        pending = false;
        if (!err) {
          ++moved;
          apo::record_step(rec);
        }
        pending = true;
      }
      counted += apo::take_step(rec);
      if (moved != (bad < 6 ? bad : 6) || counted != moved) {
        std::printf("step %d late %d: moved %lld counted %lld\n", bad, late, moved, counted);
        return 1;
      }
    }
  }
  return 0;
}

int grid() {
  std::atomic<int> asked{0}, ready{0}, wrong{0};
  auto launch = [&] {
    ++ready;
    while (ready < 8) std::this_thread::yield();
    const apo::ResidentGrid &g = apo::resident_grid([&asked] {
      ++asked;
      apo::ResidentGrid r;
      std::this_thread::sleep_for(std::chrono::milliseconds(20));
      r.full = 592;
      std::this_thread::sleep_for(std::chrono::milliseconds(20));
      r.shared = 444;
      return r;
    });
    if (g.full != 592 || g.shared != 444) ++wrong;
  };
  std::vector<std::thread> t;
  for (int k = 0; k < 8; ++k) t.emplace_back(launch);
  for (auto &x : t) x.join();
  if (asked != 1 || wrong != 0) {
    std::printf("asked %d times, %d threads saw half an answer\n", asked.load(), wrong.load());
    return 1;
  }
  return 0;
}

}  // namespace

int main(int argc, char **argv) {
  if (argc == 2 && !std::strcmp(argv[1], "step")) return step();
  if (argc == 2 && !std::strcmp(argv[1], "grid")) return grid();
  return 2;
}
