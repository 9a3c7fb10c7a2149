// Host check of end_interval (lgpu_interval_end.h), compiled with g++ by
// test_interval_end.py: a block of host threads, of which those of one warp (not
// thread 0) come late.
//
// Usage: interval_end_check threads late_warp go pos n e_max sampled. Prints "ok" or
// what differs from the same done by one thread.
#include <barrier>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>

#include "lgpu_interval_end.h"

using namespace lgpu;

// a barrier that a thread which returns early leaves, as the device's does
struct HostBlock {
  int me, all;
  std::barrier<>* bar;
  int thread() const { return me; }
  int threads() const { return all; }
  void sync() const {
    if (bar) bar->arrive_and_wait();
  }
  template <class T>
  T load(const T* p) const { return *static_cast<const volatile T*>(p); }
};

struct State {
  IntervalCtl ctl;
  DistCtl dist;
  ChainCtl chain;
  DevScalars sc, out[kChain + 1];
  int done, stopped;
};

int main(int argc, char** argv) {
  if (argc != 8) return 2;
  const int threads = std::atoi(argv[1]), late = std::atoi(argv[2]);
  static State a;
  std::memset(&a, 0, sizeof(a));
  a.ctl.go = std::atoi(argv[3]);
  a.ctl.interval = 41;
  a.chain.pos = std::atoi(argv[4]);
  a.chain.n = std::atoi(argv[5]);
  a.chain.e_lo = 1.0f;
  a.chain.e_hi = 8.0f;
  a.chain.sec_stop = 1 << 20;
  for (int k = 0; k < kChain; ++k) a.chain.phi0[k] = 0.25f * k;
  const float e = (float)std::atof(argv[6]);
  const bool sampled = std::atoi(argv[7]) != 0;
  auto* words = reinterpret_cast<unsigned int*>(&a.sc);
  for (size_t k = 0; k < sizeof(DevScalars) / 4; ++k) words[k] = 0x3f000000u + (unsigned)k;  // (no word is zero)
  a.sc.error_flag = 0;
  a.sc.sec_count = 7;
  std::memcpy(&a.sc.sample_max_bits, &e, 4);
  for (int k = 0; k < kMoments; ++k) a.sc.moments[k] = 3.0 + k;
  for (auto& row : a.out) std::memset(&row, 0x5a, sizeof(row));
  a.done = a.stopped = -1;
  static State want;
  std::memcpy(&want, &a, sizeof(a));
  auto run = [&](State& s, const HostBlock& b) {
    end_interval(b, s.ctl, s.dist, s.chain, &s.sc, 10, s.out, 1, &s.done, &s.stopped, sampled);
  };
  run(want, HostBlock{0, 1, nullptr});
  {
    std::barrier<> bar(threads);
    std::vector<std::thread> block;
    for (int t = 0; t < threads; ++t)
      block.emplace_back([&, t] {
        if (t / 32 == late && t != 0) std::this_thread::sleep_for(std::chrono::milliseconds(50));
        run(a, HostBlock{t, threads, &bar});
        bar.arrive_and_drop();
      });
    for (auto& t : block) t.join();
  }
  int bad = 0;
  auto same = [&](const char* name, const void* x, const void* y, size_t n) {
    if (std::memcmp(x, y, n) == 0) return;
    std::printf("%s differs\n", name);
    bad = 1;
  };
  same("control", &a.ctl, &want.ctl, sizeof(a.ctl));
  same("distributions", &a.dist, &want.dist, sizeof(a.dist));
  same("chain", &a.chain, &want.chain, sizeof(a.chain));
  same("scalars", &a.sc, &want.sc, sizeof(a.sc));
  for (int k = 0; k <= kChain; ++k) same("row", &a.out[k], &want.out[k], sizeof(DevScalars));
  same("done", &a.done, &want.done, sizeof(int));
  same("stopped", &a.stopped, &want.stopped, sizeof(int));
  if (!bad) std::printf("ok %d %d %d\n", a.done, a.ctl.go, a.chain.pos);
  return bad;
}
