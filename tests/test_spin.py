"""Threads that wait awake keep nobody from the processor: they sleep at once where the threads of a job have no processor
each, and stop waiting awake when they compete for one."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hetuctr_b200", "csrc")

PROGRAM = r"""
#include <pthread.h>
#include <sched.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include "utils/spin.h"
#include "utils/thread_pool.h"
using clk = std::chrono::steady_clock;
static void on(int a, int b) {
  cpu_set_t s;
  CPU_ZERO(&s);
  CPU_SET(a, &s);
  CPU_SET(b, &s);
  pthread_setaffinity_np(pthread_self(), sizeof(s), &s);
}
static double ms(clk::time_point from) { return std::chrono::duration<double, std::milli>(clk::now() - from).count(); }
// Computes until `until`, on core `core` only.
static void compute(int core, clk::time_point until) {
  on(core, core);
  while (clk::now() < until)
    for (volatile int i = 0; i < 1000; i = i + 1) {}
}
int main(int argc, char **argv) {
  const int a = std::atoi(argv[1]), b = std::atoi(argv[2]);
  {  // queued calls still run in order and hand over their failures
    hetuCTR::ThreadPool pool(1);
    std::vector<int> seen;
    for (int i = 0; i < 100; i++) {
      auto f = pool.Enqueue([&, i] { seen.push_back(i); });
      hetuCTR::wait_awake(f);
    }
    auto f = pool.Enqueue([] { throw 5; });
    try {
      hetuCTR::wait_awake(f);
      return 1;
    } catch (int v) {
      if (v != 5 || seen.size() != 100 || seen[99] != 99) return 2;
    }
  }
  if (hetuCTR::queue_workers() != 0) return 3;
  {
    hetuCTR::ThreadPool one(1), three(3);
    if (hetuCTR::queue_workers() != 4) return 3;
  }
  if (!hetuCTR::spin_for(0, 1000, [] { return true; })) return 4;
  on(a, b);
  auto past_a_look = [] {
    for (int i = 0; i < 16; i++) hetuCTR::spin_for(0, 1, [] { return false; });
  };
  past_a_look();
  auto t0 = clk::now();
  for (int i = 0; i < 20; i++)
    if (hetuCTR::spin_for(20000, 3, [] { return false; })) return 4;
  if (ms(t0) > 200) return 5;  // (400 ms awake)
  std::atomic<bool> go{false};
  std::thread later([&] {
    std::this_thread::sleep_for(std::chrono::milliseconds(20));
    go = true;
  });
  while (!hetuCTR::spin_for(1000, 2, [&] { return go.load(); })) {}
  later.join();
  // two threads compute on one core, so each of them loses it to the other; this one then sleeps 64 times
  const auto until = clk::now() + std::chrono::milliseconds(200);
  std::thread other(compute, a, until);
  compute(a, until);
  other.join();
  on(a, b);
  past_a_look();
  int slept = 0;
  for (int i = 0; i < 300; i++) {
    t0 = clk::now();
    if (hetuCTR::spin_for(2000, 2, [] { return false; })) return 6;
    if (ms(t0) < 1) slept++;
  }
  std::printf("%d waits asleep\n", slept);
  return slept >= 48 && slept < 300 ? 0 : 7;  // (some of the 64 may fall before the count)
}
"""


def test_when_a_thread_waits_awake(tmp_path):
    cores = sorted(os.sched_getaffinity(0))
    if len(cores) < 2:
        pytest.skip("needs two processors")
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe), str(cores[0]), str(cores[1])], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
