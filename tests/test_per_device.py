"""Kernel attributes and occupancies belong to a device, so what the launchers remember about them is kept per device:
the helper itself, compiled on its own, and a look that no launcher keeps such a thing in a plain static."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hetuctr_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "utils/per_device.h"
static hetuCTR::PerDevice attr, blocks;
int main() {
  std::atomic<int> calls{0};
  auto ok = [&] { calls++; return 0; };
  auto bad = [&] { calls++; return 7; };
  if (attr.once(0, bad) != 7 || attr.once(0, ok) != 0 || calls != 2) return 1;   // a failure is not remembered
  if (attr.once(0, ok) != 0 || attr.once(0, bad) != 0 || calls != 2) return 2;   // a success is
  if (attr.once(1, ok) != 0 || calls != 3) return 3;                             // for that device only
  if (attr.once(63, ok) != 0 || attr.once(64, ok) != 0 || attr.once(64, ok) != 0 || attr.once(-1, bad) != 7 || calls != 7)
    return 4;                                                                    // outside the array: every time
  if (blocks.get(0, [] { return 16; }) != 16 || blocks.get(1, [] { return 8; }) != 8 || blocks.get(0, [] { return 3; }) != 16)
    return 5;
  calls = 0;
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; t++)
    ts.emplace_back([&] {
      for (int i = 0; i < 2000; i++)
        if (attr.once(2 + i % 50, ok) != 0) calls += 1000000;
    });
  for (auto &t : ts) t.join();
  return calls >= 50 && calls <= 400 ? 0 : 6;
}
"""


def test_remembered_per_device(tmp_path):
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_launchers_keep_no_plain_static():
    found = []
    for path in glob.glob(os.path.join(CSRC, "kernels", "*.cu")):
        for n, line in enumerate(open(path), 1):
            if re.match(r"\s+static (bool|int|u32|unsigned|size_t)\b[^(]*[;=]", line) and "constexpr" not in line:
                found.append(f"{os.path.basename(path)}:{n}: {line.strip()}")
    assert not found, found


SHARED = r"""
#include "utils/same_device.h"
using namespace hetuCTR;
static DeviceIdentity id(char last) {
  DeviceIdentity d = {};
  d.uuid[15] = last;
  return d;
}
int main() {
  const std::vector<DeviceIdentity> two_threads = {id(1), id(1)}, a_gpu_each = {id(0), id(1), id(2)}, mixed = {id(4), id(5), id(4)};
  if (!shares_device(two_threads, 0) || !shares_device(two_threads, 1)) return 1;
  for (int r = 0; r < 3; r++)
    if (shares_device(a_gpu_each, r)) return 2;
  return shares_device(mixed, 0) && !shares_device(mixed, 1) && shares_device(mixed, 2) ? 0 : 3;
}
"""


def test_ranks_share_a_device_by_its_identity(tmp_path):
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(SHARED)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
    table = open(os.path.join(CSRC, "core", "hetu_table.cc")).read()
    assert "shares_device(" in table and "transport_->name()," not in table  # (not guessed from how they are connected)
