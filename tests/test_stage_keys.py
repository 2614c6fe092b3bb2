"""The checked copy of a host key batch, compiled on its own: what it copies, and that it refuses a key outside the table
wherever it stands - in the vector body, in the tail behind it, first or last; and when a way of ingesting keys that has failed
is tried again."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hetuctr_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "utils/stage_keys.h"
using namespace hetuCTR;

template <class T>
static int check(size_t length, size_t n, size_t shift) {
  std::mt19937_64 rng(n + length);
  std::vector<char> raw(8 * n + 16);
  int64_t *src = reinterpret_cast<int64_t *>(raw.data() + shift);  // (any address)
  std::vector<int64_t> want(n);
  for (auto &k : want) k = (int64_t)(rng() % length);
  if (n) want[n / 2] = (int64_t)length - 1;
  if (n > 1) want[1] = 0;
  std::memcpy(raw.data() + shift, want.data(), 8 * n);
  std::vector<T> dst(n + 1, (T)77);
  if (!stage_keys(src, dst.data(), n, length)) return 1;
  for (size_t i = 0; i < n; i++)
    if ((int64_t)dst[i] != want[i]) return 2;
  if (dst[n] != (T)77) return 3;
  for (size_t at : {(size_t)0, (size_t)3, (size_t)4, (size_t)7, (size_t)8, n / 8 * 8, n - 2, n - 1})
    for (int64_t bad : {(int64_t)-1, (int64_t)length, (int64_t)length + 1, (int64_t)1 << 40, INT64_MIN, INT64_MAX,
                        (int64_t)((uint64_t)1 << 32)}) {
      if (at >= n || (bad >= 0 && (size_t)bad < length)) continue;
      std::memcpy(raw.data() + shift + 8 * at, &bad, 8);
      if (stage_keys(src, dst.data(), n, length)) return 4;
      std::memcpy(raw.data() + shift + 8 * at, &want[at], 8);
    }
  return stage_keys(src, dst.data(), n, length) ? 0 : 5;
}

int main() {
  for (size_t n : {0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 100, 1003, 65536, 65537})
    for (size_t shift : {0, 3})
      for (size_t length : {(size_t)1, (size_t)1000, (size_t)1 << 31, (size_t)3 << 32}) {
        if (int e = check<int64_t>(length, n, shift)) return std::printf("64 bits, n %zu, length %zu: %d\n", n, length, e), 1;
        if (length > (size_t)1 << 31) continue;
        if (int e = check<int32_t>(length, n, shift)) return std::printf("32 bits, n %zu, length %zu: %d\n", n, length, e), 1;
      }
  int32_t none = 0;
  const int64_t zero = 0;
  return stage_keys(&zero, &none, 1, 0) || !stage_keys(&zero, &none, 0, 0);
}
"""


def test_keys_are_copied_and_checked(tmp_path):
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    for vector in (True, False):  # with the vector body where the processor has one, and without
        src.write_text('#include <cstring>\n%s\n#include "utils/stage_keys.cc"\n%s'
                       % ("" if vector else "#undef __x86_64__", PROGRAM))
        subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)], check=True)
        r = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
        assert r.returncode == 0, r.stdout


BACKOFF = r"""
#include "utils/backoff.h"
int main() {
  hetuCTR::Backoff b;
  for (int i = 0; i < 5; i++) {
    if (!b.tryNow()) return 1;
    b.worked();
  }
  unsigned pause = 1;
  for (int i = 0; i < 14; i++) {  // never off for good
    if (!b.tryNow()) return 2;
    b.failed();
    for (unsigned k = 0; k < pause; k++)
      if (b.tryNow()) return 3;
    pause = pause < 1024 ? 2 * pause : 1024;
  }
  if (!b.tryNow()) return 4;
  b.worked();
  if (!b.tryNow()) return 5;
  b.failed();
  return !b.tryNow() && b.tryNow() ? 0 : 6;
}
"""


def test_a_failed_way_is_tried_again(tmp_path):
    src, exe = tmp_path / "t.cc", tmp_path / "t"
    src.write_text(BACKOFF)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
