"""The host code builds for other processors than x86: its intrinsics stand in places that say so."""
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hetuctr_b200", "csrc")
AT_HOME = {"utils/cpu_relax.h", "utils/stage_keys.cc"}  # behind #if defined(__x86_64__)


def test_x86_intrinsics_are_guarded(tmp_path):
    used = set()
    for d, _, files in os.walk(CSRC):
        for f in files:
            text = open(os.path.join(d, f)).read()
            if re.search(r"__builtin_ia32|_mm\d*_|immintrin|xmmintrin|__cpuid|__rdtsc", text):
                used.add(os.path.relpath(os.path.join(d, f), CSRC))
    assert used == AT_HOME
    # those two without the macros of an x86 compiler (and with its names made unusable)
    for f in sorted(AT_HOME):
        src = tmp_path / "t.cc"
        src.write_text('#include <cstddef>\n#include <cstdint>\n#undef __x86_64__\n#undef __i386__\n#define __builtin_ia32_pause not_here\n'
                       '#define __builtin_cpu_supports not_here\n#include "%s"\n' % f)
        subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-fsyntax-only", "-I", CSRC, str(src)], check=True)
