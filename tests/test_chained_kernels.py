"""Kernels that are launched while their predecessor in the stream still runs (launch_chained): what their sources have to keep to,
and what the launcher leaves behind when a launch fails."""
import glob
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KERNELS = os.path.join(ROOT, "hetuctr_b200", "csrc", "kernels")
CONSTANT = {"row_of"}  # written by a table's constructor alone


def _sources():
    return {os.path.basename(p): open(p).read() for p in glob.glob(os.path.join(KERNELS, "*.cu"))}


def _chained(text):
    names = set(re.findall(r"launch_chained\((\w+)", text))
    if "kernel" in names:  # picked from several instances
        names.remove("kernel")
        names |= set(re.findall(r"const auto kernel = vec \? (\w+)<", text))
    return names


def test_pointers_that_a_predecessor_writes_are_not_restrict():
    found, seen = [], 0
    for name, text in _sources().items():
        for kernel in _chained(text):
            m = re.search(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\) )?%s\(([^{]*)\) \{(.*?)\n}\n" % kernel, text, re.S)
            assert m, (name, kernel)
            seen += 1
            found += [(name, kernel, p) for p in re.findall(r"__restrict__\s+(\w+)", m[1]) if p not in CONSTANT]
            assert "wait_predecessor();" in m[2], (name, kernel)
    assert seen == 8, seen
    assert not found, found
