"""Kernels that are launched while their predecessor in the stream still runs (launch_chained): what their sources have to keep to,
and what the launcher leaves behind when a launch fails."""
import glob
import os
import re
import subprocess

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
            m = re.search(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?%s\(([^{]*)\) \{(.*?)\n}\n" % kernel, text, re.S)
            assert m, (name, kernel)
            seen += 1
            found += [(name, kernel, p) for p in re.findall(r"__restrict__\s+(\w+)", m[1]) if p not in CONSTANT]
            assert "wait_predecessor();" in m[2], (name, kernel)
    assert seen == 8, seen
    assert not found, found


def test_grid_of_the_fused_expansion_is_what_its_launch_bounds_keep_resident():
    text = _sources()["p2p_pull.cu"]
    assert "__launch_bounds__(kFusedThreads, fused_blocks(LANES))" in text
    launcher = text[text.index("int hctr_p2p_refresh_expand"):]
    assert re.findall(r"cap_ = \(size_t\)kSMs \* ([^;]+);", launcher) == ["fused_blocks(L)"]


PROGRAM = r"""
#include <cuda_runtime.h>
static cudaError_t last = cudaSuccess;
static cudaError_t fake_launch_error() { return last = cudaErrorInvalidConfiguration; }
static cudaError_t fake_last_error() { const cudaError_t e = last; last = cudaSuccess; return e; }
#define cudaLaunchKernelEx(...) fake_launch_error()
#define cudaGetLastError fake_last_error
#include "kernels/common.cuh"
namespace hctr { unsigned long long g_launches = 0; }
__global__ void nothing(int) {}
int main() {
  if (hctr::launch_chained(nothing, 1, 32, 0, (cudaStream_t)0, 1) != (int)cudaErrorInvalidConfiguration) return 1;
  if (hctr::launch_status() != 0) return 2;  // the next launch has nothing to do with it
  if (hctr::launch_status(fake_launch_error()) != (int)cudaErrorInvalidConfiguration || hctr::launch_status() != 0) return 3;
  fake_launch_error();
  return hctr::launch_status(cudaSuccess) == (int)cudaErrorInvalidConfiguration ? 0 : 4;
}
"""


def test_a_failed_launch_is_reported_once(tmp_path):
    src, exe = tmp_path / "t.cu", tmp_path / "t"
    src.write_text(PROGRAM)
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "hetuctr_b200", "csrc"), "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
