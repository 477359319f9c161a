"""A launch that fails answers for itself only: its error must not stay with the thread, where the check after the next
plain launch (cudaGetLastError) would take it for that launch's own.  No GPU: in a small program two calls of the
runtime are replaced by fakes: a launch that fails, and a cudaGetLastError that takes the failure, as the real one does."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = """
int kept = 0;
extern "C" int __wrap_cudaLaunchKernelExC(const void*, const void*, void**) { return kept = 9; }
extern "C" int __wrap_cudaGetLastError() {
  const int e = kept;
  kept = 0;
  return e;
}
"""
PROGRAM = """
#include "va_common.cuh"
#include <cstdio>
extern int kept;
static void some_kernel(int) {}
int main() {
  va::launch_after(some_kernel, dim3(1), 32u, 0, nullptr, 1);
  std::printf("%d", kept);
}
"""


def test_a_failed_launch_leaves_no_error_behind(tmp_path):
    from vecattention_b200.build import CSRC, NVCC_FLAGS, _nvcc
    runtime, source, program = tmp_path / "runtime.cpp", tmp_path / "launch.cu", tmp_path / "launch"
    runtime.write_text(RUNTIME)
    source.write_text(PROGRAM)
    subprocess.run([_nvcc(), *NVCC_FLAGS, "-I", os.path.join(ROOT, "include"), "-I", CSRC, str(source), str(runtime), "-o", str(program),
                    "-Xlinker", "--wrap=cudaLaunchKernelExC", "-Xlinker", "--wrap=cudaGetLastError"], check=True)
    assert subprocess.run([str(program)], check=True, capture_output=True, text=True).stdout == "0"
