"""csrc/launch.cuh compiled for the host against a runtime whose launches fail: the error is returned and none stays pending,
which the next ordinary launch's check would take for its own."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mflux_b200" / "csrc"

RUNTIME = """
#pragma once
#include <cstddef>
#define __device__
#define __forceinline__ inline
typedef int cudaError_t;
typedef void* cudaStream_t;
constexpr int cudaSuccess = 0;
struct dim3 { unsigned x = 1, y = 1, z = 1; dim3(unsigned a = 1) : x(a) {} };
enum cudaLaunchAttributeID { cudaLaunchAttributeProgrammaticStreamSerialization };
struct cudaLaunchAttribute {
  cudaLaunchAttributeID id;
  struct { int programmaticStreamSerializationAllowed; } val;
};
struct cudaLaunchConfig_t {
  dim3 gridDim, blockDim;
  size_t dynamicSmemBytes;
  cudaStream_t stream;
  cudaLaunchAttribute* attrs;
  unsigned numAttrs;
};
static int result = 0, pending = 0;
inline cudaError_t cudaGetLastError() { int e = pending; pending = 0; return e; }
template <typename... P, typename... A>
cudaError_t cudaLaunchKernelEx(const cudaLaunchConfig_t*, void (*)(P...), A...) {
  if (result) pending = result;
  return result;
}
"""

MAIN = """
#include "launch.cuh"
void kernel(int) {}
int main() {
  result = 9;
  if (mfx::launch_overlapped(kernel, 1, 32, 0, nullptr, 1) != 9) return 1;
  if (cudaGetLastError() != 0) return 2;
  result = 0;
  pending = 7;   // not of this launch: left to whoever asks
  if (mfx::launch_overlapped(kernel, 1, 32, 0, nullptr, 1) != 0) return 3;
  return cudaGetLastError() == 7 ? 0 : 4;
}
"""


def test_a_failed_launch_leaves_nothing_pending(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(MAIN)
    out = tmp_path / "main"
    subprocess.run([cxx, "-std=c++17", "-I", str(tmp_path), "-I", str(CSRC), str(tmp_path / "main.cpp"), "-o", str(out)],
                   check=True)
    assert subprocess.run([str(out)]).returncode == 0
