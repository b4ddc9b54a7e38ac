// One value of a float32, bf16 or float16 array as float32 (dtype codes of include/mfx.h).
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/mfx.h"

namespace mfx {

// Plain loads: the array may be what the kernel before has just written (launch.cuh). 16-bit values as integers: the __ldg
// overloads of cuda_fp16.h and cuda_bf16.h are asm statements that are not volatile, pure functions to the compiler, which
// evaluated them ahead of the bounds test they stood behind (a norm of 256 columns issued 23120 load requests instead of
// 2720, up to 12 KB past the end of its vectors, and faulted there).
__device__ __forceinline__ float load_as_float(const void* p, int dtype, int64_t i) {
  if (dtype == MFX_F32) return static_cast<const float*>(p)[i];
  const unsigned short v = static_cast<const unsigned short*>(p)[i];
  return dtype == MFX_BF16 ? __uint_as_float(static_cast<uint32_t>(v) << 16) : __half2float(__ushort_as_half(v));
}

}  // namespace mfx
