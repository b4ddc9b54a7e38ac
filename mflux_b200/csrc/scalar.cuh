// One value of a float32, bf16 or float16 array as float32 (dtype codes of include/mfx.h).
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

#include "../../include/mfx.h"

namespace mfx {

// The array may be what the kernel before has just written (launch.cuh), so nothing here goes through the read-only path.
// ACROSS: the kernel does not write the array itself, and the load may pass the kernel's own stores. It is volatile assembly
// without a claim on memory: behind the wait for the predecessor and behind bounds tests, but free of the stores, which a
// plain load is not. With plain loads an epilogue has its biases and gates one after the other, each stored to shared memory
// before the next is asked for: a step of the dual-stream model for one 1024 x 1024 image 69.7 ms where this takes 68.0.
// (16-bit values as integers: the __ldg overloads of cuda_fp16.h and cuda_bf16.h are asm statements that are not volatile,
// pure functions to the compiler, which evaluated them ahead of the bounds test they stood behind; a norm of 256 columns
// issued 23120 load requests instead of 2720, up to 12 KB past the end of its vectors, and faulted there.)
template <bool ACROSS = true>
__device__ __forceinline__ float load_as_float(const void* p, int dtype, int64_t i) {
  if (dtype == MFX_F32) {
    if (!ACROSS) return static_cast<const float*>(p)[i];
    float f;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(f) : "l"(static_cast<const float*>(p) + i));
    return f;
  }
  unsigned short v;
  if (ACROSS) asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(static_cast<const unsigned short*>(p) + i));
  else v = static_cast<const unsigned short*>(p)[i];
  return dtype == MFX_BF16 ? __uint_as_float(static_cast<uint32_t>(v) << 16) : __half2float(__ushort_as_half(v));
}

}  // namespace mfx
