// Large-M quantized matmul in two launches: decode the weight to bf16 scratch, then a plain bf16 contraction.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/mfx.h"

namespace mfx {
namespace qmmd {

// The decoded weight, and what of it to ask a caller for: 0 where the one-launch kernel, at a cost of one_launch_cost
// percent of one of its widest waves, is the faster one. m_tiles = 256-row tiles of all samples.
inline size_t dense_bytes(int64_t N, int64_t K) { return static_cast<size_t>(N) * static_cast<size_t>(K) * 2; }
size_t scratch_bytes(int64_t m_tiles, int64_t N, int64_t K, int bits, int64_t one_launch_cost);
// `a` was validated by qmm::run; prepared = blob of mfx_qlinear_prepare, codes_bytes = size of its code section,
// scratch = dense_bytes() bytes of device memory, 256-byte aligned. Every epilogue but the tensor-parallel scatter.
int run(const mfx_qlinear_args& a, const void* prepared, size_t codes_bytes, void* scratch, cudaStream_t st);
int read_status(int* out, cudaStream_t stream);

}  // namespace qmmd
}  // namespace mfx
