// Epilogue of the tensor-core matmul kernels (qmm.cu, qmm_dense.cu): one accumulator row per thread, tensor memory
// -> bias / activation / gated residual -> global memory.
#pragma once
#include "qmm_common.cuh"

namespace mfx {
namespace qmm {

// One whole 32-byte sector per thread. Threads of a warp write different rows here, so a 16-byte access leaves half of
// every sector to a second instruction: twice the requests to L2, and partial-sector writes. M 73728, N 3072, K 3072, 4
// bits, gated residual on the float32 stream: 1684 us with 16-byte accesses, 1391 us with these.
__device__ __forceinline__ void st_global_32(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]),
               "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
// Volatile, so that it stays behind the tests for rows and columns past the end: to the compiler an asm statement that is
// not is a pure function of its operands, which it may evaluate ahead of a branch, and the address would then be out of
// the residual. The loads of a chunk stand ahead of its stores in the source.
__device__ __forceinline__ void ld_global_32(const void* p, uint32_t (&v)[8]) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "l"(p));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// bias and activation of eight neighbouring columns (not the residual, not SwiGLU's product)
template <int EPI, bool CALLS>
__device__ __forceinline__ void activate8(const uint32_t* acc, const float* bias_s, float (&v)[8]) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = __uint_as_float(acc[j]) + bias_s[j];
    if (EPI == MFX_EPI_GELU_ERF) v[j] = CALLS ? gelu_erf_call(v[j]) : gelu_erf(v[j]);
    else if (EPI == MFX_EPI_GELU_TANH) v[j] = CALLS ? gelu_tanh_call(v[j]) : gelu_tanh(v[j]);
    else if (EPI == MFX_EPI_SILU) v[j] = silu(v[j]);
  }
}

// v = residual + gate * v on eight neighbouring columns, 16-byte loads
template <typename OUT>
__device__ __forceinline__ void add_residual8(const OUT* rrow, const float* gate_s, float (&v)[8]) {
  float rs[8];
  if constexpr (sizeof(OUT) == 4) {
    const float4 r0 = *reinterpret_cast<const float4*>(rrow), r1 = *reinterpret_cast<const float4*>(rrow + 4);
    rs[0] = r0.x; rs[1] = r0.y; rs[2] = r0.z; rs[3] = r0.w;
    rs[4] = r1.x; rs[5] = r1.y; rs[6] = r1.z; rs[7] = r1.w;
  } else {
    const uint4 raw = *reinterpret_cast<const uint4*>(rrow);
    const uint32_t r4[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      rs[2 * j] = __uint_as_float(r4[j] << 16);
      rs[2 * j + 1] = __uint_as_float(r4[j] & 0xFFFF0000u);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = rs[j] + gate_s[j] * v[j];
}

// Asks for columns [c0, c1) of a residual row: called before the wait for the accumulator, so that the row's trip from
// HBM overlaps the main loop. With short K the epilogue is what a tile waits for (M 14290, N 3072, K 3072: 285 -> 278 us
// in one launch, 262 -> 253 us in two); with K of 12288 it hides behind the main loop anyway, and lines asked for
// that early cost 1-2 %.
constexpr int PREFETCH_K = 4096;
template <typename OUT>
__device__ __forceinline__ void prefetch_row(const OUT* rrow, int c0, int c1, int n_left) {
  for (int c = c0; c < min(c1, n_left); c += 128 / static_cast<int>(sizeof(OUT)))
    asm volatile("prefetch.global.L2 [%0];" ::"l"(rrow + c));
}

// 32-byte accesses need the row's addresses on that boundary; the entry point only promises 16.
template <typename OUT, int EPI>
inline bool wide_rows(const void* y, int64_t y_row_stride, int64_t y_batch_stride, const void* residual,
                      int64_t res_row_stride, int64_t res_batch_stride) {
  auto odd = [](const void* p, int64_t rs, int64_t bs) {
    return (reinterpret_cast<uintptr_t>(p) | static_cast<uintptr_t>(rs * sizeof(OUT)) |
            static_cast<uintptr_t>(bs * sizeof(OUT))) & 31u;
  };
  return !odd(y, y_row_stride, y_batch_stride) &&
         (EPI != MFX_EPI_GATE_RESIDUAL || !odd(residual, res_row_stride, res_batch_stride));
}

// Writes columns [c0, c1) (multiples of 32) of one output row of a tile. t_addr = the warp's lanes of the accumulator,
// n_left = output columns of the layer from the tile's first one on, yrow / rrow = the row's first column of this
// tile, wide = wide_rows(), CALLS = out-of-line activations. Rows past the end (row_ok false) take part in the
// tensor-memory loads only, which are collective: lanes take different paths below, so the warp meets before each.
template <typename OUT, int EPI, bool CALLS>
__device__ __forceinline__ void write_row(uint32_t t_addr, int c0, int c1, int n_left, bool row_ok, bool wide, OUT* yrow,
                                          const OUT* rrow, const float* bias_s, const float* gate_s) {
#pragma unroll 1
  for (int c = c0; c < c1; c += 32) {
    uint32_t acc[32];
    __syncwarp();
    tmem_ld_32x32(t_addr + c, acc);
    tmem_ld_wait();
    if (!row_ok) continue;
    if (wide && c + 32 <= n_left) {
      uint32_t o[8];
      uint32_t rs[4][8];   // the chunk's residual: four loads in flight instead of one at a time
      if constexpr (EPI == MFX_EPI_GATE_RESIDUAL && sizeof(OUT) == 4) {
#pragma unroll
        for (int g8 = 0; g8 < 4; ++g8) ld_global_32(rrow + c + g8 * 8, rs[g8]);
      }
#pragma unroll
      for (int g8 = 0; g8 < 4; ++g8) {
        const int col = c + g8 * 8;
        float v[8];
        activate8<EPI, CALLS>(acc + g8 * 8, bias_s + col, v);
        if constexpr (EPI == MFX_EPI_SWIGLU) {
          float s[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) s[j] = silu(v[2 * j]) * v[2 * j + 1];
          if constexpr (sizeof(OUT) == 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j) o[(g8 & 1) * 4 + j] = __float_as_uint(s[j]);
            if (g8 & 1) st_global_32(yrow + col / 2 - 4, o);
          } else {
            o[2 * g8] = pack_bf16(s[0], s[1]);
            o[2 * g8 + 1] = pack_bf16(s[2], s[3]);
            if (g8 == 3) st_global_32(yrow + c / 2, o);
          }
        } else if constexpr (sizeof(OUT) == 4) {
          if constexpr (EPI == MFX_EPI_GATE_RESIDUAL) {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(rs[g8][j]) + gate_s[col + j] * v[j];
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = __float_as_uint(v[j]);
          st_global_32(yrow + col, o);
        } else {
          if constexpr (EPI == MFX_EPI_GATE_RESIDUAL) add_residual8<OUT>(rrow + col, gate_s + col, v);
#pragma unroll
          for (int j = 0; j < 4; ++j) o[(g8 & 1) * 4 + j] = pack_bf16(v[2 * j], v[2 * j + 1]);
          if (g8 & 1) st_global_32(yrow + col - 8, o);
        }
      }
      continue;
    }
#pragma unroll
    for (int g8 = 0; g8 < 4; ++g8) {
      const int col = c + g8 * 8;
      if (col >= n_left) break;
      float v[8];
      activate8<EPI, CALLS>(acc + g8 * 8, bias_s + col, v);
      if constexpr (EPI == MFX_EPI_SWIGLU) {
        float s[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = silu(v[2 * j]) * v[2 * j + 1];
        if constexpr (sizeof(OUT) == 4)
          *reinterpret_cast<float4*>(yrow + col / 2) = make_float4(s[0], s[1], s[2], s[3]);
        else
          *reinterpret_cast<uint2*>(yrow + col / 2) = make_uint2(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]));
      } else {
        if constexpr (EPI == MFX_EPI_GATE_RESIDUAL) add_residual8<OUT>(rrow + col, gate_s + col, v);
        if constexpr (sizeof(OUT) == 4) {
          *reinterpret_cast<float4*>(yrow + col) = make_float4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<float4*>(yrow + col + 4) = make_float4(v[4], v[5], v[6], v[7]);
        } else {
          *reinterpret_cast<uint4*>(yrow + col) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]),
                                                             pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
        }
      }
    }
  }
}

}  // namespace qmm
}  // namespace mfx
