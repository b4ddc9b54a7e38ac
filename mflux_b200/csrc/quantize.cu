// Group-wise affine weight quantizer and dequantizer (HBM-bound, load-time kernels).
//
// Semantics follow mx.quantize(w, group_size=64, bits) as reached from the reference through
// mlx.nn.quantize (src/mflux/models/common/weights/loading/weight_applier.py:93-103): groups of 64
// along the input dimension, float32 arithmetic, codes packed little-end first: code j of a row occupies
// bits [j*bits, (j+1)*bits) of the row's bit stream, which for 4 and 8 bits is "8 / 4 codes per uint32" and for
// 3, 5 and 6 bits (the other widths the reference's CLI offers, src/mflux/cli/defaults/defaults.py:63) lets
// codes straddle byte and word boundaries (8 codes in 3 or 5 bytes, 4 codes in 3 bytes).
// Four lanes own one group (16 values each); min/max go through warp shuffles.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "host_util.cuh"

namespace mfx {
namespace {

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

template <typename T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half from_f32<__half>(float v) { return __float2half_rn(v); }

constexpr int PER_THREAD = 16;   // values of one group a thread holds

template <typename T>
__device__ __forceinline__ void load16(const T* p, float (&v)[16]) {
  if constexpr (sizeof(T) == 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(p) + i);
      v[4 * i] = a.x; v[4 * i + 1] = a.y; v[4 * i + 2] = a.z; v[4 * i + 3] = a.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint4 raw = __ldg(reinterpret_cast<const uint4*>(p) + k);
      const T* h = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[8 * k + i] = to_f32<T>(h[i]);
    }
  }
}

// The quantizer's definition of a code: the correctly rounded quotient, rounded to even, clamped.
__device__ __forceinline__ float exact_code(float d, float scale, float n_bins) {
  float q = rintf(__fdiv_rn(d, scale));
  if (!(fabsf(q) <= 3.0e38f)) q = 0.0f;  // constant group with scale == 0: code 0
  return fminf(fmaxf(q, 0.0f), n_bins);
}

// One thread: 16 consecutive values of a row; lanes 4g..4g+3 of a warp form one 64-wide group.
// A division per value was what the kernel spent its time on. It multiplies by the reciprocal of the scale instead and
// takes the rounded product where that must be the rounded quotient too: reciprocal, product and the quotient itself
// are each off by at most 2^-24 of their value, together 1.8e-7 of at most n_bins + 1, so a product further than that
// from every k + 0.5 rounds like the quotient. Threads with a value nearer to one (one in 1000 at 4 bits) divide.
template <typename T, int BITS, int QMODE>
__global__ void __launch_bounds__(256) quantize_kernel(const T* __restrict__ w, int64_t n_groups_total,
                                                       uint32_t* __restrict__ wq, T* __restrict__ scales,
                                                       T* __restrict__ biases) {
  const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int64_t group = tid >> 2;
  const bool active = group < n_groups_total;
  const int64_t g = active ? group : n_groups_total - 1;  // keep whole warps in the shuffles
  const int sub = static_cast<int>(tid & 3);
  float v[16];
  load16<T>(w + g * 64 + sub * 16, v);
  float mx = v[0], mn = v[0];
#pragma unroll
  for (int i = 1; i < 16; ++i) {
    mx = fmaxf(mx, v[i]);
    mn = fminf(mn, v[i]);
  }
#pragma unroll
  for (int off = 2; off >= 1; off >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
  }
  constexpr float n_bins = static_cast<float>((1 << BITS) - 1);
  float scale, bias;
  if (QMODE == MFX_QMODE_MLX) {
    scale = fmaxf(__fdiv_rn(__fsub_rn(mx, mn), n_bins), 1e-7f);
    const bool side = fabsf(mn) > fabsf(mx);
    scale = side ? scale : -scale;
    const float edge = side ? mn : mx;
    const float q0 = rintf(__fdiv_rn(edge, scale));
    if (q0 == 0.0f) {
      bias = 0.0f;
    } else {
      scale = __fdiv_rn(edge, q0);
      bias = edge;
    }
  } else {
    scale = __fdiv_rn(__fsub_rn(mx, mn), n_bins);
    bias = mn;
  }
  const float mag = fabsf(scale);
  bool divide = !(mag > 1e-30f && mag < 1e30f);   // the reciprocal has to be a normal number
  const float inv = __frcp_rn(scale);
  constexpr float MAGIC = 12582912.0f;            // 1.5 * 2^23: adding it rounds to even at the units place
  float q[16];
  float far = 0.0f;                               // largest distance of a product from its integer
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const float r = fminf(fmaxf(__fmul_rn(__fsub_rn(v[i], bias), inv), 0.0f), n_bins);
    q[i] = __fsub_rn(__fadd_rn(r, MAGIC), MAGIC);
    far = fmaxf(far, fabsf(__fsub_rn(r, q[i])));
  }
  divide |= far > 0.5f - (n_bins + 1.0f) * 2.4e-7f;
  if (divide) {
#pragma unroll
    for (int i = 0; i < 16; ++i) q[i] = exact_code(__fsub_rn(v[i], bias), scale, n_bins);
  }
  if (!active) return;
  if constexpr (BITS == 4) {
    // four codes at a time as an exact float below 2^16
    uint32_t half[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      half[i] = static_cast<uint32_t>(fmaf(fmaf(fmaf(q[4 * i + 3], 16.0f, q[4 * i + 2]), 16.0f, q[4 * i + 1]), 16.0f,
                                           q[4 * i]));
    reinterpret_cast<uint2*>(wq)[g * 4 + sub] = make_uint2(half[0] | (half[1] << 16), half[2] | (half[3] << 16));
  } else if constexpr (BITS == 8) {
    uint32_t word[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t lo = static_cast<uint32_t>(fmaf(q[4 * i + 1], 256.0f, q[4 * i]));
      const uint32_t hi = static_cast<uint32_t>(fmaf(q[4 * i + 3], 256.0f, q[4 * i + 2]));
      word[i] = lo | (hi << 16);
    }
    reinterpret_cast<uint4*>(wq)[g * 4 + sub] = make_uint4(word[0], word[1], word[2], word[3]);
  } else {
    // 8 codes = BITS bytes of the bit stream; 16 of them are BITS 16-bit words at an even address
    unsigned long long lo = 0, hi = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      lo |= static_cast<unsigned long long>(static_cast<uint32_t>(q[i])) << (BITS * i);
      hi |= static_cast<unsigned long long>(static_cast<uint32_t>(q[8 + i])) << (BITS * i);
    }
    const unsigned long long w0 = lo | (hi << (8 * BITS)), w1 = hi >> (64 - 8 * BITS);
    uint16_t* dst = reinterpret_cast<uint16_t*>(wq) + (g * 4 + sub) * BITS;
#pragma unroll
    for (int i = 0; i < BITS; ++i) dst[i] = static_cast<uint16_t>(i < 4 ? w0 >> (16 * i) : w1 >> (16 * (i & 3)));
  }
  if (sub == 0) {
    scales[g] = from_f32<T>(scale);
    biases[g] = from_f32<T>(bias);
  }
}

// One thread: V (8 or 16) consecutive outputs of a row.
template <typename SB, typename OUT, int BITS, int V>
__global__ void __launch_bounds__(256) dequantize_kernel(const uint32_t* __restrict__ wq,
                                                         const SB* __restrict__ scales,
                                                         const SB* __restrict__ biases, int64_t n_chunks,
                                                         OUT* __restrict__ out) {
  const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (tid >= n_chunks) return;
  const int64_t g = tid / (64 / V);
  const float s = to_f32<SB>(scales[g]);
  const float b = to_f32<SB>(biases[g]);
  uint32_t codes[V];
  if constexpr (BITS == 4 || BITS == 8) {
    constexpr int WORDS = V * BITS / 32;
    uint32_t words[WORDS];
    if constexpr (WORDS == 1) {
      words[0] = __ldg(wq + tid);
    } else if constexpr (WORDS == 2) {
      const uint2 v = __ldg(reinterpret_cast<const uint2*>(wq) + tid);
      words[0] = v.x; words[1] = v.y;
    } else {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(wq) + tid);
      words[0] = v.x; words[1] = v.y; words[2] = v.z; words[3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < V; ++i) codes[i] = (words[i * BITS / 32] >> (i * BITS % 32)) & ((1u << BITS) - 1u);
  } else {
    // eight codes are BITS bytes of the bit stream, sixteen are BITS 16-bit words at an even address
    unsigned long long eight[V / 8];
    if constexpr (V == 8) {
      const uint8_t* src = reinterpret_cast<const uint8_t*>(wq) + tid * BITS;
      eight[0] = 0;
#pragma unroll
      for (int i = 0; i < BITS; ++i) eight[0] |= static_cast<unsigned long long>(__ldg(src + i)) << (8 * i);
    } else {
      const uint16_t* src = reinterpret_cast<const uint16_t*>(wq) + tid * BITS;
      unsigned long long w0 = 0, w1 = 0;
#pragma unroll
      for (int i = 0; i < BITS; ++i) {
        const unsigned long long v = __ldg(src + i);
        if (i < 4) w0 |= v << (16 * i);
        else w1 |= v << (16 * (i & 3));
      }
      eight[0] = w0;
      eight[1] = (w0 >> (8 * BITS)) | (w1 << (64 - 8 * BITS));
    }
#pragma unroll
    for (int i = 0; i < V; ++i)
      codes[i] = static_cast<uint32_t>(eight[i / 8] >> (BITS * (i % 8))) & ((1u << BITS) - 1u);
  }
  __align__(16) OUT res[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    // sixteen conversions in a row wait for the converter: the code under the exponent of 2^23 instead
    const float c = V == 8 ? static_cast<float>(codes[i]) : __uint_as_float(0x4B000000u | codes[i]) - 8388608.0f;
    res[i] = from_f32<OUT>(__fadd_rn(__fmul_rn(c, s), b));
  }
  uint4* dst = reinterpret_cast<uint4*>(out + tid * V);
#pragma unroll
  for (int i = 0; i < V * static_cast<int>(sizeof(OUT)) / 16; ++i) dst[i] = reinterpret_cast<const uint4*>(res)[i];
}

template <typename T>
int launch_quantize(const void* w, int64_t n_groups, int bits, int qmode, uint32_t* wq, void* scales, void* biases,
                    cudaStream_t st) {
  const int64_t threads = n_groups * (64 / PER_THREAD);
  const unsigned blocks = static_cast<unsigned>((threads + 255) / 256);
  const T* wp = static_cast<const T*>(w);
  T* sp = static_cast<T*>(scales);
  T* bp = static_cast<T*>(biases);
#define MFX_QUANT_CASE(B)                                                                        \
  case B:                                                                                       \
    if (qmode == MFX_QMODE_MLX)                                                                 \
      quantize_kernel<T, B, MFX_QMODE_MLX><<<blocks, 256, 0, st>>>(wp, n_groups, wq, sp, bp);   \
    else                                                                                        \
      quantize_kernel<T, B, MFX_QMODE_DOC><<<blocks, 256, 0, st>>>(wp, n_groups, wq, sp, bp);   \
    break;
  switch (bits) {
    MFX_QUANT_CASE(3)
    MFX_QUANT_CASE(4)
    MFX_QUANT_CASE(5)
    MFX_QUANT_CASE(6)
    MFX_QUANT_CASE(8)
    default: return MFX_ERR_UNSUPPORTED_BITS;
  }
#undef MFX_QUANT_CASE
  MFX_CUDA_TRY(cudaGetLastError());
  return MFX_OK;
}

template <typename SB, typename OUT, int BITS>
void launch_dequantize_bits(const uint32_t* wq, const SB* scales, const SB* biases, int64_t values, OUT* out,
                            cudaStream_t st) {
  auto blocks = [&](int v) { return static_cast<unsigned>((values / v + 255) / 256); };
  // Sixteen values a thread halve the threads and the scale loads, which pays once the output fills the GPU many times
  // over (8 M values of float32, 32 M of 16 bits); below that fewer threads hide less of a trip to memory, and at 5 and 6
  // bits the gathering of ten or twelve bytes from 16-bit words outweighs it in 16-bit outputs. Buffers past L2, us, 8 / 16
  // values: to bf16, 12288 x 3072, 4 bits 22.4 / 22.0, 8 bits 22.9 / 21.9, 6 bits 25.5 / 26.9; 6144 x 3072, 3 bits 12.1 /
  // 12.5; 3072 x 3072, 4 bits 6.9 / 7.2, 6 bits 8.1 / 9.0; to float32, 3072 x 3072, 4 bits 12.9 / 12.7, 6 bits 14.8 / 13.5;
  // 1024 x 3072, 3 bits 5.9 / 6.0; 256 x 256 2.1 / 2.3.
  constexpr bool few = sizeof(OUT) == 2 && (BITS == 5 || BITS == 6);
  if (!few && values >= (sizeof(OUT) == 4 ? 8 << 20 : 32 << 20))
    dequantize_kernel<SB, OUT, BITS, 16><<<blocks(16), 256, 0, st>>>(wq, scales, biases, values / 16, out);
  else
    dequantize_kernel<SB, OUT, BITS, 8><<<blocks(8), 256, 0, st>>>(wq, scales, biases, values / 8, out);
}

template <typename SB, typename OUT>
int launch_dequantize(const uint32_t* wq, const void* scales, const void* biases, int64_t values, int bits,
                      void* out, cudaStream_t st) {
  const SB* sp = static_cast<const SB*>(scales);
  const SB* bp = static_cast<const SB*>(biases);
  OUT* op = static_cast<OUT*>(out);
  switch (bits) {
    case 3: launch_dequantize_bits<SB, OUT, 3>(wq, sp, bp, values, op, st); break;
    case 4: launch_dequantize_bits<SB, OUT, 4>(wq, sp, bp, values, op, st); break;
    case 5: launch_dequantize_bits<SB, OUT, 5>(wq, sp, bp, values, op, st); break;
    case 6: launch_dequantize_bits<SB, OUT, 6>(wq, sp, bp, values, op, st); break;
    case 8: launch_dequantize_bits<SB, OUT, 8>(wq, sp, bp, values, op, st); break;
    default: return MFX_ERR_UNSUPPORTED_BITS;
  }
  MFX_CUDA_TRY(cudaGetLastError());
  return MFX_OK;
}

template <typename SB>
int dispatch_dequant_out(const uint32_t* wq, const void* scales, const void* biases, int64_t values, int bits,
                         void* out, int out_dtype, cudaStream_t st) {
  switch (out_dtype) {
    case MFX_F32: return launch_dequantize<SB, float>(wq, scales, biases, values, bits, out, st);
    case MFX_BF16: return launch_dequantize<SB, __nv_bfloat16>(wq, scales, biases, values, bits, out, st);
    case MFX_F16: return launch_dequantize<SB, __half>(wq, scales, biases, values, bits, out, st);
    default: return MFX_ERR_DTYPE;
  }
}

}  // namespace
}  // namespace mfx

extern "C" {

int mfx_quantize_affine(const void* w, int w_dtype, int64_t N, int64_t K, int bits, int group_size, int qmode,
                        uint32_t* wq, void* scales, void* biases, void* stream) {
  using namespace mfx;
  if (!w || !wq || !scales || !biases) return MFX_ERR_NULL;
  if (!valid_bits(bits) || group_size != 64) return MFX_ERR_UNSUPPORTED_BITS;
  if (qmode != MFX_QMODE_MLX && qmode != MFX_QMODE_DOC) return MFX_ERR_SHAPE;
  if (N <= 0 || K <= 0 || K % 64 != 0) return MFX_ERR_SHAPE;
  if (!valid_dtype(w_dtype)) return MFX_ERR_DTYPE;
  if (!aligned16(w) || !aligned16(wq)) return MFX_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t n_groups = N * (K / 64);
  switch (w_dtype) {
    case MFX_F32: return launch_quantize<float>(w, n_groups, bits, qmode, wq, scales, biases, st);
    case MFX_BF16: return launch_quantize<__nv_bfloat16>(w, n_groups, bits, qmode, wq, scales, biases, st);
    default: return launch_quantize<__half>(w, n_groups, bits, qmode, wq, scales, biases, st);
  }
}

int mfx_dequantize_affine(const uint32_t* wq, const void* scales, const void* biases, int sb_dtype, int64_t N,
                          int64_t K, int bits, int group_size, void* out, int out_dtype, void* stream) {
  using namespace mfx;
  if (!wq || !scales || !biases || !out) return MFX_ERR_NULL;
  if (!valid_bits(bits) || group_size != 64) return MFX_ERR_UNSUPPORTED_BITS;
  if (N <= 0 || K <= 0 || K % 64 != 0) return MFX_ERR_SHAPE;
  if (!valid_dtype(sb_dtype) || !valid_dtype(out_dtype)) return MFX_ERR_DTYPE;
  if (!aligned16(wq) || !aligned16(out)) return MFX_ERR_ALIGN;
  if (int rc = check_arch()) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t values = N * K;
  switch (sb_dtype) {
    case MFX_F32: return dispatch_dequant_out<float>(wq, scales, biases, values, bits, out, out_dtype, st);
    case MFX_BF16:
      return dispatch_dequant_out<__nv_bfloat16>(wq, scales, biases, values, bits, out, out_dtype, st);
    default: return dispatch_dequant_out<__half>(wq, scales, biases, values, bits, out, out_dtype, st);
  }
}

}  // extern "C"
