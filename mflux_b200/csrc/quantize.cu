// Group-wise affine weight quantizer and dequantizer (HBM-bound, load-time kernels).
//
// Semantics follow mx.quantize(w, group_size=64, bits) as reached from the reference through
// mlx.nn.quantize (src/mflux/models/common/weights/loading/weight_applier.py:93-103): groups of 64
// along the input dimension, float32 arithmetic, codes packed little-end first: code j of a row occupies
// bits [j*bits, (j+1)*bits) of the row's bit stream, which for 4 and 8 bits is "8 / 4 codes per uint32" and for
// 3, 5 and 6 bits (the other widths the reference's CLI offers, src/mflux/cli/defaults/defaults.py:63) lets
// codes straddle byte and word boundaries (8 codes in 3 or 5 bytes, 4 codes in 3 bytes).
// Two or four lanes own one group; min/max go through warp shuffles.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "host_util.cuh"
#include "launch.cuh"

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

__device__ __forceinline__ void st_32(void* p, const uint4& a, const uint4& b) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z),
               "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
               : "memory");
}

// The PT (16 or 32) values of a thread as they lie in memory: 16-bit values two to a register, whose extremes are taken in
// pairs.
template <typename T, int PT>
struct Values {
  using Pair = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
  Pair h[PT / 2];
  __device__ __forceinline__ void load(const T* p) {
#pragma unroll
    for (int i = 0; i < PT / 8; ++i) {
      const uint4 raw = reinterpret_cast<const uint4*>(p)[i];
      const Pair* r = reinterpret_cast<const Pair*>(&raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[4 * i + j] = r[j];
    }
  }
  __device__ __forceinline__ void extremes(float& mx, float& mn) const {
    Pair hi = h[0], lo = h[0];
#pragma unroll
    for (int i = 1; i < PT / 2; ++i) {
      hi = __hmax2(hi, h[i]);
      lo = __hmin2(lo, h[i]);
    }
    mx = fmaxf(to_f32<T>(hi.x), to_f32<T>(hi.y));
    mn = fminf(to_f32<T>(lo.x), to_f32<T>(lo.y));
  }
  __device__ __forceinline__ float get(int i) const { return to_f32<T>(i & 1 ? h[i / 2].y : h[i / 2].x); }
};
template <int PT>
struct Values<float, PT> {
  float f[PT];
  __device__ __forceinline__ void load(const float* p) {
#pragma unroll
    for (int i = 0; i < PT / 4; ++i) {
      const float4 a = reinterpret_cast<const float4*>(p)[i];
      f[4 * i] = a.x; f[4 * i + 1] = a.y; f[4 * i + 2] = a.z; f[4 * i + 3] = a.w;
    }
  }
  __device__ __forceinline__ void extremes(float& mx, float& mn) const {
    mx = mn = f[0];
#pragma unroll
    for (int i = 1; i < PT; ++i) {
      mx = fmaxf(mx, f[i]);
      mn = fminf(mn, f[i]);
    }
  }
  __device__ __forceinline__ float get(int i) const { return f[i]; }
};

__device__ __forceinline__ uint64_t pair_f32(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void split_f32(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// The quantizer's definition of a code: the correctly rounded quotient, rounded to even, clamped.
__device__ __forceinline__ float exact_code(float d, float scale, float n_bins) {
  float q = rintf(__fdiv_rn(d, scale));
  if (!(fabsf(q) <= 3.0e38f)) q = 0.0f;  // constant group with scale == 0: code 0
  return fminf(fmaxf(q, 0.0f), n_bins);
}

// One thread: PT consecutive values of a row; 64 / PT neighbouring lanes form one group.
// Instruction issue bounds it, so: sums, products and roundings go in packed pairs of float32 (each half rounds like the
// scalar instruction), extremes of 16-bit weights in packed pairs of them, clamping in packed pairs of 16-bit integers,
// and with PT = 32 twice as many values share the scale's handful of divisions.
// A division per value is replaced by the reciprocal of the scale and the rounded product where that must be the rounded
// quotient too: reciprocal, product and the quotient itself are each off by at most 2^-24 of their value, together 1.8e-7
// of at most n_bins + 1, so a product further than that from every k + 0.5 rounds like the quotient. Values nearer to one
// (one in 1000 at 4 bits) are divided.
template <typename T, int BITS, int QMODE, int PT>
__global__ void __launch_bounds__(128) quantize_kernel(const T* w, int64_t n_groups_total,
                                                       uint32_t* wq, T* scales,
                                                       T* biases) {
  wait_for_predecessor();
  allow_successor();
  const int64_t tid = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  constexpr int LANES = 64 / PT;                  // of a group
  const int64_t group = tid / LANES;
  const bool active = group < n_groups_total;
  const int64_t g = active ? group : n_groups_total - 1;  // keep whole warps in the shuffles
  const int sub = static_cast<int>(tid % LANES);
  Values<T, PT> v;
  v.load(w + g * 64 + sub * PT);
  float mx, mn;
  v.extremes(mx, mn);
#pragma unroll
  for (int o = LANES / 2; o >= 1; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
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
  // the reciprocal has to be a normal number; a negative limit sends every value to the division
  const float limit = mag > 1e-30f && mag < 1e30f ? 0.5f - (n_bins + 1.0f) * 2.4e-7f : -1.0f;
  const float inv = __frcp_rn(scale);
  constexpr float MAGIC = 12582912.0f;            // 1.5 * 2^23: adding it rounds to even at the units place
  const uint64_t inv2 = pair_f32(inv, inv), neg_bias2 = pair_f32(-bias, -bias), magic2 = pair_f32(MAGIC, MAGIC),
                 neg_magic2 = pair_f32(-MAGIC, -MAGIC), minus2 = pair_f32(-1.0f, -1.0f);
  constexpr int WORDS = (BITS * PT + 31) / 32;
  uint32_t word[WORDS + 1];                       // the thread's codes
#pragma unroll
  for (int i = 0; i <= WORDS; ++i) word[i] = 0;
#pragma unroll
  for (int k = 0; k < PT / 8; ++k) {              // eight values
    float t[8], off[8];                           // MAGIC + code; distance of the product from its integer
    float far = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      uint64_t r2 = pair_f32(v.get(8 * k + i), v.get(8 * k + i + 1)), t2, e2;
      asm("add.rn.f32x2 %0, %0, %1;" : "+l"(r2) : "l"(neg_bias2));
      asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(r2) : "l"(inv2));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(t2) : "l"(r2), "l"(magic2));
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(e2) : "l"(t2), "l"(neg_magic2));
      asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(e2) : "l"(minus2), "l"(r2));
      split_f32(t2, t[i], t[i + 1]);
      split_f32(e2, off[i], off[i + 1]);
      far = fmaxf(far, fmaxf(fabsf(off[i]), fabsf(off[i + 1])));
    }
    if (far > limit) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (!(fabsf(off[i]) <= limit))
          t[i] = __fadd_rn(exact_code(__fsub_rn(v.get(8 * k + i), bias), scale, n_bins), MAGIC);
    }
    // codes clamped to [0, n_bins] in 16-bit pairs (i, i + 4): the low half of MAGIC + code is the code, also below zero
    uint32_t c[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      c[i] = __vimin_s16x2_relu(__byte_perm(__float_as_uint(t[i]), __float_as_uint(t[i + 4]), 0x5410),
                                ((1u << BITS) - 1u) * 0x10001u);
    if constexpr (BITS == 4) {
      word[k] = c[0] + c[1] * 16u + c[2] * 256u + c[3] * 4096u;
    } else if constexpr (BITS == 8) {
      word[2 * k] = __byte_perm(c[0] + c[1] * 256u, c[2] + c[3] * 256u, 0x5410);
      word[2 * k + 1] = __byte_perm(c[0] + c[1] * 256u, c[2] + c[3] * 256u, 0x7632);
    } else {
      // eight codes are 8 * BITS bits of the stream, from bit 8 * BITS * k of the thread's
      unsigned long long eight = 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        eight |= static_cast<unsigned long long>(c[i] & 0xFFFFu) << (BITS * i);
        eight |= static_cast<unsigned long long>(c[i] >> 16) << (BITS * (i + 4));
      }
      constexpr int LEN = 8 * BITS;
      const int at = (LEN * k) / 32, sh = (LEN * k) % 32;
      word[at] |= static_cast<uint32_t>(eight << sh);
      if (sh + LEN > 32) word[at + 1] |= static_cast<uint32_t>((eight << sh) >> 32);
    }
  }
  if (!active) return;
  if constexpr (BITS == 4 || BITS == 8) {
    uint32_t* dst = wq + (g * LANES + sub) * WORDS;
    if constexpr (WORDS == 2) {
      *reinterpret_cast<uint2*>(dst) = make_uint2(word[0], word[1]);
    } else {
#pragma unroll
      for (int i = 0; i < WORDS; i += 4)
        *reinterpret_cast<uint4*>(dst + i) = make_uint4(word[i], word[i + 1], word[i + 2], word[i + 3]);
    }
  } else if constexpr (PT == 32) {
    uint32_t* dst = wq + (g * LANES + sub) * BITS;
#pragma unroll
    for (int i = 0; i < BITS; ++i) dst[i] = word[i];
  } else {                                        // 16 codes are BITS 16-bit words at an even address
    uint16_t* dst = reinterpret_cast<uint16_t*>(wq) + (g * LANES + sub) * BITS;
#pragma unroll
    for (int i = 0; i < BITS; ++i) dst[i] = static_cast<uint16_t>(word[i / 2] >> (16 * (i & 1)));
  }
  if (sub == 0) {
    scales[g] = from_f32<T>(scale);
    biases[g] = from_f32<T>(bias);
  }
}

// One thread: V (8 or 16) consecutive outputs of a row.
template <typename SB, typename OUT, int BITS, int V>
__global__ void __launch_bounds__(256) dequantize_kernel(const uint32_t* wq,
                                                         const SB* scales,
                                                         const SB* biases, int64_t n_chunks,
                                                         bool wide, OUT* out) {
  wait_for_predecessor();
  allow_successor();
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
      words[0] = wq[tid];
    } else if constexpr (WORDS == 2) {
      const uint2 v = reinterpret_cast<const uint2*>(wq)[tid];
      words[0] = v.x; words[1] = v.y;
    } else {
      const uint4 v = reinterpret_cast<const uint4*>(wq)[tid];
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
      for (int i = 0; i < BITS; ++i) eight[0] |= static_cast<unsigned long long>(src[i]) << (8 * i);
    } else {
      const uint16_t* src = reinterpret_cast<const uint16_t*>(wq) + tid * BITS;
      unsigned long long w0 = 0, w1 = 0;
#pragma unroll
      for (int i = 0; i < BITS; ++i) {
        const unsigned long long v = src[i];
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
  const uint4* from = reinterpret_cast<const uint4*>(res);
  constexpr int VECS = V * static_cast<int>(sizeof(OUT)) / 16;
  if (VECS > 1 && wide) {
#pragma unroll
    for (int i = 0; i + 1 < VECS; i += 2) st_32(dst + i, from[i], from[i + 1]);
  } else {
#pragma unroll
    for (int i = 0; i < VECS; ++i) dst[i] = from[i];
  }
}

template <typename T, int BITS, int PT>
cudaError_t launch_quantize_pt(const T* w, int64_t n_groups, int qmode, uint32_t* wq, T* scales, T* biases,
                               cudaStream_t st) {
  const unsigned blocks = static_cast<unsigned>((n_groups * (64 / PT) + 127) / 128);
  return launch_overlapped(qmode == MFX_QMODE_MLX ? quantize_kernel<T, BITS, MFX_QMODE_MLX, PT>
                                                  : quantize_kernel<T, BITS, MFX_QMODE_DOC, PT>,
                           blocks, 128, 0, st, w, n_groups, wq, scales, biases);
}

// Values a thread takes of 16-bit weights: 32 share the scale's divisions once there are threads enough without 16. us,
// 16 / 32 values, bf16, 4 bits (8 bits): 12288 x 3072 28.0 / 25.5 (32.6 / 29.0), 3072 x 3072 9.2 / 8.9 (10.2 / 9.7), 1024 x
// 512 2.65 / 3.24 (2.99 / 3.76); before, at 16 values and unpacked, 41.7 (44.4), 13.5 (13.6) and 2.9 (3.0). Float32 weights
// would need 128 bytes per thread at 32: 28 us at 16 for 12288 x 3072, 37 at 32 (29 before).
constexpr int64_t LARGE_WEIGHT = 4 << 20;
template <typename T, int BITS>
cudaError_t launch_quantize_bits(const T* w, int64_t n_groups, int qmode, uint32_t* wq, T* scales, T* biases,
                                 cudaStream_t st) {
  if constexpr (sizeof(T) == 2) {
    if (n_groups * 64 >= LARGE_WEIGHT) return launch_quantize_pt<T, BITS, 32>(w, n_groups, qmode, wq, scales, biases, st);
  }
  return launch_quantize_pt<T, BITS, 16>(w, n_groups, qmode, wq, scales, biases, st);
}

template <typename T>
int launch_quantize(const void* w, int64_t n_groups, int bits, int qmode, uint32_t* wq, void* scales, void* biases,
                    cudaStream_t st) {
  const T* wp = static_cast<const T*>(w);
  T* sp = static_cast<T*>(scales);
  T* bp = static_cast<T*>(biases);
  switch (bits) {
    case 3: MFX_CUDA_TRY((launch_quantize_bits<T, 3>(wp, n_groups, qmode, wq, sp, bp, st))); break;
    case 4: MFX_CUDA_TRY((launch_quantize_bits<T, 4>(wp, n_groups, qmode, wq, sp, bp, st))); break;
    case 5: MFX_CUDA_TRY((launch_quantize_bits<T, 5>(wp, n_groups, qmode, wq, sp, bp, st))); break;
    case 6: MFX_CUDA_TRY((launch_quantize_bits<T, 6>(wp, n_groups, qmode, wq, sp, bp, st))); break;
    case 8: MFX_CUDA_TRY((launch_quantize_bits<T, 8>(wp, n_groups, qmode, wq, sp, bp, st))); break;
    default: return MFX_ERR_UNSUPPORTED_BITS;
  }
  return MFX_OK;
}

template <typename SB, typename OUT, int BITS>
cudaError_t launch_dequantize_bits(const uint32_t* wq, const SB* scales, const SB* biases, int64_t values, OUT* out,
                                   cudaStream_t st) {
  auto blocks = [&](int v) { return static_cast<unsigned>((values / v + 255) / 256); };
  // Sixteen values a thread, stored 32 bytes at a time, from 8 M values on; below that fewer threads hide less of a trip to
  // memory. Stores are what bounds it: 16 bytes at a time leave half of every sector to a second instruction. Buffers past
  // L2, us, 16-byte stores / 8 values and 32-byte stores where 8 values have them / 16: to bf16, 12288 x 3072, 4 bits 21.9 /
  // 21.9 / 17.0, 6 bits 25.2 / 24.4 / 20.7, 3072 x 3072, 4 bits 5.0 / 5.6 / 4.3, 6 bits 6.1 / 6.2 / 5.3, 3072 x 1024, 4 bits
  // 2.7 / 2.5 / 2.5; to float32, 12288 x 3072, 4 bits 42.9 / - / 26.9, 3072 x 1024 4.9 / 3.0 / 3.6.
  const bool wide = (reinterpret_cast<uintptr_t>(out) & 31u) == 0;   // the entry point promises 16
  if (wide && values >= (8 << 20))
    return launch_overlapped(dequantize_kernel<SB, OUT, BITS, 16>, blocks(16), 256, 0, st, wq, scales, biases, values / 16,
                             wide, out);
  return launch_overlapped(dequantize_kernel<SB, OUT, BITS, 8>, blocks(8), 256, 0, st, wq, scales, biases, values / 8, wide,
                           out);
}

template <typename SB, typename OUT>
int launch_dequantize(const uint32_t* wq, const void* scales, const void* biases, int64_t values, int bits,
                      void* out, cudaStream_t st) {
  const SB* sp = static_cast<const SB*>(scales);
  const SB* bp = static_cast<const SB*>(biases);
  OUT* op = static_cast<OUT*>(out);
  switch (bits) {
    case 3: MFX_CUDA_TRY((launch_dequantize_bits<SB, OUT, 3>(wq, sp, bp, values, op, st))); break;
    case 4: MFX_CUDA_TRY((launch_dequantize_bits<SB, OUT, 4>(wq, sp, bp, values, op, st))); break;
    case 5: MFX_CUDA_TRY((launch_dequantize_bits<SB, OUT, 5>(wq, sp, bp, values, op, st))); break;
    case 6: MFX_CUDA_TRY((launch_dequantize_bits<SB, OUT, 6>(wq, sp, bp, values, op, st))); break;
    case 8: MFX_CUDA_TRY((launch_dequantize_bits<SB, OUT, 8>(wq, sp, bp, values, op, st))); break;
    default: return MFX_ERR_UNSUPPORTED_BITS;
  }
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
