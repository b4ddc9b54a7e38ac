// Quantized linear for at most 16 activation rows (the AdaLN / embedder linears that see one vector per image):
// y[M, N] = x[M, K] . dequant(W)^T + bias, M <= 16. The work is streaming the packed weights once, so the kernel
// is laid out for HBM bandwidth, not for the tcgen05 pipeline of the large-M kernel:
//   * it reads the same prepared weight blob (codes with the nibble / byte order that gives two neighbouring
//     values per mask, scale|bias pairs transposed to [group][N]);
//   * a warp owns R groups of 8 weight rows and every eighth 128-wide slice of K; a lane loads 16 bytes of codes
//     per group and slice (32 or 16 consecutive k of one row) and the group's pair, one slice ahead of their use;
//   * the 16 x 8 x 16 products run on mma.sync (bf16 in, f32 out) with the activation rows as A. A lane feeds the
//     k-slots of a step with its own four consecutive k, and reads the same four k of x for A: a dot product does
//     not care about the order of its terms, so no shuffle is needed to match the instruction's k layout;
//   * the eight warps' partial sums meet in shared memory; bias, SiLU and the store follow.
// Measured, the kernel moves 1.0-2.0 TB/s and its time follows the number of weights, not their bytes: five instructions
// per weight (issue slots 65 % busy while a block runs) and the trips to memory of short-lived blocks bound it, not HBM. A
// few rows over a large weight go to the kernel in namespace stream below.
// Reference call sites: every nn.Linear that is applied to a conditioning vector, e.g. the AdaLayerNormZero
// linears (src/mflux/models/flux/model/flux_transformer/ada_layer_norm_zero.py:16-18) and the time/text
// embedders (time_text_embed.py:19-31); after quantization they are mlx.nn.QuantizedLinear like all others.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "host_util.cuh"
#include "launch.cuh"
#include "scalar.cuh"
#include "qmv.cuh"

namespace mfx {
namespace qmv {

constexpr int THREADS = 256;
constexpr int WARPS = 8;

struct Params {
  const __nv_bfloat16* x;
  int64_t x_row_stride;
  int M, N, K;
  const uint32_t* codes;   // prepared codes [N][K * bits / 32]
  const uint32_t* sb;      // [K / 64][N]: bf16 scale | bf16 bias << 16
  const void* bias;
  int bias_dtype;
  int epilogue;            // MFX_EPI_NONE or MFX_EPI_SILU
  void* y;
  int y_dtype;
  int64_t y_row_stride;
};

__device__ __forceinline__ uint32_t sub_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
               "{%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

constexpr uint32_t MAGIC = 0x43004300u;  // bf16 pair (128.0, 128.0): OR-ing a 4-bit code gives 128 + code exactly

// Two neighbouring weights (k, k+1) of a 4-bit row: pair index i of a prepared word.
__device__ __forceinline__ uint32_t deq4(uint32_t w, int i, uint32_t scale2, uint32_t bias2) {
  const uint32_t v = ((w >> (4 * i)) & 0x000F000Fu) | MAGIC;
  return fma_bf16x2(sub_bf16x2(v, MAGIC), scale2, bias2);
}
// The four weights of one prepared 8-bit word (bytes e0,e2,e1,e3) as two bf16 pairs (e0,e1), (e2,e3), through
// float32: a byte under the exponent of 2^23 is the float 2^23 + code; packed f32x2 add and fma, one rounding to
// bf16 at the end (the same arithmetic as the large-M kernel's 8-bit path). sc2 / bi2: (scale, scale) and
// (bias, bias) as float32 pairs.
__device__ __forceinline__ void deq8_word(uint32_t w, uint64_t sc2, uint64_t bi2, uint32_t& b0, uint32_t& b1) {
  constexpr uint32_t TWO23 = 0x4B000000u;
  const uint64_t neg = 0xCB000000CB000000ull;  // (-2^23, -2^23)
  uint64_t v01, v23;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v01) : "r"(__byte_perm(w, TWO23, 0x7440)), "r"(__byte_perm(w, TWO23, 0x7442)));
  asm("mov.b64 %0, {%1, %2};" : "=l"(v23) : "r"(__byte_perm(w, TWO23, 0x7441)), "r"(__byte_perm(w, TWO23, 0x7443)));
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v01) : "l"(neg));
  asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v23) : "l"(neg));
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(v01) : "l"(sc2), "l"(bi2));
  asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(v23) : "l"(sc2), "l"(bi2));
  float a, b, c, d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v01));
  asm("mov.b64 {%0, %1}, %2;" : "=f"(c), "=f"(d) : "l"(v23));
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  b0 = *reinterpret_cast<const uint32_t*>(&lo);
  b1 = *reinterpret_cast<const uint32_t*>(&hi);
}

// R = groups of 8 weight rows per warp (the A fragments are reused across them). BITS = 4 or 8.
template <int BITS, int R>
__global__ void __launch_bounds__(THREADS) qmv_kernel(const Params p) {
  allow_successor();
  constexpr int KPL = 128 / BITS;            // k values a lane covers per slice with one 16-byte load: 32 or 16
  constexpr int SLICE = 4 * KPL;             // k per slice: 128 (4-bit) or 64 (8-bit)
  constexpr int STEPS = KPL / 4;             // mma steps per slice: 8 or 4
  __shared__ float red[WARPS][R][32][4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n_base = blockIdx.x * (8 * R);
  const int words_per_row = p.K * BITS / 32;
  const int slices = (p.K + SLICE - 1) / SLICE;

  float acc[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = acc[r][2] = acc[r][3] = 0.f;

  const bool row_lo = g < p.M, row_hi = g + 8 < p.M;
  const __nv_bfloat16* x_lo = p.x + static_cast<int64_t>(g) * p.x_row_stride;
  const __nv_bfloat16* x_hi = p.x + static_cast<int64_t>(g + 8) * p.x_row_stride;

  // codes (16 bytes) and (scale, bias) pairs of the R rows for one slice, loaded one iteration ahead of their use: a
  // load at its point of use exposes a trip to HBM per slice. With only the codes ahead, M 1, 4 bits: N 3072, K 15360
  // 21.6 us, N 18432, K 3072 16.7 us; with the pairs too 16.3 and 15.5 us. Two or three slices ahead need 64 to 117
  // registers and lose more in resident blocks than they gain (17.9 and 18.9 us on the second shape).
  auto load_slice = [&](int s, uint4 (&wv)[R], uint32_t (&pv)[R]) {
    const int k0 = s * SLICE + t * KPL;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int n = n_base + 8 * r + g;
      const bool live = s < slices && k0 < p.K && n < p.N;
      wv[r] = live ? __ldg(reinterpret_cast<const uint4*>(p.codes + static_cast<int64_t>(n) * words_per_row +
                                                          k0 * BITS / 32))
                   : make_uint4(0, 0, 0, 0);
      pv[r] = live ? __ldg(p.sb + static_cast<int64_t>(k0 >> 6) * p.N + n) : 0u;
    }
  };
  uint4 wnext[R];
  uint32_t pnext[R];
  load_slice(warp, wnext, pnext);
  for (int s = warp; s < slices; s += WARPS) {
    const int k0 = s * SLICE + t * KPL;      // first k of this lane in the slice
    const bool live = k0 < p.K;              // ragged last slice (K is a multiple of 64, a 4-bit slice is 128):
                                             // dead lanes feed zeros, every lane still takes part in the mma
    uint4 wv[R];
    uint32_t pv[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      wv[r] = wnext[r];
      pv[r] = pnext[r];
    }
    load_slice(s + WARPS, wnext, pnext);
    // activations of rows g and g + 8 for the same k (KPL values = KPL / 8 16-byte loads each)
    uint32_t xa[KPL / 2], xb[KPL / 2];
#pragma unroll
    for (int i = 0; i < KPL / 8; ++i) {
      const uint4 a = (live && row_lo) ? __ldg(reinterpret_cast<const uint4*>(x_lo + k0) + i) : make_uint4(0, 0, 0, 0);
      const uint4 b = (live && row_hi) ? __ldg(reinterpret_cast<const uint4*>(x_hi + k0) + i) : make_uint4(0, 0, 0, 0);
      xa[4 * i] = a.x; xa[4 * i + 1] = a.y; xa[4 * i + 2] = a.z; xa[4 * i + 3] = a.w;
      xb[4 * i] = b.x; xb[4 * i + 1] = b.y; xb[4 * i + 2] = b.z; xb[4 * i + 3] = b.w;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t sbv = pv[r];
      const uint32_t scale2 = __byte_perm(sbv, sbv, 0x1010), bias2 = __byte_perm(sbv, sbv, 0x3232);
      uint64_t sc2 = 0, bi2 = 0;
      if (BITS == 8) {   // the same scale and bias as float32 pairs
        asm("mov.b64 %0, {%1, %1};" : "=l"(sc2) : "r"(sbv << 16));
        asm("mov.b64 %0, {%1, %1};" : "=l"(bi2) : "r"(sbv & 0xFFFF0000u));
      }
      const uint32_t w[4] = {wv[r].x, wv[r].y, wv[r].z, wv[r].w};
#pragma unroll
      for (int st = 0; st < STEPS; ++st) {
        uint32_t b0, b1;
        if (BITS == 4) {
          b0 = deq4(w[st >> 1], 2 * (st & 1), scale2, bias2);
          b1 = deq4(w[st >> 1], 2 * (st & 1) + 1, scale2, bias2);
        } else {
          deq8_word(w[st], sc2, bi2, b0, b1);
        }
        mma_16816(acc[r], xa[2 * st], xb[2 * st], xa[2 * st + 1], xb[2 * st + 1], b0, b1);
      }
    }
  }

#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int i = 0; i < 4; ++i) red[warp][r][lane][i] = acc[r][i];
  __syncthreads();
  // 16 x (8 R) outputs per block; accumulator i of lane (g, t): row g + 8 * (i >> 1), column 2 t + (i & 1)
  for (int o = threadIdx.x; o < R * 128; o += THREADS) {
    const int r = o >> 7, l = (o >> 2) & 31, i = o & 3;
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) v += red[w][r][l][i];
    const int m = (l >> 2) + 8 * (i >> 1);
    const int n = n_base + 8 * r + 2 * (l & 3) + (i & 1);
    if (m < p.M && n < p.N) {
      if (p.bias) v += load_as_float(p.bias, p.bias_dtype, n);
      if (p.epilogue == MFX_EPI_SILU) v = v / (1.0f + __expf(-v));
      if (p.y_dtype == MFX_F32) static_cast<float*>(p.y)[m * p.y_row_stride + n] = v;
      else static_cast<__nv_bfloat16*>(p.y)[m * p.y_row_stride + n] = __float2bfloat16_rn(v);
    }
  }
}

// A few rows over a large weight: one block of 16 warps per SM, every warp with a ring of its own in shared memory
// that cp.async fills a piece ahead, so that the copies run on while the warps compute. A piece is 16 weight rows x 256
// bytes of codes (512 or 256 k) and their (scale, bias) pairs. S warps share a tile of 16 rows; tiles are dealt out to the
// blocks in turn.
// Instructions are the next bound, so no weight is formed: the products are Sum x (128 + code) (4 bits) or Sum x code (8
// bits) of one group on mma.sync, with the weights as the 16-row operand, and scale, bias and the offset come in once per
// group, in float32: scale * (P - 128 X) + bias * X with X = Sum x, which every block computes once. That leaves out the
// rounding of the weights to bf16, too: 1e-6 (4 bits) and 1e-7 (8 bits) from float64 in the 2-norm, where the other kernels
// are 1.1e-3 off.
namespace stream {

constexpr int NWARPS = 16;
constexpr int ROWS = 16;                    // weight rows per tile
constexpr int MAX_SMEM = 227 * 1024;
constexpr int ROW_BYTES = 256;              // codes of one row in a piece
constexpr int RING = 2;                     // 128-byte pieces with 4 or 5 in a ring: 10 % slower
constexpr int CODES_BYTES = ROWS * ROW_BYTES;

template <int BITS>
struct Piece {
  static constexpr int K = ROW_BYTES * 8 / BITS;       // 512 or 256
  static constexpr int GROUPS = K / 64;                // 8 or 4
  static constexpr int BYTES = CODES_BYTES + GROUPS * ROWS * 4;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// 16 codes of one weight row in K order as the A fragments of four products, pairs 2 i and 2 i + 1 of product i; 4 bits:
// 128 + code, 8 bits: the code, both exact in bf16.
__device__ __forceinline__ void unpack16(const uint2& w, uint32_t (&a)[8]) {
  const uint32_t v[2] = {w.x, w.y};
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = ((v[i >> 2] >> (4 * (i & 3))) & 0x000F000Fu) | MAGIC;
}
__device__ __forceinline__ void unpack16(const uint4& w, uint32_t (&a)[8]) {
  constexpr uint32_t TWO23 = 0x4B000000u;
  const uint64_t neg = 0xCB000000CB000000ull;  // (-2^23, -2^23)
  const uint32_t v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {                // prepared byte order e0, e2, e1, e3
    uint64_t f;
    asm("mov.b64 %0, {%1, %2};"
        : "=l"(f)
        : "r"(__byte_perm(v[i >> 1], TWO23, i & 1 ? 0x7441 : 0x7440)),
          "r"(__byte_perm(v[i >> 1], TWO23, i & 1 ? 0x7443 : 0x7442)));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(f) : "l"(neg));
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(f));
    a[i] = __byte_perm(lo, hi, 0x7632);        // eight significant bits: the upper halves are exact
  }
}

// Shared memory: rings | partial sums [NWARPS][4][32] | X [K / 64][8] | x [M][K] bf16, rows 16 bytes apart (two rows of a
// quarter warp then read different halves of the banks).
template <int BITS>
__host__ __device__ constexpr int x_offset() {
  return NWARPS * RING * Piece<BITS>::BYTES + NWARPS * 4 * 32 * 4;
}

// One output term by term, on weights rounded to bf16. For sums that are not finite: where an activation is infinite or near
// the largest float, P and 128 X (or bias * X) are infinities of either sign although the terms' own sum is not NaN.
template <int BITS>
__device__ __noinline__ float direct_dot(const uint32_t* row, const uint32_t* sb, int64_t sb_stride,
                                         const __nv_bfloat16* x_row, int K) {
  const unsigned short* x = reinterpret_cast<const unsigned short*>(x_row);
  float sum = 0.f;
  for (int k = 0; k < K; ++k) {
    const uint32_t pair = sb[(k >> 6) * sb_stride];
    constexpr int PER_WORD = 32 / BITS;
    const int e = k % PER_WORD;                // prepared order: nibbles e0,e2,e4,e6,e1,e3,e5,e7; bytes e0,e2,e1,e3
    const int at = BITS == 4 ? (e >> 1) + 4 * (e & 1) : (e >> 1) + 2 * (e & 1);
    const uint32_t code = (row[k / PER_WORD] >> (BITS * at)) & ((1u << BITS) - 1u);
    const float w = fmaf(static_cast<float>(code), __uint_as_float(pair << 16), __uint_as_float(pair & 0xFFFF0000u));
    const float xv = __uint_as_float(static_cast<uint32_t>(x[k]) << 16);
    sum = fmaf(__bfloat162float(__float2bfloat16_rn(w)), xv, sum);
  }
  return sum;
}

template <int BITS>
int smem_bytes(int M, int K) {
  return x_offset<BITS>() + K / 64 * 32 + M * (2 * K + 16);
}

template <int BITS, int S>
__global__ void __launch_bounds__(NWARPS * 32, 1) stream_kernel(const Params p) {
  using P = Piece<BITS>;
  using Codes = typename std::conditional<BITS == 4, uint2, uint4>::type;   // a lane's 16 codes of a group
  constexpr int TILES = NWARPS / S;          // tiles a block works on at a time
  extern __shared__ __align__(128) uint8_t smem[];
  wait_for_predecessor();
  allow_successor();
  const int block = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int part = warp % S, slot = warp / S;
  const int groups = p.K >> 6;
  const int tiles = (p.N + ROWS - 1) / ROWS;
  const int pieces = (groups + P::GROUPS - 1) / P::GROUPS;
  const int mine = part < pieces ? (pieces - part + S - 1) / S : 0;          // pieces of a tile that are this warp's
  const int rounds = (tiles + TILES * static_cast<int>(gridDim.x) - 1) / (TILES * static_cast<int>(gridDim.x));
  const int64_t row_bytes = static_cast<int64_t>(p.K) * BITS / 8;
  uint8_t* ring = smem + warp * (RING * P::BYTES);
  const uint32_t ring_s = static_cast<uint32_t>(__cvta_generic_to_shared(ring));
  float* red = reinterpret_cast<float*>(smem + NWARPS * RING * P::BYTES);
  float* xsum = reinterpret_cast<float*>(smem + x_offset<BITS>());
  auto tile_of = [&](int round) { return (round * TILES + slot) * static_cast<int>(gridDim.x) + block; };

  // piece number `k` of this warp's sequence (rounds one after the other) into ring slot k % RING
  int next = 0, next_round = 0, next_piece = part;
  auto issue = [&]() {
    if (next_round < rounds && mine > 0) {
      const int tile = tile_of(next_round);
      if (tile < tiles) {
        const uint32_t dst = ring_s + (next % RING) * P::BYTES;
        const int n0 = tile * ROWS;
        const int64_t off = static_cast<int64_t>(next_piece) * ROW_BYTES;
#pragma unroll
        for (int i = 0; i < CODES_BYTES / 16 / 32; ++i) {
          const int id = i * 32 + lane, row = id / (ROW_BYTES / 16), c = id % (ROW_BYTES / 16);
          // 16-byte chunks swizzled so that the rows of a quarter or half warp read different banks
          const int cs = BITS == 4 ? c ^ ((row & 3) << 1) : c ^ ((row & 1) << 2);
          if (off + c * 16 < row_bytes)
            cp_async16(dst + row * ROW_BYTES + cs * 16,
                       reinterpret_cast<const uint8_t*>(p.codes) + min(n0 + row, p.N - 1) * row_bytes + off + c * 16);
        }
        const int grp = next_piece * P::GROUPS + (lane >> 2), n = n0 + (lane & 3) * 4;
        if (lane < P::GROUPS * 4 && grp < groups && n < p.N)
          cp_async16(dst + CODES_BYTES + lane * 16, p.sb + static_cast<int64_t>(grp) * p.N + n);
      }
      ++next;
      next_piece += S;
      if (next_piece >= pieces) {
        next_piece = part;
        ++next_round;
      }
    }
    cp_async_commit();
  };
  for (int i = 0; i < RING - 1; ++i) issue();

  const int x_pitch = 2 * p.K + 16;
  uint8_t* xs_mem = smem + x_offset<BITS>() + groups * 32;
  for (int m = 0; m < p.M; ++m)
    for (int c = threadIdx.x; c < p.K / 8; c += NWARPS * 32)
      *reinterpret_cast<uint4*>(xs_mem + m * x_pitch + c * 16) =
          reinterpret_cast<const uint4*>(p.x + static_cast<int64_t>(m) * p.x_row_stride)[c];
  const uint8_t* x_mine = xs_mem + min(g, p.M - 1) * x_pitch + t * 32;

  // X[group][m]: four lanes sum a group of one row, 16 activations each
  for (int i = threadIdx.x; i < groups * p.M * 4; i += NWARPS * 32) {
    const int m = (i >> 2) / groups, grp = (i >> 2) - m * groups;
    const uint4* src =
        reinterpret_cast<const uint4*>(p.x + static_cast<int64_t>(m) * p.x_row_stride + grp * 64 + (i & 3) * 16);
    const uint4 v0 = src[0], v1 = src[1];
    const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      a += __uint_as_float(w[j] << 16);
      b += __uint_as_float(w[j] & 0xFFFF0000u);
    }
    a += b;
    const unsigned quad = 0xFu << (threadIdx.x & 28);    // the four lanes take the branch together
    a += __shfl_xor_sync(quad, a, 1);
    a += __shfl_xor_sync(quad, a, 2);
    if ((i & 3) == 0) xsum[grp * 8 + m] = a;
  }
  __syncthreads();

  int k = 0;
  for (int round = 0; round < rounds; ++round) {
    const int tile = tile_of(round);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int i = 0; i < mine; ++i, ++k) {
      __syncwarp();                          // the slot the next copies go to has been read
      issue();
      cp_async_wait<RING - 1>();
      __syncwarp();                          // every lane's copies of piece k have landed
      if (tile >= tiles) continue;
      const uint8_t* src = ring + (k % RING) * P::BYTES;
      const int g0 = (part + i * S) * P::GROUPS;
#pragma unroll
      for (int j = 0; j < P::GROUPS; ++j) {
        if (g0 + j >= groups) break;
        const uint4 v0 = *reinterpret_cast<const uint4*>(x_mine + (g0 + j) * 128);
        const uint4 v1 = *reinterpret_cast<const uint4*>(x_mine + (g0 + j) * 128 + 16);
        const int at = BITS == 4 ? ((2 * j) ^ ((g & 3) << 1)) * 16 + t * 8 : ((4 * j) ^ ((g & 1) << 2)) * 16 + t * 16;
        uint32_t lo[8], hi[8];
        unpack16(*reinterpret_cast<const Codes*>(src + g * ROW_BYTES + at), lo);
        unpack16(*reinterpret_cast<const Codes*>(src + (g + 8) * ROW_BYTES + at), hi);
        const uint32_t* pr = reinterpret_cast<const uint32_t*>(src + CODES_BYTES) + j * ROWS + g;
        const uint32_t p_lo = pr[0], p_hi = pr[8];
        const float2 xs = *reinterpret_cast<const float2*>(xsum + (g0 + j) * 8 + 2 * t);
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        mma_16816(d, lo[0], hi[0], lo[1], hi[1], v0.x, v0.y);
        mma_16816(d, lo[2], hi[2], lo[3], hi[3], v0.z, v0.w);
        mma_16816(d, lo[4], hi[4], lo[5], hi[5], v1.x, v1.y);
        mma_16816(d, lo[6], hi[6], lo[7], hi[7], v1.z, v1.w);
        if (BITS == 4) {
          d[0] = fmaf(-128.f, xs.x, d[0]);
          d[1] = fmaf(-128.f, xs.y, d[1]);
          d[2] = fmaf(-128.f, xs.x, d[2]);
          d[3] = fmaf(-128.f, xs.y, d[3]);
        }
        const float s_lo = __uint_as_float(p_lo << 16), b_lo = __uint_as_float(p_lo & 0xFFFF0000u);
        const float s_hi = __uint_as_float(p_hi << 16), b_hi = __uint_as_float(p_hi & 0xFFFF0000u);
        acc[0] = fmaf(s_lo, d[0], fmaf(b_lo, xs.x, acc[0]));
        acc[1] = fmaf(s_lo, d[1], fmaf(b_lo, xs.y, acc[1]));
        acc[2] = fmaf(s_hi, d[2], fmaf(b_hi, xs.x, acc[2]));
        acc[3] = fmaf(s_hi, d[3], fmaf(b_hi, xs.y, acc[3]));
      }
    }
    if constexpr (S > 1) {
      if (round > 0) __syncthreads();        // the sums of the round before have been read
#pragma unroll
      for (int i = 0; i < 4; ++i) red[(warp * 4 + i) * 32 + lane] = acc[i];
      __syncthreads();
      if (part == 0) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int o = 1; o < S; ++o) acc[i] += red[((warp + o) * 4 + i) * 32 + lane];
      }
    }
    if (part != 0 || tile >= tiles) continue;
    // accumulator i of lane (g, t): weight row g + 8 * (i >> 1) of the tile, activation row 2 t + (i & 1)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = tile * ROWS + 8 * h + g;
      if (n >= p.N) continue;
      const float bias = p.bias ? load_as_float(p.bias, p.bias_dtype, n) : 0.f;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int row = 2 * t + i;
        if (row >= p.M) continue;
        float v = acc[2 * h + i];
        if (!(fabsf(v) <= 3.0e38f))
          v = direct_dot<BITS>(p.codes + n * (row_bytes / 4), p.sb + n, p.N, p.x + row * p.x_row_stride, p.K);
        v += bias;
        if (p.epilogue == MFX_EPI_SILU) v = v / (1.0f + __expf(-v));
        if (p.y_dtype == MFX_F32) static_cast<float*>(p.y)[row * p.y_row_stride + n] = v;
        else static_cast<__nv_bfloat16*>(p.y)[row * p.y_row_stride + n] = __float2bfloat16_rn(v);
      }
    }
  }
}

template <int BITS, int S>
int launch(const Params& p, cudaStream_t st) {
  static SmemConfigured configured;
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(stream_kernel<BITS, S>), MAX_SMEM, configured)) return rc;
  const int blocks = std::min(device_sm_count(), (p.N + ROWS - 1) / ROWS);
  MFX_CUDA_TRY(launch_overlapped(stream_kernel<BITS, S>, blocks, NWARPS * 32, smem_bytes<BITS>(p.M, p.K), st, p));
  return MFX_OK;
}

// Warps per tile, by pieces a warp has over all rounds, a piece and a half for the barriers of every further round and 1.2 for
// every doubling of the warps that add their sums. us at 1 / 2 / 4 / 8, one row: N 18432, K 3072, 4 bits 13.1 / 12.4 / 15.8 /
// 16.3; N 9216, K 3072, 4 bits 10.6 / 9.2 / 10.4 / 10.8, 8 bits 12.9 / 10.7 / 10.1 / 11.0; N 12288, K 3072, 8 bits 16.5 / 12.7
// / 13.9 / 14.2; N 20480, K 3840, 8 bits 24.0 / 25.1 / 23.1 / 23.1; N 3072, K 15360, 4 bits 37.2 / 20.8 / 16.7 / 15.6.
template <int BITS>
int split(const Params& p) {
  const int64_t tiles = (p.N + ROWS - 1) / ROWS, pieces = (p.K + Piece<BITS>::K - 1) / Piece<BITS>::K;
  const int64_t warps = static_cast<int64_t>(NWARPS) * device_sm_count();
  int best = 1;
  int64_t best_cost = 0;                       // in tenths of a piece
  for (int s = 1, doublings = 0; s <= 8; s *= 2, ++doublings) {
    const int64_t rounds = (tiles * s + warps - 1) / warps, each = (pieces + s - 1) / s;
    const int64_t cost = 10 * rounds * each + 15 * (rounds - 1) + 12 * doublings;
    if (s == 1 || cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

template <int BITS>
int run(const Params& p, cudaStream_t st) {
  switch (split<BITS>(p)) {
    case 1: return launch<BITS, 1>(p, st);
    case 2: return launch<BITS, 2>(p, st);
    case 4: return launch<BITS, 4>(p, st);
    default: return launch<BITS, 8>(p, st);
  }
}

// From 24 M weights on; with fewer the start of a block of this size is what a call takes (N 6144, K 3072, 4 bits, three
// rows: 8.6 us against 7.5). The other kernel / this one, at 1, 4, 8 rows: 4 bits, N 9216, K 3072 10.1 / 8.6, 10.2 / 9.7,
// 10.9 / 11.4; N 11520, K 4096 13.2 / 12.4, 13.3 / 13.5, 14.3 / 15.5; N 12288, K 4096 15.9 / 12.6, 15.9 / 13.8, 16.1 / 15.6;
// N 20480, K 3840 21.5 / 19.4, 21.8 / 20.6, 22.5 / 22.3; 8 bits, N 8192, K 4096 14.1 / 11.5, 14.1 / 12.7, 14.1 / 14.6; N
// 12288, K 3072 15.5 / 12.3, 15.5 / 13.4, 15.6 / 14.6; N 15360, K 3840 21.1 / 17.7, 21.2 / 18.9, 21.3 / 20.7. Every row costs
// here (it is copied into each block's shared memory and its sums per group are formed there) and almost nothing there, so
// more rows need more weights to read; at 4 bits, three rows, N 10240, K 3840 13.1 / 13.4. A plain read of the 33 MB of the
// 8-bit N 8192, K 4096 takes 6.2 us. The two kernels round differently (weights to bf16 there, not here), so a row's result
// may differ by about 1e-3 with the number of rows beside it; the C header says so.
template <int BITS>
bool pays(const Params& p) {
  const int64_t weights = static_cast<int64_t>(p.N) * p.K;
  return p.M <= (weights >= ((BITS == 4 ? 48ll : 36ll) << 20) ? 8 : BITS / 2) && weights >= (24ll << 20) && p.K <= (1 << 20) &&
         smem_bytes<BITS>(p.M, p.K) <= MAX_SMEM;
}

}  // namespace stream

bool eligible(const mfx_qlinear_args& a) {
  return a.batch == 1 && a.rows <= 16 && (a.epilogue == MFX_EPI_NONE || a.epilogue == MFX_EPI_SILU);
}

int run(const mfx_qlinear_args& a, const void* prepared, size_t codes_bytes, cudaStream_t st) {
  Params p;
  p.x = static_cast<const __nv_bfloat16*>(a.x);
  p.x_row_stride = a.x_row_stride;
  p.M = static_cast<int>(a.rows);
  p.N = static_cast<int>(a.N);
  p.K = static_cast<int>(a.K);
  p.codes = static_cast<const uint32_t*>(prepared);
  p.sb = reinterpret_cast<const uint32_t*>(static_cast<const uint8_t*>(prepared) + codes_bytes);
  p.bias = a.bias;
  p.bias_dtype = a.bias_dtype;
  p.epilogue = a.epilogue;
  p.y = a.y;
  p.y_dtype = a.y_dtype;
  p.y_row_stride = a.y_row_stride;
  if (kernel_bits(a.bits) == 4 ? stream::pays<4>(p) : stream::pays<8>(p))
    return kernel_bits(a.bits) == 4 ? stream::run<4>(p, st) : stream::run<8>(p, st);
  // 16 rows per block while that still gives every SM two blocks, else 8 rows per block (32 rows per block take 100
  // registers and leave two blocks per SM: 10-25 % slower on 9216 to 18432 rows)
  const bool wide = (a.N + 15) / 16 >= 2 * device_sm_count();
  const unsigned blocks = static_cast<unsigned>(wide ? (a.N + 15) / 16 : (a.N + 7) / 8);
  auto kern = kernel_bits(a.bits) == 4 ? (wide ? qmv_kernel<4, 2> : qmv_kernel<4, 1>)
                                       : (wide ? qmv_kernel<8, 2> : qmv_kernel<8, 1>);
  // An ordinary launch, before which everything in the stream has finished: this kernel does not wait for its predecessor.
  // Overlapped, most calls would gain up to half a microsecond and some lose more, by no rule of blocks or bytes that we
  // found. Overlapped / ordinary, us, one after the other: four rows, N 3072, K 4096, 8 bits 8.4 / 7.1, five rows, N 3840, K
  // 12288, 4 bits 20.1 / 17.8, 16 rows, N 9216, K 3072, 4 bits 15.4 / 14.4, two rows, N 3072, K 768, 4 bits 2.56 / 2.45; two
  // rows, N 15360, K 256, 8 bits 4.0 / 4.2, one row, N 3072, K 256, 8 bits 1.84 / 1.93, N 6144, K 3072, 4 bits 6.7 / 7.3.
  kern<<<blocks, THREADS, 0, st>>>(p);
  MFX_CUDA_TRY(cudaGetLastError());
  return MFX_OK;
}

}  // namespace qmv
}  // namespace mfx
