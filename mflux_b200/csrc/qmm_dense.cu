// Quantized linear layer for many activation rows, in two launches: decode_kernel writes the weight once as bf16 to
// scratch, dense_kernel is a bf16 contraction over it. The one-launch kernel (qmm.cu) decodes every weight tile again
// for every 256 activation rows; beside the tensor cores that costs shared-memory bandwidth (1330 cycles of it per
// 1024 cycles of products) and, at the power limit where long steps run, energy. The decoded values are the same
// bf16 values the one-launch kernel feeds its tensor cores, and the products run in the same order of K.
// Measured, looped at the power limit, decode included, one launch -> two: 8 bits, M 8426, N 3840, K 10240: 591 -> 545 us;
// 4 bits, M 14290, N 3072, K 3072, gated residual: 278 -> 253 us; M 73728, N 9216, K 3072: 3194 -> 3110 us (1342 TFLOP/s).
//
// dense_kernel: persistent, one CTA pair (cluster of 2, tcgen05 cta_group::2) per 256 x 256 output tile. Per CTA:
//   warp 0      TMA producer: the 128 activation rows and 128 weight rows of its half of the tile, 64 k per stage,
//               as 128-byte-swizzled slabs counted on the leader's barrier. Six stages of 64 k beat three of 128 k by
//               1-2 % (a freed slab is refilled half a stage earlier)
//   warp 1      allocates TMEM; in the leader issues tcgen05.mma.cta_group::2 (M 256, N 256, K 16)
//   warps 4-11  epilogue, two warps per 32 rows, overlapped with the main loop of the next tile (two accumulators)
// All waits are bounded.
#include <cuda_bf16.h>

#include "host_util.cuh"
#include "launch.cuh"
#include "ptx.cuh"
#include "qmm_common.cuh"
#include "qmm_dense.cuh"
#include "qmm_epilogue.cuh"

namespace mfx {
namespace qmmd {

constexpr int BM = 128;                   // activation rows per CTA
constexpr int BN = 256;                   // output columns per pair tile; each CTA loads 128 weight rows
constexpr int BK = 64;                    // k per stage: one 128-byte swizzle row
constexpr int ST = 6;                     // stages
constexpr int SLAB = 128 * BK * 2;        // 16 KiB
constexpr int STAGE = 2 * SLAB;           // activations and weights
constexpr int EPI_WARPS = 8;
constexpr int FIRST_EPI_WARP = 4;
constexpr int NUM_THREADS = (FIRST_EPI_WARP + EPI_WARPS) * 32;
constexpr uint32_t TMEM_COLS = 512;
constexpr int OFF_VEC = ST * STAGE;       // bias[2][256] + gate[2][256] floats
constexpr int OFF_BAR = OFF_VEC + 4 * BN * 4;
constexpr int NUM_BARS = 2 * ST + 4;
constexpr int OFF_TMEM = OFF_BAR + NUM_BARS * 8;
constexpr int DYN_BYTES = OFF_TMEM + 16 + 1024;   // slack for manual 1024-byte alignment
static_assert(DYN_BYTES <= 227 * 1024, "shared memory of the dense kernel");

// Weights of one band of n-tiles, which stay in L2 while every activation tile passes over them. 48 MB against 32:
// M 14290, N 3072, K 12288: 950 -> 898 us (two passes over the activations instead of three); 64 MB and one band lose
// 2 and 14 % at M 73728, N 12288, K 3072, where the weights no longer stay.
constexpr int64_t BAND_BYTES = 48ll << 20;

struct Params {
  int rows, batch, N, K;
  int tiles_m_per_sample, tiles_m, tiles_n, total_tiles;
  int band_n;          // n-tiles per band of the tile order
  int ext_r;           // rank of the low-rank term, rounded up to 16 (0: none)
  const void* bias;
  int bias_dtype;
  const void* gate;
  int gate_dtype;
  int64_t gate_batch_stride;
  const void* residual;
  int64_t res_row_stride, res_batch_stride;
  void* y;
  int64_t y_row_stride, y_batch_stride;
  bool wide;           // 32-byte aligned output and residual rows
};

// Inside a band of n-tiles the n-tile index runs fastest.
__device__ __forceinline__ void tile_coords(const Params& p, int tile, int& tm, int& tn) {
  const int per_band = p.tiles_m * p.band_n;
  const int band = tile / per_band;
  const int r = tile - band * per_band;
  const int n_first = band * p.band_n;
  const int width = min(p.band_n, p.tiles_n - n_first);
  tm = r / width;
  tn = n_first + r - tm * width;
}

// EXT: after the K / 64 slabs of a tile, the slabs of the low-rank term (activations t, weights lora_b).
template <typename OUT, int EPI, bool EXT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NUM_THREADS, 1)
dense_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w,
             const __grid_constant__ CUtensorMap tmap_t, const __grid_constant__ CUtensorMap tmap_lb, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  float* vec_s = reinterpret_cast<float*>(smem_gen + OFF_VEC);
  const uint32_t bar0 = smem_base + OFF_BAR;
  auto full = [&](int s) { return bar0 + 8u * s; };                    // leader: the tiles of both CTAs landed
  auto empty = [&](int s) { return bar0 + 8u * (ST + s); };            // local: the stage's products are done
  auto acc_full = [&](int s) { return bar0 + 8u * (2 * ST + s); };     // local
  auto acc_empty = [&](int s) { return bar0 + 8u * (2 * ST + 2 + s); };  // leader
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_gen + OFF_TMEM);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_st = p.K / BK;
  const int num_ext = EXT ? (p.ext_r + BK - 1) / BK : 0;
  const int num_all = num_st + num_ext;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);    // the leader's expect_tx covers both CTAs' tiles
      mbar_init(empty(s), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(acc_full(s), 1);
      mbar_init(acc_empty(s), 2 * EPI_WARPS);
    }
    fence_mbar_init();
    tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_w);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_base + OFF_TMEM, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anyone signals across the pair
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  wait_for_predecessor();
  allow_successor();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    int st = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int tile = pair; tile < p.total_tiles && ok; tile += num_pairs) {
      int tm, tn;
      tile_coords(p, tile, tm, tn);
      const int b = tm / p.tiles_m_per_sample;
      const int r0 = (tm % p.tiles_m_per_sample) * (2 * BM) + static_cast<int>(rank) * BM;
      const int n0 = tn * BN + static_cast<int>(rank) * (BN / 2);
      for (int s = 0; s < num_all; ++s) {
        if (!mbar_wait(empty(st), ph ^ 1u, DEV_TIMEOUT_TMA_EMPTY)) {
          ok = false;
          break;
        }
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(full(st), 2 * STAGE);
          const uint32_t dst = smem_base + st * STAGE;
          const bool ext = EXT && s >= num_st;
          const int k0 = (ext ? s - num_st : s) * BK;
          tma_load_3d_pair(dst, ext ? &tmap_t : &tmap_x, full(st), k0, r0, b);
          tma_load_3d_pair(dst + SLAB, ext ? &tmap_lb : &tmap_w, full(st), k0, n0, 0);
        }
        __syncwarp();
        if (++st == ST) {
          st = 0;
          ph ^= 1u;
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader CTA only)
    if (rank == 0) {
      constexpr uint32_t IDESC = make_idesc(FMT_BF16, FMT_BF16, 2 * BM, BN);
      const uint64_t desc0 = smem_desc_sw128(smem_base);
      int st = 0;
      uint32_t ph = 0;
      bool ok = true;
      int it = 0;
      for (int tile = pair; tile < p.total_tiles && ok; tile += num_pairs, ++it) {
        const int a = it & 1;
        if (!mbar_wait(acc_empty(a), ((it >> 1) & 1) ^ 1u, DEV_TIMEOUT_ACC_EMPTY)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + a * BN;
        for (int s = 0; s < num_all; ++s) {
          if (!mbar_wait(full(st), ph, DEV_TIMEOUT_TMA_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          if (elect_one()) {
            const uint64_t d = desc0 + (st * STAGE >> 4);
#pragma unroll
            for (int k4 = 0; k4 < BK / 16; ++k4) {
              // +32 bytes per 16-element K step inside the 128-byte swizzle row; past the rank the low-rank slabs hold
              // zeros, which need no product
              if (EXT && s >= num_st && (s - num_st) * BK + 16 * k4 >= p.ext_r) continue;
              umma_f16_ss_pair(d_tmem, d + 2 * k4, d + (SLAB >> 4) + 2 * k4, IDESC, (s | k4) != 0 ? 1u : 0u);
            }
            umma_commit_pair(empty(st));
            if (s == num_all - 1) umma_commit_pair(acc_full(a));
          }
          __syncwarp();
          if (++st == ST) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
    }
  } else if (warp >= FIRST_EPI_WARP) {
    // ------------------------------------------------------------ epilogue
    const int q = warp & 3;                                 // TMEM lane quarter this warp may read
    const int half = (warp - FIRST_EPI_WARP) >> 2;          // which 128 of the tile's columns
    const int et = threadIdx.x - FIRST_EPI_WARP * 32;       // 0..255
    const int row = q * 32 + lane;
    int it = 0;
    for (int tile = pair; tile < p.total_tiles; tile += num_pairs, ++it) {
      const int a = it & 1;
      int tm, tn;
      tile_coords(p, tile, tm, tn);
      const int b = tm / p.tiles_m_per_sample;
      const int r = (tm % p.tiles_m_per_sample) * (2 * BM) + static_cast<int>(rank) * BM + row;
      const int n0 = tn * BN;
      float* bias_s = vec_s + a * BN;
      float* gate_s = vec_s + 2 * BN + a * BN;
      const int n = n0 + et;
      bias_s[et] = (p.bias != nullptr && n < p.N) ? load_as_float(p.bias, p.bias_dtype, n) : 0.f;
      if (EPI == MFX_EPI_GATE_RESIDUAL)
        gate_s[et] = (n < p.N) ? load_as_float(p.gate, p.gate_dtype, b * p.gate_batch_stride + n) : 0.f;
      named_bar_sync(1, EPI_WARPS * 32);
      const bool row_ok = r < p.rows;
      // SwiGLU writes one value per (gate, up) column pair: output column n/2
      OUT* yrow = static_cast<OUT*>(p.y) + b * p.y_batch_stride + static_cast<int64_t>(r) * p.y_row_stride +
                  (EPI == MFX_EPI_SWIGLU ? n0 / 2 : n0);
      const int c0 = half * (BN / 2), c1 = c0 + BN / 2;
      const OUT* rrow = nullptr;
      if (EPI == MFX_EPI_GATE_RESIDUAL) {
        // rows past the end point at the sample's first row: no address of theirs leaves the buffer, read or not
        rrow = static_cast<const OUT*>(p.residual) + b * p.res_batch_stride +
               static_cast<int64_t>(row_ok ? r : 0) * p.res_row_stride + n0;
        if (row_ok && p.K <= qmm::PREFETCH_K) qmm::prefetch_row(rrow, c0, c1, p.N - n0);
      }
      if (!mbar_wait_sleep(acc_full(a), (it >> 1) & 1, DEV_TIMEOUT_ACC_FULL)) break;
      tc_fence_after();
      const uint32_t t_addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + a * BN;
      qmm::write_row<OUT, EPI, true>(t_addr, c0, c1, p.N - n0, row_ok, p.wide, yrow, rrow, bias_s, gate_s);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_leader(acc_empty(a));
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer may still be reading this CTA's shared/tensor memory until here
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

MFX_DEFINE_STATUS_READER(read_status)

// Prepared codes -> bf16 [N][K], HBM-bound. A lane decodes 16 neighbouring values (one 32-byte store, a warp 1 KiB in
// a row), a warp one weight row, the 8 warps of a block 8 neighbouring rows, which share the 32-byte sectors of the
// transposed (scale, bias) pairs. gridDim.y cuts K into slices of DEC_ITERS * 512 values, all loads of which a thread
// issues before it decodes.
constexpr int DEC_ITERS = 3;
template <int BITS>
__global__ void __launch_bounds__(256) decode_kernel(const uint8_t* __restrict__ codes, const uint32_t* __restrict__ sb,
                                                     int N, int K, __nv_bfloat16* __restrict__ out) {
  allow_successor();
  const int n = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (n >= N) return;
  const int kb = blockIdx.y * (DEC_ITERS * 512) + (threadIdx.x & 31) * 16;
  const int64_t row = static_cast<int64_t>(n) * K;
  uint32_t w[DEC_ITERS][BITS / 2];
  uint32_t pr[DEC_ITERS];
#pragma unroll
  for (int i = 0; i < DEC_ITERS; ++i) {
    const int k = kb + i * 512;
    if (k < K) {
      const uint8_t* src = codes + (row + k) * BITS / 8;
      if constexpr (BITS == 4) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(src));
        w[i][0] = v.x; w[i][1] = v.y;
      } else {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
        w[i][0] = v.x; w[i][1] = v.y; w[i][2] = v.z; w[i][3] = v.w;
      }
      pr[i] = __ldg(sb + static_cast<int64_t>(k >> 6) * N + n);
    }
  }
#pragma unroll
  for (int i = 0; i < DEC_ITERS; ++i) {
    const int k = kb + i * 512;
    if (k < K) {
      uint32_t o[8];
      if constexpr (BITS == 4) {
        const uint32_t s2 = __byte_perm(pr[i], pr[i], 0x1010), b2 = __byte_perm(pr[i], pr[i], 0x3232);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint4 d = qmm::dequant_w4(w[i][j], s2, b2);
          o[4 * j] = d.x; o[4 * j + 1] = d.y; o[4 * j + 2] = d.z; o[4 * j + 3] = d.w;
        }
      } else {
        uint64_t sc2, bi2;
        asm("mov.b64 %0, {%1, %1};" : "=l"(sc2) : "r"(pr[i] << 16));
        asm("mov.b64 %0, {%1, %1};" : "=l"(bi2) : "r"(pr[i] & 0xFFFF0000u));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint2 d = qmm::dequant_w8_f32(w[i][j], sc2, bi2);
          o[2 * j] = d.x; o[2 * j + 1] = d.y;
        }
      }
      qmm::st_global_32(out + row + k, o);   // scratch is 256-byte aligned, k a multiple of 16, K of 64
    }
  }
}

template <typename OUT, int EPI, bool EXT>
int launch(const CUtensorMap& tx, const CUtensorMap& tw, const CUtensorMap& tt, const CUtensorMap& tlb, Params p,
           int grid, cudaStream_t st) {
  p.wide = qmm::wide_rows<OUT, EPI>(p.y, p.y_row_stride, p.y_batch_stride, p.residual, p.res_row_stride,
                                    p.res_batch_stride);
  auto kern = dense_kernel<OUT, EPI, EXT>;
  static SmemConfigured configured;  // one record per instantiation of the kernel
  if (int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), DYN_BYTES, configured)) return rc;
  MFX_CUDA_TRY(launch_overlapped(kern, grid, NUM_THREADS, DYN_BYTES, st, tx, tw, tt, tlb, p));
  return MFX_OK;
}

template <typename OUT, bool EXT>
int launch_epi(int epilogue, const CUtensorMap& tx, const CUtensorMap& tw, const CUtensorMap& tt,
               const CUtensorMap& tlb, const Params& p, int grid, cudaStream_t st) {
  switch (epilogue) {
    case MFX_EPI_GELU_ERF: return launch<OUT, MFX_EPI_GELU_ERF, EXT>(tx, tw, tt, tlb, p, grid, st);
    case MFX_EPI_GELU_TANH: return launch<OUT, MFX_EPI_GELU_TANH, EXT>(tx, tw, tt, tlb, p, grid, st);
    case MFX_EPI_GATE_RESIDUAL: return launch<OUT, MFX_EPI_GATE_RESIDUAL, EXT>(tx, tw, tt, tlb, p, grid, st);
    case MFX_EPI_SILU: return launch<OUT, MFX_EPI_SILU, EXT>(tx, tw, tt, tlb, p, grid, st);
    case MFX_EPI_SWIGLU: return launch<OUT, MFX_EPI_SWIGLU, EXT>(tx, tw, tt, tlb, p, grid, st);
    default: return launch<OUT, MFX_EPI_NONE, EXT>(tx, tw, tt, tlb, p, grid, st);
  }
}

// Bands of weight rows of `row_bytes` bytes that stay in L2 one at a time: the passes over the activations.
static int64_t num_bands(int64_t N, int64_t row_bytes, int64_t limit) {
  return ((N + BN - 1) / BN * BN * row_bytes + limit - 1) / limit;
}

// Where the two launches win: their cost against the best the one-launch kernel can do with its tile widths
// (one_launch_cost), both in percent of a wave of that kernel's 256-column tiles, so that a part-filled last wave counts
// for either side. A wave here takes 83 % of it for 8 bits and 93 % for 4 (95 % where the bf16 weight is past 32 MB); the
// decode moves 2.6 (4 bits) or 3.1 bytes of HBM traffic per weight, which is 0.0065 of a wave per output column; the second
// launch costs 2.5 us, a wave 8 ns per k. Two passes over the activations more than the packed weight needs, or one that
// feeds few output columns, cost 4-bit layers more than all that gains (N 3072, K 12288: 9 % at 4608 rows, 5 % at 8426).
// Measured, looped at the power limit, one launch / two, us. 8 bits: M 2304, N 12288, K 3072 161 / 156, 4608 317 / 285;
// M 2816, N 3840, K 10240 (165 tiles, 2.2 waves) 208 / 224, 3328 (195 tiles) 252 / 239; M 3328, N 3072, K 3072 61.3 /
// 63.9, 4096 75.7 / 70.9. 4 bits: M 4608, N 3072, K 3072 71.2 / 75.5, 8192 135.5 / 132.7, 18432 282 / 269; M 8192, N
// 9216, K 3072 364 / 362, 18432 818 / 791. Below the limit the one-launch kernel gains more from the higher clock (4 bits,
// M 8426, N 3072, K 3072: 125 / 135), so a predicted gain of less than 2.5 % does not count.
size_t scratch_bytes(int64_t m_tiles, int64_t N, int64_t K, int bits, int64_t one_launch_cost) {
  const int kb = kernel_bits(bits);
  const int64_t extra = num_bands(N, 2 * K, BAND_BYTES) - num_bands(N, K * kb / 8 + K / 16, 32ll << 20);
  if (N < 8192 * extra || (kb == 4 && extra > 1)) return 0;
  // (too little work to judge a cost in waves of the main loop by)
  if (2.0 * 256.0 * static_cast<double>(m_tiles) * static_cast<double>(N) * static_cast<double>(K) < 5e10) return 0;
  const int64_t pairs = device_sm_count() / 2;
  const int64_t waves = (m_tiles * ((N + BN - 1) / BN) + pairs - 1) / pairs;
  const int64_t wave = kb == 8 ? 83 : dense_bytes(N, K) <= (32u << 20) ? 93 : 95;
  const int64_t cost = waves * wave + N * 13 / 2000 + 31000 / K;
  return cost * 40 <= one_launch_cost * 39 ? dense_bytes(N, K) : 0;
}

int run(const mfx_qlinear_args& a, const void* prepared, size_t codes_bytes, void* scratch, cudaStream_t st) {
  const int kb = kernel_bits(a.bits);
  const uint8_t* codes = static_cast<const uint8_t*>(prepared);
  const uint32_t* sb = reinterpret_cast<const uint32_t*>(codes + codes_bytes);
  const int N = static_cast<int>(a.N), K = static_cast<int>(a.K);
  const dim3 dgrid(static_cast<unsigned>((N + 7) / 8),
                   static_cast<unsigned>((K + DEC_ITERS * 512 - 1) / (DEC_ITERS * 512)));
  if (dgrid.y > 65535) return MFX_ERR_TOO_LARGE;
  __nv_bfloat16* w = static_cast<__nv_bfloat16*>(scratch);
  // An ordinary launch, by measurement (8 bits, M 4096, N 12288, K 3072: 252.1 us, overlapped 255.0, both kernels ordinary
  // 252.5; M 73728, N 9216, 4 bits: 3018, 3027, 3032): the decoder does not wait for its predecessor.
  if (kb == 4) decode_kernel<4><<<dgrid, 256, 0, st>>>(codes, sb, N, K, w);
  else decode_kernel<8><<<dgrid, 256, 0, st>>>(codes, sb, N, K, w);
  MFX_CUDA_TRY(cudaGetLastError());

  CUtensorMap tx, tw, tt, tlb;
  const uint32_t box[3] = {BK, 128, 1};
  // [batch][rows][cols] bf16 with a dense last dim; a single sample may carry a zero batch stride, the tensor map
  // wants a positive one
  auto rows_map = [&](CUtensorMap* m, const void* ptr, int64_t cols, int64_t rows, int64_t batch, int64_t row_stride,
                      int64_t batch_stride) {
    const uint64_t dims[3] = {static_cast<uint64_t>(cols), static_cast<uint64_t>(rows), static_cast<uint64_t>(batch)};
    const uint64_t strides[2] = {static_cast<uint64_t>(row_stride) * 2,
                                 static_cast<uint64_t>(batch > 1 ? batch_stride : row_stride * rows) * 2};
    return encode_tmap(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  };
  if (int rc = rows_map(&tx, a.x, a.K, a.rows, a.batch, a.x_row_stride, a.x_batch_stride)) return rc;
  if (int rc = rows_map(&tw, w, a.K, a.N, 1, a.K, 0)) return rc;
  const bool low_rank = a.lora_r > 0;
  if (low_rank) {
    if (int rc = rows_map(&tt, a.lora_t, a.lora_ld, a.rows, a.batch, a.lora_t_row_stride, a.lora_t_batch_stride))
      return rc;
    if (int rc = rows_map(&tlb, a.lora_b, a.lora_ld, a.N, 1, a.lora_ld, 0)) return rc;
  } else {
    tt = tx;   // never read
    tlb = tw;
  }
  Params p;
  p.rows = static_cast<int>(a.rows);
  p.batch = static_cast<int>(a.batch);
  p.N = N;
  p.K = K;
  p.tiles_m_per_sample = static_cast<int>((a.rows + 2 * BM - 1) / (2 * BM));
  const int64_t tiles_m = static_cast<int64_t>(p.tiles_m_per_sample) * p.batch;
  p.tiles_n = (N + BN - 1) / BN;
  if (tiles_m * p.tiles_n > (1ll << 30)) return MFX_ERR_TOO_LARGE;
  p.tiles_m = static_cast<int>(tiles_m);
  p.total_tiles = p.tiles_m * p.tiles_n;
  const int64_t bands = num_bands(N, 2 * a.K, BAND_BYTES);
  p.band_n = static_cast<int>((p.tiles_n + bands - 1) / bands);
  if (p.band_n < 1) p.band_n = 1;
  p.ext_r = low_rank ? static_cast<int>((a.lora_r + 15) / 16 * 16) : 0;
  p.bias = a.bias;
  p.bias_dtype = a.bias_dtype;
  p.gate = a.gate;
  p.gate_dtype = a.gate_dtype;
  p.gate_batch_stride = a.gate_batch_stride;
  p.residual = a.residual;
  p.res_row_stride = a.res_row_stride;
  p.res_batch_stride = a.res_batch_stride;
  p.y = a.y;
  p.y_row_stride = a.y_row_stride;
  p.y_batch_stride = a.y_batch_stride;
  const int pairs = device_sm_count() / 2;
  const int grid = 2 * (p.total_tiles < pairs ? p.total_tiles : pairs);
  if (a.y_dtype == MFX_F32)
    return low_rank ? launch_epi<float, true>(a.epilogue, tx, tw, tt, tlb, p, grid, st)
                    : launch_epi<float, false>(a.epilogue, tx, tw, tt, tlb, p, grid, st);
  return low_rank ? launch_epi<__nv_bfloat16, true>(a.epilogue, tx, tw, tt, tlb, p, grid, st)
                  : launch_epi<__nv_bfloat16, false>(a.epilogue, tx, tw, tt, tlb, p, grid, st);
}

}  // namespace qmmd
}  // namespace mfx
