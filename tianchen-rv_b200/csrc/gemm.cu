// Prefill GEMM host side: the unpack ("prepare") kernels that turn plain block_q4_0 /
// block_q8_0 rows into the planar layout the tensor-core kernel consumes, the TMA tensor
// maps, and the launchers.
//
// Planar layout (all regions 256-byte aligned inside the caller's workspace):
//   weights      8-bit [nr][K]           value = nibble - 8, as e4m3 (every integer in [-8, 7] is exact)
//   weight scale fp32 [nr][nbp]          nbp = blocks per row rounded up to 4
//   activations  8-bit [nc][K] twice     an int8 q as two e4m3 planes: q & 15 and q - (q & 15), q = sum of both
//   act. scale   fp32 [nb][ncp]          transposed; ncp = columns rounded up to 4
#include <atomic>
#include <type_traits>
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include "gemm_tc.cuh"
#include "launchers.h"

namespace tcrv {

namespace {

constexpr size_t kAlign = 256;
inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Four bytes u, each standing for the integer u - bias (which e4m3 represents exactly: at most 16 in
// magnitude, or a multiple of 16 up to 128), to four e4m3 bytes.  0x6400 | u is the fp16 number
// 1024 + u, so one exact fp16 subtraction and one conversion serve two values.
template <int kBias>
__device__ __forceinline__ uint32_t e4m3x4_from_u8x4(uint32_t u) {
  const __half2 bias = __half2half2(__ushort_as_half(static_cast<unsigned short>(0x6400 + kBias)));
  uint32_t r = 0;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t h = __byte_perm(u, 0x64646464u, k == 0 ? 0x4140 : 0x4342);
    const __half2 v = __hsub2(*reinterpret_cast<const __half2 *>(&h), bias);
    r |= static_cast<uint32_t>(__nv_cvt_halfraw2_to_fp8x2(static_cast<__half2_raw>(v), __NV_SATFINITE, __NV_E4M3))
         << (16 * k);
  }
  return r;
}

// 32 bytes, a whole sector, in one store (the planes start on 256-byte boundaries).
__device__ __forceinline__ void store_32(int8_t *dst, const uint32_t (&w)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// Stores the 32 weight values of a block (q = its 16 nibble bytes, element j in the low nibble of
// byte j and element j + 16 in the high one, value = nibble - 8).
__device__ __forceinline__ void store_weight_block(int8_t *dst32, const uint32_t (&q)[4]) {
  uint32_t w[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    w[j] = e4m3x4_from_u8x4<8>(q[j] & 0x0f0f0f0fu);
    w[4 + j] = e4m3x4_from_u8x4<8>((q[j] >> 4) & 0x0f0f0f0fu);
  }
  store_32(dst32, w);
}

// Stores 32 int8 activation values q[8] as the two e4m3 planes q & 15 (0..15)
// and q & 0xf0 read as a signed byte (16 * (q >> 4): -128, -112, ..., 112), `plane` bytes apart.
__device__ __forceinline__ void store_act_block(int8_t *dst32, size_t plane, const uint32_t (&q)[8]) {
  uint32_t l[8], h[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    l[j] = e4m3x4_from_u8x4<0>(q[j] & 0x0f0f0f0fu);
    h[j] = e4m3x4_from_u8x4<128>((q[j] & 0xf0f0f0f0u) ^ 0x80808080u);
  }
  store_32(dst32, l);
  store_32(dst32 + plane, h);
}

// A block's scale.  The TMA boxes of the scales cover the rows' (columns') padding, which has to read
// as zero: the last block of a row (the last column) writes it.
__device__ __forceinline__ void store_weight_scale(float *dw, size_t row, uint32_t ib, uint32_t nb, uint32_t nbp,
                                                   uint32_t d) {
  dw[row * nbp + ib] = half_bits_to_float(d);
  if (ib + 1 == nb)
    for (uint32_t p = nb; p < nbp; ++p)
      dw[row * nbp + p] = 0.0f;
}
__device__ __forceinline__ void store_act_scale(float *dxt, size_t col, size_t ib, uint32_t nc, uint32_t ncp,
                                                uint32_t d) {
  dxt[ib * ncp + col] = half_bits_to_float(d);
  if (col + 1 == nc)
    for (uint32_t p = nc; p < ncp; ++p)
      dxt[ib * ncp + p] = 0.0f;
}

// ---------------------------------------------------------------- unpack kernels

// Rows that follow one another without gaps, on a 16-byte boundary: 512 blocks at a time come in
// with 16-byte loads; a thread then takes a pair of blocks (36 bytes: nine whole words, an odd
// stride, so its shared-memory loads are free of conflicts) and writes whole sectors.  Bound by HBM
// (18 B in, 36 B out per block): with the
// activations, 49.0 -> 41.2 us for 32000 x 4096 against one thread per block and byte-wise
// conversion (223 MB: 34 us at the measured copy rate).
constexpr int kUnpackBlocks = 512;
__global__ void __launch_bounds__(256) unpack_q4_0_dense_kernel(const uint8_t *__restrict__ vx, uint32_t nr,
                                                                uint32_t nb, uint32_t nbp, int8_t *__restrict__ w8,
                                                                float *__restrict__ dw) {
  __shared__ __align__(16) uint32_t tile[kUnpackBlocks * kQ4Block / 4];
  pdl_enter();
  const size_t total = static_cast<size_t>(nr) * nb;
  for (size_t first = static_cast<size_t>(blockIdx.x) * kUnpackBlocks; first < total;
       first += static_cast<size_t>(gridDim.x) * kUnpackBlocks) {
    const uint32_t count = static_cast<uint32_t>(total - first < kUnpackBlocks ? total - first : kUnpackBlocks);
    const uint8_t *src = vx + first * kQ4Block;
    const uint32_t bytes = count * kQ4Block;
    for (uint32_t i = threadIdx.x; i < bytes / 16; i += 256)
      reinterpret_cast<uint4 *>(tile)[i] = __ldg(reinterpret_cast<const uint4 *>(src) + i);
    for (uint32_t i = bytes / 16 * 8 + threadIdx.x; i < bytes / 2; i += 256)
      reinterpret_cast<unsigned short *>(tile)[i] = reinterpret_cast<const unsigned short *>(src)[i];
    __syncthreads();
    const uint32_t pair = 2 * threadIdx.x;
    if (pair < count) {
      uint32_t w[9];
#pragma unroll
      for (int j = 0; j < 9; ++j)
        w[j] = tile[9 * threadIdx.x + j];
      const size_t i = first + pair, row = i / nb;
      const uint32_t ib = static_cast<uint32_t>(i - row * nb);
      const uint32_t even[4] = {__funnelshift_r(w[0], w[1], 16), __funnelshift_r(w[1], w[2], 16),
                                __funnelshift_r(w[2], w[3], 16), __funnelshift_r(w[3], w[4], 16)};
      store_weight_block(w8 + i * kQK, even);
      store_weight_scale(dw, row, ib, nb, nbp, w[0] & 0xffffu);
      if (pair + 1 < count) {
        const uint32_t odd[4] = {w[5], w[6], w[7], w[8]};
        store_weight_block(w8 + (i + 1) * kQK, odd);
        const bool next = ib + 1 == nb;
        store_weight_scale(dw, row + next, next ? 0 : ib + 1, nb, nbp, w[4] >> 16);
      }
    }
    __syncthreads();
  }
}

// Any alignment and row stride.  One thread per (row, block): 18 bytes in, 32 values + one scale out.
__global__ void __launch_bounds__(256) unpack_q4_0_kernel(const uint8_t *__restrict__ vx, size_t bx, uint32_t nr,
                                                          uint32_t nb, uint32_t nbp, int8_t *__restrict__ w8,
                                                          float *__restrict__ dw, bool aligned2) {
  pdl_enter();
  const size_t total = static_cast<size_t>(nr) * nb;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const size_t row = i / nb, ib = i - row * nb;
    const uint8_t *blk = vx + row * bx + ib * kQ4Block;
    uint32_t d, q[4];
    if (aligned2) {
      const unsigned short *h = reinterpret_cast<const unsigned short *>(blk);
      d = h[0];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        q[j] = static_cast<uint32_t>(h[1 + 2 * j]) | (static_cast<uint32_t>(h[2 + 2 * j]) << 16);
    } else {
      d = load_u16(blk);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        q[j] = load_u32_bytes(blk + 2 + 4 * j);
    }
    store_weight_block(w8 + i * kQK, q);
    store_weight_scale(dw, row, static_cast<uint32_t>(ib), nb, nbp, d);
  }
}

// Columns on 16-byte boundaries: a CTA takes 8 columns x 32 blocks.  They come in with 16-byte loads; a
// thread then converts one block (a warp: 32 blocks of a column, whole lines of both planes) and the scales
// leave as sectors of 8 columns.  Bound by latency, load to store, at the sizes of a prompt.
constexpr int kUnpackCols = 8, kUnpackColBlocks = 32;
__global__ void __launch_bounds__(256) unpack_q8_0_tiles_kernel(const uint8_t *__restrict__ vy, size_t by, uint32_t nc,
                                                                uint32_t nb, uint32_t ncp, int8_t *__restrict__ x8,
                                                                size_t plane, float *__restrict__ dxt) {
  constexpr uint32_t kColBytes = kUnpackColBlocks * kQ8Block;  // 1088
  __shared__ __align__(16) uint8_t tile[kUnpackCols * kColBytes];
  __shared__ float scales[kUnpackColBlocks][kUnpackCols + 1];
  pdl_enter();
  const uint32_t c0 = blockIdx.y * kUnpackCols, b0 = blockIdx.x * kUnpackColBlocks;
  const uint32_t blocks = min(static_cast<uint32_t>(kUnpackColBlocks), nb - b0);
  const uint32_t bytes = blocks * kQ8Block, pieces = bytes / 16;  // of a column; what is left of it is half words
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, col = c0 + warp;
  if (col < nc) {
    const uint8_t *src = vy + static_cast<size_t>(col) * by + static_cast<size_t>(b0) * kQ8Block;
    uint8_t *dst = tile + warp * kColBytes;
#pragma unroll
    for (uint32_t k = 0; k < (kColBytes / 16 + 31) / 32; ++k)
      if (k * 32 + lane < pieces)
        reinterpret_cast<uint4 *>(dst)[k * 32 + lane] = __ldg(reinterpret_cast<const uint4 *>(src) + k * 32 + lane);
    if (pieces * 8 + lane < bytes / 2)
      reinterpret_cast<unsigned short *>(dst)[pieces * 8 + lane] = reinterpret_cast<const unsigned short *>(src)[pieces * 8 + lane];
    __syncwarp();
    if (lane < blocks) {
      const unsigned short *h = reinterpret_cast<const unsigned short *>(dst + lane * kQ8Block);
      uint32_t q[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        q[j] = static_cast<uint32_t>(h[1 + 2 * j]) | (static_cast<uint32_t>(h[2 + 2 * j]) << 16);
      store_act_block(x8 + (static_cast<size_t>(col) * nb + b0 + lane) * kQK, plane, q);
      scales[lane][warp] = half_bits_to_float(h[0]);
    }
  } else {
    scales[lane][warp] = 0.0f;  // columns' padding (see store_act_scale)
  }
  __syncthreads();
  const uint32_t block = threadIdx.x / kUnpackCols, c = threadIdx.x % kUnpackCols;
  if (block < blocks && c0 + c < ncp)
    dxt[static_cast<size_t>(b0 + block) * ncp + c0 + c] = scales[block][c];
}

// Any alignment.  One thread per (column, block).
__global__ void __launch_bounds__(256) unpack_q8_0_kernel(const uint8_t *__restrict__ vy, size_t by, uint32_t nc,
                                                          uint32_t nb, uint32_t ncp, int8_t *__restrict__ x8,
                                                          size_t plane, float *__restrict__ dxt, bool aligned2) {
  pdl_enter();
  const size_t total = static_cast<size_t>(nc) * nb;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const size_t col = i / nb, ib = i - col * nb;
    const uint8_t *blk = vy + col * by + ib * kQ8Block;
    uint32_t d, q[8];
    if (aligned2) {
      const unsigned short *h = reinterpret_cast<const unsigned short *>(blk);
      d = h[0];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        q[j] = static_cast<uint32_t>(h[1 + 2 * j]) | (static_cast<uint32_t>(h[2 + 2 * j]) << 16);
    } else {
      d = load_u16(blk);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        q[j] = load_u32_bytes(blk + 2 + 4 * j);
    }
    store_act_block(x8 + i * kQK, plane, q);
    store_act_scale(dxt, col, ib, nc, ncp, d);
  }
}

// One thread per (row group, block, row): block_q4_0x16 (16 fp16 scales, then byte 32 + 16*i + r
// = elements i and i+16 of row r as nibbles xor 0x88, i.e. 4-bit two's complement) to the
// same planar form.
__global__ void __launch_bounds__(256) unpack_q4_0x16_kernel(const uint8_t *__restrict__ vx, uint32_t rows, uint32_t nb,
                                                             uint32_t nbp, int8_t *__restrict__ w8,
                                                             float *__restrict__ dw) {
  pdl_enter();
  const size_t total = static_cast<size_t>(rows) * nb;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const uint32_t r = static_cast<uint32_t>(i % 16);
    const size_t gl = i / 16, ib = gl % nb, g = gl / nb;
    const uint8_t *blk = vx + gl * 288;
    uint32_t q[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      q[j] = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        q[j] |= static_cast<uint32_t>(blk[32 + (4 * j + k) * 16 + r]) << (8 * k);
      q[j] ^= 0x88888888u;  // back to offset-binary nibbles
    }
    const size_t row = g * 16 + r;
    store_weight_block(w8 + (row * nb + ib) * kQK, q);
    store_weight_scale(dw, row, static_cast<uint32_t>(ib), nb, nbp, load_u16(blk + 2 * r));
  }
}

// One thread per (column group, block, column): block_q8_0x4 (4 fp16 scales, then byte
// 8 + 4*i + c = element i of column c) to the planar activations.
__global__ void __launch_bounds__(256) unpack_q8_0x4_kernel(const uint8_t *__restrict__ vy, uint32_t cols, uint32_t nb,
                                                            uint32_t ncp, int8_t *__restrict__ x8, size_t plane,
                                                            float *__restrict__ dxt) {
  pdl_enter();
  const size_t total = static_cast<size_t>(cols) * nb;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const uint32_t c = static_cast<uint32_t>(i % 4);
    const size_t yl = i / 4, ib = yl % nb, y = yl / nb;
    const uint8_t *blk = vy + yl * 136;
    uint32_t q[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      q[j] = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        q[j] |= static_cast<uint32_t>(blk[8 + (4 * j + k) * 4 + c]) << (8 * k);
    }
    const size_t col = y * 4 + c;
    store_act_block(x8 + (col * nb + ib) * kQK, plane, q);
    store_act_scale(dxt, col, ib, cols, ncp, load_u16(blk + 2 * c));
  }
}

// ------------------------------------------------------------------- tensor maps

using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int get_encode_fn(EncodeTiledFn *out) {
  static std::atomic<EncodeTiledFn> cached{nullptr};  // host threads may race to fill it with the same value
  if (cached.load() == nullptr) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    TCRV_CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
    if (qres != cudaDriverEntryPointSuccess || fn == nullptr)
      return record_cuda_error(cudaErrorNotSupported, "cuTensorMapEncodeTiled entry point");
    cached = reinterpret_cast<EncodeTiledFn>(fn);
  }
  *out = cached;
  return TCRV_CUDA_OK;
}

int make_map_2d(CUtensorMap *map, CUtensorMapDataType type, size_t elem_bytes, const void *base, uint64_t inner,
                uint64_t outer, uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer,
                CUtensorMapSwizzle swizzle) {
  EncodeTiledFn encode;
  const int st = get_encode_fn(&encode);
  if (st != TCRV_CUDA_OK)
    return st;
  (void)elem_bytes;
  const cuuint64_t dims[2] = {inner, outer};
  const cuuint64_t strides[1] = {row_stride_bytes};
  const cuuint32_t box[2] = {box_inner, box_outer};
  const cuuint32_t elem_strides[2] = {1, 1};
  const CUresult res = encode(map, type, 2, const_cast<void *>(base), dims, strides, box, elem_strides,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (res != CUDA_SUCCESS)
    return record_cuda_error(cudaErrorInvalidValue, "cuTensorMapEncodeTiled");
  return TCRV_CUDA_OK;
}

struct PlanarSizes {
  size_t nb, nbp, ncp, k;
  size_t w8, dw, x8, dxt;  // region sizes (aligned)
  size_t x_plane;          // one activation plane; x8 holds two (low, high)
};

PlanarSizes planar_sizes(size_t n, size_t nr, size_t nc) {
  PlanarSizes p;
  p.nb = n / kQK;
  p.nbp = align_up(p.nb, 4);
  p.ncp = align_up(nc, 4);
  p.k = n;
  p.w8 = align_up(nr * n, kAlign);
  p.dw = align_up(nr * p.nbp * 4, kAlign);
  p.x_plane = align_up(nc * n, kAlign);
  p.x8 = 2 * p.x_plane;
  p.dxt = align_up(p.nb * p.ncp * 4, kAlign);
  return p;
}

inline int blocks_for(size_t items) {
  size_t b = (items + 255) / 256;
  const size_t cap = static_cast<size_t>(sm_count()) * 16;
  return static_cast<int>(b < cap ? (b ? b : 1) : cap);
}

// Which items a launch deals out: 256 x 64 ones (0; their last round is cut into 128 x 64 halves where those
// fill no more than half of the SMs), 128 x 32 (32) or 128 x 16 (16).  Rounds of each kind times what an item
// takes, in hundredths of a 256 x 64 one: with 128 blocks to a row a round takes 33 us whole, 20 in halves, 11.2 and
// 7.4 to 8.3 narrow.  Narrow items win where the others leave SMs without work.  us a call (weights prepared), 256 x
// 64 / 128 x 32 / 128 x 16: 77 x 4096 x 11008 51.1 / 34.0 / 45.2, 40 x 4096 x 4096 22.1 / 15.0 / 11.6, 16 x 32000 x 4096 39.2 / 34.3 / 31.2,
// 33 x 20000 x 1024 14.1 / 16.0 / 14.3, 200 x 4096 x 4096 24.6 / 29.3 / 29.2, 512 x 11008 x 4096 91.7 / 119 / 146.
int narrow_items(size_t nr, size_t nc, size_t ctas) {
  const auto cdiv = [](size_t a, size_t b) { return (a + b - 1) / b; };
  const size_t tiles = cdiv(nr, 256) * cdiv(nc, 64), rem = tiles % ctas;
  const size_t wide = tiles / ctas * 100 + (rem == 0 ? 0 : 2 * rem <= ctas ? 60 : 100);
  const size_t by32 = cdiv(cdiv(nr, 128) * cdiv(nc, 32), ctas) * 34;
  const size_t by16 = cdiv(cdiv(nr, 128) * cdiv(nc, 16), ctas) * 24;
  return by16 < by32 && by16 < wide ? 16 : by32 < wide ? 32 : 0;
}

// One instantiation of the kernel: its tensor maps, its work items, its launch.
template <bool kMulti, bool kRepack, int kNarrow>
int launch_gemm_kernel(const PlanarSizes &p, const uint8_t *weights_planar, const uint8_t *acts_planar, GemmArgs &args,
                       cudaStream_t stream) {
  using Plan = GemmPlan<kNarrow>;
  const int8_t *w8 = reinterpret_cast<const int8_t *>(weights_planar);
  const float *dw = reinterpret_cast<const float *>(weights_planar + p.w8);
  const int8_t *x8 = reinterpret_cast<const int8_t *>(acts_planar);
  const float *dxt = reinterpret_cast<const float *>(acts_planar + p.x8);
  const size_t n = p.k, nr = args.nr, nc = args.nc;

  CUtensorMap map_w, map_x, map_xhi, map_dw, map_dx;
  int st = make_map_2d(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w8, n, nr, n, kGemmStageBlocks * kQK, kGemmTileRows,
                       CU_TENSOR_MAP_SWIZZLE_128B);
  if (st == TCRV_CUDA_OK)
    st = make_map_2d(&map_x, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, x8, n, nc, n, kGemmStageBlocks * kQK, Plan::kBoxCols,
                     CU_TENSOR_MAP_SWIZZLE_128B);
  if (st == TCRV_CUDA_OK)
    st = make_map_2d(&map_xhi, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, x8 + p.x_plane, n, nc, n, kGemmStageBlocks * kQK,
                     Plan::kBoxCols, CU_TENSOR_MAP_SWIZZLE_128B);
  if (st == TCRV_CUDA_OK)
    st = make_map_2d(&map_dw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dw, p.nbp, nr, p.nbp * 4, kGemmStageBlocks,
                     kGemmTileRows, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (st == TCRV_CUDA_OK)
    st = make_map_2d(&map_dx, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, dxt, p.ncp, p.nb, p.ncp * 4, Plan::kBoxCols,
                     kGemmStageBlocks, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (st != TCRV_CUDA_OK)
    return st;

  args.tiles_m = static_cast<uint32_t>((nc + Plan::Full::kCols - 1) / Plan::Full::kCols);
  const uint32_t tiles = static_cast<uint32_t>((nr + Plan::Full::kRows - 1) / Plan::Full::kRows) * args.tiles_m;
  const uint32_t ctas = static_cast<uint32_t>(sm_count());
  const uint32_t rem = tiles % ctas;
  args.full_items = kNarrow == 0 && 2 * rem <= ctas ? tiles - rem : tiles;
  args.items = args.full_items + 2 * (tiles - args.full_items);
  const int grid = static_cast<int>(args.items < ctas ? args.items : ctas);

  constexpr size_t smem = GemmSmem<kMulti, kNarrow>::kBytes;
  static std::atomic<bool> configured[64];
  int dev = 0;
  TCRV_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64)
    return TCRV_CUDA_ERR_UNSUPPORTED;
  const auto kernel = gemm_q4_0_q8_0_tc_kernel<kMulti, kRepack, kNarrow>;
  if (!configured[dev]) {
    // a block that starts with fewer registers than its warps ask for would wait for them for ever
    cudaFuncAttributes attributes;
    TCRV_CUDA_TRY(cudaFuncGetAttributes(&attributes, kernel));
    if (attributes.numRegs * kGemmThreads < kGemmSplitRegs)
      return TCRV_CUDA_ERR_UNSUPPORTED;
    TCRV_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    configured[dev] = true;
  }
  TCRV_CUDA_TRY(launch_pdl(kernel, grid, kGemmThreads, smem, stream, map_w, map_x, map_xhi, map_dw, map_dx, args));
  TCRV_CUDA_TRY(cudaGetLastError());
  return TCRV_CUDA_OK;
}

// `repack`: fold with the scales multiplied first and store token-major (dst[0][col*bs + row]).
int run_gemm(size_t n, float *const *dst, size_t ndst, const uint8_t *weights_planar, const uint8_t *acts_planar,
             size_t nr, size_t nc, size_t bs, cudaStream_t stream, bool repack = false) {
  const PlanarSizes p = planar_sizes(n, nr, nc);
  const bool multi = ndst > 1;
  if (repack && multi)
    return TCRV_CUDA_ERR_UNSUPPORTED;
  GemmArgs args = {};
  for (size_t d = 0; d < ndst; ++d)
    args.dst[d] = dst[d];
  args.ndst = static_cast<uint32_t>(ndst);
  args.bs = bs;
  args.nr = static_cast<uint32_t>(nr);
  args.nc = static_cast<uint32_t>(nc);
  args.nb = static_cast<uint32_t>(p.nb);
  const int st = device_error_words(&args.errors);
  if (st != TCRV_CUDA_OK)
    return st;
  const auto launch = [&](auto narrow) {
    constexpr int kNarrow = decltype(narrow)::value;
    return repack ? launch_gemm_kernel<false, true, kNarrow>(p, weights_planar, acts_planar, args, stream)
                  : launch_gemm_kernel<false, false, kNarrow>(p, weights_planar, acts_planar, args, stream);
  };
  if (multi)
    return launch_gemm_kernel<true, false, 0>(p, weights_planar, acts_planar, args, stream);
  switch (narrow_items(nr, nc, static_cast<size_t>(sm_count()))) {
    case 16: return launch(std::integral_constant<int, 16>());
    case 32: return launch(std::integral_constant<int, 32>());
    default: return launch(std::integral_constant<int, 0>());
  }
}

}  // namespace

size_t gemm_weights_bytes(size_t n, size_t nr) {
  const PlanarSizes p = planar_sizes(n, nr, 0);
  return p.w8 + p.dw;
}

size_t gemm_acts_bytes(size_t n, size_t nc) {
  const PlanarSizes p = planar_sizes(n, 0, nc);
  return p.x8 + p.dxt;
}

int launch_gemm_prepare_weights_q4_0(size_t n, const uint8_t *vx, size_t bx, size_t nr, uint8_t *prepared,
                                     cudaStream_t stream) {
  const PlanarSizes p = planar_sizes(n, nr, 0);
  if (nr == 0 || p.nb == 0)
    return TCRV_CUDA_OK;
  const bool aligned2 = (reinterpret_cast<uintptr_t>(vx) % 2 == 0) && (bx % 2 == 0);
  int8_t *w8 = reinterpret_cast<int8_t *>(prepared);
  float *dw = reinterpret_cast<float *>(prepared + p.w8);
  const uint32_t rows = static_cast<uint32_t>(nr), nb = static_cast<uint32_t>(p.nb), nbp = static_cast<uint32_t>(p.nbp);
  if ((bx == p.nb * kQ4Block || nr == 1) && reinterpret_cast<uintptr_t>(vx) % 16 == 0)
    TCRV_CUDA_TRY(launch_pdl(unpack_q4_0_dense_kernel, blocks_for((nr * p.nb + 1) / 2), 256, 0, stream, vx, rows, nb, nbp,
                             w8, dw));
  else
    TCRV_CUDA_TRY(launch_pdl(unpack_q4_0_kernel, blocks_for(nr * p.nb), 256, 0, stream, vx, bx, rows, nb, nbp, w8, dw,
                             aligned2));
  TCRV_CUDA_TRY(cudaGetLastError());
  return TCRV_CUDA_OK;
}

int launch_gemm_prepare_acts_q8_0(size_t n, const uint8_t *vy, size_t by, size_t nc, uint8_t *prepared,
                                  cudaStream_t stream) {
  const PlanarSizes p = planar_sizes(n, 0, nc);
  if (nc == 0 || p.nb == 0)
    return TCRV_CUDA_OK;
  const size_t col_tiles = (nc + kUnpackCols - 1) / kUnpackCols;
  if (reinterpret_cast<uintptr_t>(vy) % 16 == 0 && (by % 16 == 0 || nc == 1) && col_tiles <= 65535) {
    const dim3 grid(static_cast<unsigned>((p.nb + kUnpackColBlocks - 1) / kUnpackColBlocks), static_cast<unsigned>(col_tiles));
    TCRV_CUDA_TRY(launch_pdl(unpack_q8_0_tiles_kernel, grid, 256, 0, stream, vy, by, static_cast<uint32_t>(nc),
                             static_cast<uint32_t>(p.nb), static_cast<uint32_t>(p.ncp), reinterpret_cast<int8_t *>(prepared),
                             p.x_plane, reinterpret_cast<float *>(prepared + p.x8)));
    return TCRV_CUDA_OK;
  }
  const bool aligned2 = (reinterpret_cast<uintptr_t>(vy) % 2 == 0) && (by % 2 == 0);
  TCRV_CUDA_TRY(launch_pdl(unpack_q8_0_kernel, blocks_for(nc * p.nb), 256, 0, stream, vy, by, static_cast<uint32_t>(nc),
                           static_cast<uint32_t>(p.nb), static_cast<uint32_t>(p.ncp),
                           reinterpret_cast<int8_t *>(prepared), p.x_plane,
                           reinterpret_cast<float *>(prepared + p.x8), aligned2));
  TCRV_CUDA_TRY(cudaGetLastError());
  return TCRV_CUDA_OK;
}

int launch_gemm_prepared(size_t n, float *s, const uint8_t *weights_planar, const uint8_t *acts_planar, size_t nr,
                         size_t nc, size_t bs, cudaStream_t stream) {
  if (nr == 0 || nc == 0)
    return TCRV_CUDA_OK;
  return run_gemm(n, &s, 1, weights_planar, acts_planar, nr, nc, bs, stream);
}

int launch_gemm_prepared_multi(size_t n, float *const *dst, size_t ndst, const uint8_t *weights_planar,
                               const uint8_t *acts_planar, size_t nr, size_t nc, size_t bs, cudaStream_t stream) {
  if (ndst == 0 || ndst > static_cast<size_t>(kGemmMaxDst))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nr == 0 || nc == 0)
    return TCRV_CUDA_OK;
  return run_gemm(n, dst, ndst, weights_planar, acts_planar, nr, nc, bs, stream);
}

// ------------------------------------------------------------ interleaved-layout consumer
//
// tcrv_rvv.repack_gemm_q4_0_q8_0: weights in block_q4_0x16 groups (`wrows` weight rows),
// activations in block_q8_0x4 groups (`tokens` columns); both are unpacked into the planar
// form and contracted by the same tensor-core kernel (kRepack instantiation).

int launch_repack_gemm_prepare_weights_q4_0x16(size_t n, const uint8_t *vx, size_t wrows, uint8_t *prepared,
                                               cudaStream_t stream) {
  const PlanarSizes p = planar_sizes(n, wrows, 0);
  if (wrows == 0 || p.nb == 0)
    return TCRV_CUDA_OK;
  TCRV_CUDA_TRY(launch_pdl(unpack_q4_0x16_kernel, blocks_for(wrows * p.nb), 256, 0, stream, vx,
                           static_cast<uint32_t>(wrows), static_cast<uint32_t>(p.nb), static_cast<uint32_t>(p.nbp),
                           reinterpret_cast<int8_t *>(prepared), reinterpret_cast<float *>(prepared + p.w8)));
  TCRV_CUDA_TRY(cudaGetLastError());
  return TCRV_CUDA_OK;
}

int launch_repack_gemm_prepared(size_t n, float *s, const uint8_t *weights_planar, const uint8_t *vy, size_t tokens,
                                size_t wrows, size_t bs, uint8_t *acts_planar, cudaStream_t stream) {
  const PlanarSizes p = planar_sizes(n, 0, tokens);
  if (tokens == 0 || wrows == 0 || p.nb == 0)
    return TCRV_CUDA_OK;
  TCRV_CUDA_TRY(launch_pdl(unpack_q8_0x4_kernel, blocks_for(tokens * p.nb), 256, 0, stream, vy,
                           static_cast<uint32_t>(tokens), static_cast<uint32_t>(p.nb), static_cast<uint32_t>(p.ncp),
                           reinterpret_cast<int8_t *>(acts_planar), p.x_plane,
                           reinterpret_cast<float *>(acts_planar + p.x8)));
  TCRV_CUDA_TRY(cudaGetLastError());
  return run_gemm(n, &s, 1, weights_planar, acts_planar, wrows, tokens, bs, stream, /*repack=*/true);
}

// ------------------------------------------------------------ allocation-free variant
//
// Scratch for callers that must not allocate device memory: the planar operand copies live
// in this fixed array instead of a caller-provided workspace.  The array is part of the
// library image, so every GPU that loads the library sets aside kStaticScratchBytes for it
// until the process exits.  In host code the array's name only stands for the symbol; the
// device address has to be asked for (once per device, with that device current).
constexpr size_t kStaticScratchBytes = TCRV_CUDA_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) uint8_t g_static_scratch[kStaticScratchBytes];

int launch_gemm_static_scratch(size_t n, float *s, const uint8_t *vx, size_t bx, const uint8_t *vy, size_t by,
                               size_t nr, size_t nc, size_t bs, cudaStream_t stream) {
  if (nr == 0 || nc == 0 || n == 0)
    return TCRV_CUDA_OK;
  const size_t wbytes = gemm_weights_bytes(n, nr), abytes = gemm_acts_bytes(n, nc);
  if (wbytes + abytes > kStaticScratchBytes)
    return TCRV_CUDA_ERR_WORKSPACE;
  static std::atomic<uint8_t *> base[64];
  int dev = 0;
  TCRV_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64)
    return TCRV_CUDA_ERR_UNSUPPORTED;
  if (base[dev] == nullptr) {
    void *addr = nullptr;
    TCRV_CUDA_TRY(cudaGetSymbolAddress(&addr, g_static_scratch));
    base[dev] = static_cast<uint8_t *>(addr);
  }
  uint8_t *weights = base[dev], *acts = base[dev] + wbytes;
  int st = launch_gemm_prepare_weights_q4_0(n, vx, bx, nr, weights, stream);
  if (st == TCRV_CUDA_OK)
    st = launch_gemm_prepare_acts_q8_0(n, vy, by, nc, acts, stream);
  if (st == TCRV_CUDA_OK)
    st = run_gemm(n, &s, 1, weights, acts, nr, nc, bs, stream);
  return st;
}

}  // namespace tcrv
