// Block dots of the sibling ggml formats the reference also compiles: Q4_1 x Q8_1, Q5_0 x Q8_0
// and Q5_1 x Q8_1.  The launchers choose between two streaming kernels, gemv_any.cuh (a table of block
// terms per warp) and strict_stream.cuh (one per CTA), and the general kernel below: one warp per
// (weight row, activation column); every lane computes one block of a group of 32 (byte-granular
// loads: no alignment assumptions), then the 32 terms are folded one after another.  All fold in
// ascending block order, so the result is the sequential fold bit for bit.
//   Q5_0:        sumf = fma(d_x*d_y, (float)sumi, sumf)
//   Q4_1, Q5_1:  sumf = sumf + fma(d_x*d_y, (float)sumi, m_x*s_y)
// (the contraction one C expression gets; lib/Conversion/RVV/RVVToEmitCBlockQuantLinear.cpp:
// 6817-7263, 472-915, 916-1391).
#include "gemv_any.cuh"
#include "launchers.h"
#include "strict_stream.cuh"
#include "tcrv_common.cuh"

namespace tcrv {

namespace {

template <int kFormat>
using Sibling = StrictFormat<kFormat>;

// The same from block pointers of any alignment (byte-granular loads).
template <int kFormat>
__device__ __forceinline__ int sibling_sumi(const uint8_t *xb, const uint8_t *yb) {
  using F = Sibling<kFormat>;
  uint32_t qh = 0;
  if constexpr (F::kQh != 0)
    qh = load_u16(xb + F::kQh) | (load_u16(xb + F::kQh + 2) << 16);
  uint32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0}, y[8];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    q[w] = load_u32_bytes(xb + F::kWq + 4 * w);
    y[w] = load_u32_bytes(yb + F::kAq + 4 * w);
    y[4 + w] = load_u32_bytes(yb + F::kAq + 16 + 4 * w);
  }
  return strict_sumi_words<kFormat>(q, qh, y, F::kBias != 0 ? strict_ysum(y) : 0);
}

template <int kFormat>
__global__ void __launch_bounds__(256) sibling_sums_kernel(const uint8_t *__restrict__ vx, const uint8_t *__restrict__ vy,
                                                           int32_t *__restrict__ sumi, size_t bx, size_t by,
                                                           uint32_t nr, uint32_t nc, uint32_t nb) {
  using F = Sibling<kFormat>;
  const size_t total = static_cast<size_t>(nr) * nc * nb;
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
    const size_t ib = i % nb, rc = i / nb, col = rc % nc, row = rc / nc;
    sumi[i] = sibling_sumi<kFormat>(vx + row * bx + ib * F::kW, vy + col * by + ib * F::kA);
  }
}

template <int kFormat>
__global__ void __launch_bounds__(256) sibling_dot_kernel(const uint8_t *__restrict__ vx, const uint8_t *__restrict__ vy,
                                                          float *__restrict__ s, size_t bx, size_t by, size_t bs,
                                                          uint32_t nr, uint32_t nc, uint32_t nb) {
  using F = Sibling<kFormat>;
  pdl_enter();
  const int lane = threadIdx.x & 31;
  const size_t warp = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const size_t nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  const size_t total = static_cast<size_t>(nr) * nc;
  for (size_t item = warp; item < total; item += nwarps) {
    const size_t row = item / nc, col = item - row * nc;
    const uint8_t *wr = vx + row * bx;
    const uint8_t *xc = vy + col * by;
    float acc = 0.0f;
    for (uint32_t base = 0; base < nb; base += 32) {
      const uint32_t ib = base + lane;
      float term_a = 0.0f, term_b = 0.0f;  // min formats: a = the block's whole term; Q5_0: a = sumi, b = d_x*d_y
      if (ib < nb) {
        const uint8_t *xb = wr + static_cast<size_t>(ib) * F::kW;
        const uint8_t *yb = xc + static_cast<size_t>(ib) * F::kA;
        const float p = __fmul_rn(half_bits_to_float(load_u16(xb)), half_bits_to_float(load_u16(yb)));
        const float fs = __int2float_rn(sibling_sumi<kFormat>(xb, yb));
        if constexpr (F::kFold == kFoldMin) {
          const float ms = __fmul_rn(half_bits_to_float(load_u16(xb + 2)), half_bits_to_float(load_u16(yb + 2)));
          term_a = __fmaf_rn(p, fs, ms);
        } else {
          term_a = fs;
          term_b = p;
        }
      }
      const uint32_t live = min(32u, nb - base);
      for (uint32_t j = 0; j < live; ++j) {
        const float a = __shfl_sync(0xffffffffu, term_a, j);
        if constexpr (F::kFold == kFoldMin) {
          acc = __fadd_rn(acc, a);
        } else {
          acc = __fmaf_rn(__shfl_sync(0xffffffffu, term_b, j), a, acc);
        }
      }
    }
    if (lane == 0)
      s[row * bs + col] = acc;
  }
}

// Which of the two streaming kernels takes a call that both accept: strict_stream.cuh (a term table per
// CTA, 512 workers on one slot) or gemv_any.cuh (a table per warp, a row is one warp's work).  One column is the
// former's.  With several the latter wins where each of its warps has its rows in one slot and enough of them
// have work, and with up to 4 columns at middling row lengths, where its lanes are full and two rows share the
// columns' loads (not for Q5_0 below 4 columns: its table has two planes).  Both kernels timed on 2304 calls, 3
// formats x 1..8 columns x 512..32000 rows x K 256..28672, weights from HBM: the rule is 0.4 % over the better
// one on average, 19 % at worst, always the former 0.7 %, always the latter 21 %.  us, table per CTA / per warp:
//   1 column   Q5_0 11008 x 4096 9.0 / 12.3, 512 x 8192 3.6 / 5.4; Q4_1 11008 x 4096 8.2 / 9.1, 4096 x 11008 10.8 / 11.0; Q5_1 32000 x
//              4096 20.0 / 23.1
//   2          Q4_1 4096 x 4096 6.4 / 6.0, 11008 x 4096 12.2 / 11.6, 4096 x 11008 13.5 / 15.6; Q5_0 11008 x 4096 13.9 / 14.7; Q5_1 11008 x
//              6400 20.0 / 22.9; Q5_0 1024 x 4096 (a slot to a warp) 3.9 / 3.7
//   3, 4       Q4_1 4096 x 4096, 3 columns 7.7 / 6.4; 11008 x 4096, 4 columns Q4_1 15.6 / 14.0, Q5_0 19.7 / 18.4, Q5_1 17.9 / 16.9; Q5_1
//              11008 x 1024 6.7 / 7.0, 11008 x 6400 26.6 / 30.3; Q4_1 11008 x 4608 18.2 / 17.5; Q5_0 32000 x 512, 3 columns 9.3 / 16.8
//   5..8       Q5_1 11008 x 4096, 8 columns 26.7 / 28.0, 4096 x 11008, 6 columns 25.6 / 41.9; a slot to a warp: Q5_0 1536 x 4096, 8
//              columns 8.3 / 7.5, but 512 rows 4.7 / 6.5 (Q5_1)
//   few rows   (1476 more calls with 64..1600) Q5_0 100 x 512, 8 columns 3.3 / 2.6, 444 x 1024, 4 columns 3.2 / 2.7, 450 rows 3.0 / 3.5,
//              888 rows, 2 columns 2.9 / 2.6, 1100 rows 2.8 / 3.3; Q4_1 148 x 4096, 2 columns 3.0 / 3.4
template <int kFormat>
bool table_per_cta(const GemvAnyPlan &plan, uint32_t nb, size_t nr, size_t nc, int sms) {
  if (nc == 1)
    return true;
  const GemvAnyArgs &a = plan.args;
  const size_t blocks = nb * nc, n = static_cast<size_t>(sms);
  if (nr <= n * a.nwarps * a.rps) {
    if (kFormat == 2 && nb <= 64 && (nr <= 3 * n || (nr >= 5 * n && nr <= 7 * n)))
      return false;
    return nr < 5 * n || blocks < 256;
  }
  if (nc > 4 || (kFormat == 2 && nc < 4))
    return true;
  return nr < 20 * n || nb > 160 || blocks < 256 || blocks > 600;
}

// One column against rows so long that shared memory has a ring for one warp only: past seven rows for it the
// general kernel, which reads them in place, is no slower (us, that one / this: 1000 x 61440 Q4_1 113 / 75, Q5_0 130 / 80,
// Q5_1 103 / 84; 1184 rows 69 / 85, 77 / 91, 72 / 96; 4096 rows 191 / 287, 226 / 307, 213 / 325).
inline bool one_ring_too_many_rows(const GemvAnyPlan &plan, size_t nr, size_t nc, int sms) {
  return nc == 1 && plan.args.nwarps == 1 && nr > 7 * static_cast<size_t>(sms);
}

template <int kFormat>
int launch_one(size_t n, float *s, int32_t *sums, const uint8_t *vx, const uint8_t *vy, size_t by, size_t nr, size_t nc,
               size_t bx, size_t bs, cudaStream_t stream) {
  const uint32_t nb = static_cast<uint32_t>(n / kQK);
  if (nr == 0 || nc == 0)
    return TCRV_CUDA_OK;
  const size_t cap = static_cast<size_t>(sm_count()) * 8;
  if (sums != nullptr) {
    if (nb == 0)
      return TCRV_CUDA_OK;
    const size_t want = (nr * nc * nb + 255) / 256;
    sibling_sums_kernel<kFormat><<<static_cast<int>(want < cap ? want : cap), 256, 0, stream>>>(
        vx, vy, sums, bx, by, static_cast<uint32_t>(nr), static_cast<uint32_t>(nc), nb);
  } else {
    const int sms = sm_count();
    const uint32_t rps = strict_stream_rows<kFormat>(nb, nr, nc, vx, bx, sms);  // 0: not for that kernel
    GemvAnyPlan plan;
    const bool any = nr >= 8 && (rps != 0 || !any_tiny(nb, nr, nc, /*strict=*/true, sms)) &&
                     plan_gemv_any<kFormat>(n, s, vx, vy, by, nr, nc, bx, bs, /*strict=*/true, /*static_weights=*/false, sms, plan) &&
                     !one_ring_too_many_rows(plan, nr, nc, sms);
    // (activations at odd addresses are not for the table per warp)
    if (rps != 0 && (!any || table_per_cta<kFormat>(plan, nb, nr, nc, sms)))
      return launch_strict_stream<kFormat>(n, s, vx, vy, by, nr, nc, bx, bs, rps, sms, stream);
    if (any)
      return launch_gemv_any<kFormat, true>(plan, stream);
    const size_t want = (nr * nc + 7) / 8;
    TCRV_CUDA_TRY(launch_pdl(sibling_dot_kernel<kFormat>, static_cast<int>(want < cap ? want : cap), 256, 0, stream, vx, vy, s,
                             bx, by, bs, static_cast<uint32_t>(nr), static_cast<uint32_t>(nc), nb));
  }
  TCRV_CUDA_TRY(cudaGetLastError());
  return TCRV_CUDA_OK;
}

// out[0] = acc[0] + sum over the n weight bytes of v0 * qlo + v1 * qhi, v0 / v1 the low / high
// nibble of (byte ^ 0x88) sign-extended: the reference's integer-core kernel.  int32 wraps, so
// the order of the additions does not matter; one CTA.
__global__ void __launch_bounds__(256) integer_core_kernel(const int8_t *__restrict__ w, const int8_t *__restrict__ qlo,
                                                           const int8_t *__restrict__ qhi,
                                                           const int32_t *__restrict__ acc, int32_t *__restrict__ out,
                                                           size_t n) {
  __shared__ uint32_t partial[8];
  uint32_t sum = 0;
  for (size_t j = threadIdx.x; j < n; j += blockDim.x) {
    const uint8_t t = static_cast<uint8_t>(w[j]) ^ 0x88u;
    const int v0 = static_cast<int8_t>(static_cast<uint8_t>(t << 4)) >> 4, v1 = static_cast<int8_t>(t) >> 4;
    sum += static_cast<uint32_t>(v0 * qlo[j] + v1 * qhi[j]);
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1)
    sum += __shfl_xor_sync(0xffffffffu, sum, off);
  if ((threadIdx.x & 31) == 0)
    partial[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t total = static_cast<uint32_t>(acc[0]);
    for (int i = 0; i < 8; ++i)
      total += partial[i];
    out[0] = static_cast<int32_t>(total);
  }
}

}  // namespace

int launch_q4_0_q8_0_integer_core(const int8_t *w, const int8_t *qlo, const int8_t *qhi, const int32_t *acc,
                                  int32_t *out, size_t n, cudaStream_t stream) {
  integer_core_kernel<<<1, 256, 0, stream>>>(w, qlo, qhi, acc, out, n);
  TCRV_CUDA_TRY(cudaGetLastError());
  return TCRV_CUDA_OK;
}

int sibling_block_bytes(int format, size_t *weight, size_t *activation) {
  switch (format) {
    case 1: *weight = 20, *activation = 36; return TCRV_CUDA_OK;
    case 2: *weight = 22, *activation = 34; return TCRV_CUDA_OK;
    case 3: *weight = 24, *activation = 36; return TCRV_CUDA_OK;
    default: return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  }
}

int launch_sibling_dot(int format, size_t n, float *s, int32_t *sums, const uint8_t *vx, const uint8_t *vy, size_t by,
                       size_t nr, size_t nc, size_t bx, size_t bs, cudaStream_t stream) {
  switch (format) {
    case 1: return launch_one<1>(n, s, sums, vx, vy, by, nr, nc, bx, bs, stream);
    case 2: return launch_one<2>(n, s, sums, vx, vy, by, nr, nc, bx, bs, stream);
    case 3: return launch_one<3>(n, s, sums, vx, vy, by, nr, nc, bx, bs, stream);
    default: return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  }
}

}  // namespace tcrv
