// Streaming GEMV for rows of ANY block count: s[row*bs + col] for up to 8 activation columns,
// weights in any of the five block formats, rows that start anywhere on a 2-byte boundary.
//
// The kernels of gemv_stream.cuh, gemv_mma*.cuh and strict_stream.cuh need rows that start on 16
// bytes (a block count that is a multiple of 8 for the 18- and 34-byte blocks).  A model whose
// width is no multiple of 256 has other rows, and the general warp-per-output kernels read those
// byte by byte: 13.6 us for 4000 x 2912 Q4_0, 13 times the weights' time on the bus.  Here the
// weights still come in by the bulk copy engine: a slot of rows is fetched from the 16-byte
// boundary below its first byte to the one above its last (both inside the matrix; the few bytes
// at the very beginning or end of a matrix that would lie outside are read by the lanes), and a
// lane re-aligns its words with one funnel shift each when its row starts in the middle of a word.
//
// Same structure as gemv_stream.cuh: one CTA per SM, up to 16 warps, each with a private ring of
// two slots that it feeds itself with one copy in flight; a lane owns PAIRS of blocks where blocks
// are an odd number of half words (18, 22, 34 bytes), single blocks otherwise (20, 24 bytes), so
// that the stride between lanes is an odd number of words (24-byte blocks: two-way conflicts).
//
// fp32 order.  kStrict = false (Q4_0, Q8_0): lane l folds pairs l, l+32, ... ascending and a
// butterfly combines the lanes.  kStrict = true: the block terms go into the warp's table
// term[column][row][block] and lane (column, row) folds them block after block, the operations of
// the sequential fold (see strict_stream.cuh for the three forms).
#pragma once

#include "async_copy.cuh"
#include "strict_stream.cuh"
#include "tcrv_common.cuh"

namespace tcrv {

constexpr int kAnyMaxWarps = 16;
constexpr int kAnyRing = 2;
constexpr int kAnyBarrierBytes = kAnyMaxWarps * kAnyRing * 8;

struct GemvAnyArgs {
  const uint8_t *vx;
  const uint8_t *vy;
  float *s;
  size_t bx, by, bs;
  size_t total;  // bytes of the matrix: (nr - 1) * bx + row_bytes
  uint32_t nr, nc, nb, row_bytes;
  uint32_t nwarps, rps, slot_bytes, row_pitch, table_bytes;
  uint32_t contiguous, static_weights;
};

template <int kFormat>
struct AnyFormat {
  using F = StrictFormat<kFormat>;
  static constexpr bool kPairs = F::kW % 4 != 0;
  static constexpr uint32_t kUnit = kPairs ? 2 : 1;              // blocks per work item
  static constexpr uint32_t kUnitWords = kUnit * F::kW / 4;      // 9, 17, 11 / 5, 6
  static constexpr uint32_t kQWords = F::kNibbles ? 4 : 8;
  static constexpr bool kTwo = F::kFold == kFoldProduct;         // (float)sumi and the scale product kept apart
};

// Items per row, and the block count the per-block arrays are padded to (zero terms fold to nothing).
template <int kFormat>
__host__ __device__ inline uint32_t any_units(uint32_t nb) {
  return (nb + AnyFormat<kFormat>::kUnit - 1) / AnyFormat<kFormat>::kUnit;
}
__host__ __device__ inline uint32_t any_padded(uint32_t nb) { return (nb + 3) / 4 * 4; }
// a column: kUnit * 2 planes of 16 bytes per item, then scale and integer sum (or s) per block
// (where the block's sum starts, or s)
template <int kFormat>
__host__ __device__ inline uint32_t any_xcol_bytes(uint32_t nb) {
  return any_units<kFormat>(nb) * AnyFormat<kFormat>::kUnit * 32u + any_padded(nb) * 8u;
}
template <int kFormat>
__host__ __device__ inline uint32_t any_table_bytes(uint32_t nb, uint32_t rps, uint32_t cols) {
  return cols * rps * (any_padded(nb) + 4u) * 4u * (AnyFormat<kFormat>::kTwo ? 2u : 1u);
}

// One block of an item, cut out of the item's words.
struct AnyBlock {
  uint32_t d, m, qh;
  uint32_t q[8];
};
template <int kFormat>
__device__ __forceinline__ void any_block(const uint32_t (&w)[AnyFormat<kFormat>::kUnitWords], uint32_t h, AnyBlock &b) {
  using F = StrictFormat<kFormat>;
  constexpr uint32_t QW = AnyFormat<kFormat>::kQWords;
  b.m = b.qh = 0;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    b.q[k] = 0;
  if constexpr (!AnyFormat<kFormat>::kPairs) {
    b.d = w[0] & 0xffffu, b.m = w[0] >> 16;
#pragma unroll
    for (uint32_t k = 0; k < QW; ++k)
      b.q[k] = w[F::kWq / 4 + k];
    if constexpr (F::kQh != 0)
      b.qh = w[F::kQh / 4];
  } else if (h == 0) {
    b.d = w[0] & 0xffffu;
#pragma unroll
    for (uint32_t k = 0; k < QW; ++k)
      b.q[k] = __funnelshift_r(w[(F::kWq + 4 * k) / 4], w[(F::kWq + 4 * k) / 4 + 1], 16);
    if constexpr (F::kQh != 0)
      b.qh = __funnelshift_r(w[F::kQh / 4], w[F::kQh / 4 + 1], 16);
  } else {
    b.d = w[F::kW / 4] >> 16;
#pragma unroll
    for (uint32_t k = 0; k < QW; ++k)
      b.q[k] = w[(F::kW + F::kWq + 4 * k) / 4];
    if constexpr (F::kQh != 0)
      b.qh = w[(F::kW + F::kQh) / 4];
  }
}

// The activation values that meet one item.
template <int kFormat>
struct AnyX {
  uint32_t y[AnyFormat<kFormat>::kUnit][8];
  float d[AnyFormat<kFormat>::kUnit];
  uint32_t s[AnyFormat<kFormat>::kUnit];  // where the block's sum starts (strict_start), or Q8_1's s as float bits
};
template <int kFormat>
__device__ __forceinline__ void any_load_x(AnyX<kFormat> &x, const uint8_t *xcol, uint32_t units, uint32_t nbp, uint32_t p) {
  constexpr uint32_t U = AnyFormat<kFormat>::kUnit;
  const uint4 *planes = reinterpret_cast<const uint4 *>(xcol);
  const uint8_t *tail = xcol + units * U * 32u;
#pragma unroll
  for (uint32_t h = 0; h < U; ++h) {
    const uint4 a = planes[(2 * h) * units + p], b = planes[(2 * h + 1) * units + p];
    x.y[h][0] = a.x, x.y[h][1] = a.y, x.y[h][2] = a.z, x.y[h][3] = a.w;
    x.y[h][4] = b.x, x.y[h][5] = b.y, x.y[h][6] = b.z, x.y[h][7] = b.w;
  }
  if constexpr (U == 2) {
    const float2 d = reinterpret_cast<const float2 *>(tail)[p];
    const uint2 s = reinterpret_cast<const uint2 *>(tail + nbp * 4u)[p];
    x.d[0] = d.x, x.d[1] = d.y, x.s[0] = s.x, x.s[1] = s.y;
  } else {
    x.d[0] = reinterpret_cast<const float *>(tail)[p];
    x.s[0] = reinterpret_cast<const uint32_t *>(tail + nbp * 4u)[p];
  }
}

// Items of a lane that fit in registers for a whole kernel (one column): rows of up to 128 blocks.
template <int kFormat>
constexpr int kAnyXItems = AnyFormat<kFormat>::kPairs ? 2 : 4;

// kRows rows of a slot against every column.  kMis: a row may start in the middle of a word.
// kXReg: the lane's activation items are in `xr` (one column, at most kAnyXItems items a lane).
template <int kFormat, int kCols, bool kStrict, bool kMis, bool kXReg, int kRows>
__device__ __forceinline__ void any_rows(const GemvAnyArgs &a, const uint8_t *slot, const uint32_t (&off)[4],
                                         const AnyX<kFormat> *xr, const uint8_t *xsm, uint32_t xcol_bytes, float *table,
                                         uint32_t row, int lane) {
  using F = StrictFormat<kFormat>;
  using A = AnyFormat<kFormat>;
  constexpr uint32_t U = A::kUnit, UW = A::kUnitWords;
  const uint32_t nb = a.nb, units = any_units<kFormat>(nb), nbp = any_padded(nb), pitch = nbp + 4u;
  const uint32_t ncols = kCols == 1 ? 1u : a.nc;
  const uint32_t *base[kRows];
  uint32_t sh[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    base[r] = reinterpret_cast<const uint32_t *>(slot + (kMis ? off[r] & ~3u : off[r]));
    sh[r] = (off[r] & 2u) * 8u;
  }
  float acc[kRows][kCols];
#pragma unroll
  for (int r = 0; r < kRows; ++r)
#pragma unroll
    for (int c = 0; c < kCols; ++c)
      acc[r][c] = 0.0f;
  float *prod = table + ncols * kRows * pitch;  // kTwo: the second plane
  auto one_item = [&](uint32_t p, [[maybe_unused]] const AnyX<kFormat> *xp) {
    uint32_t w[kRows][UW];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      if constexpr (kMis) {
        uint32_t t[UW + 1];
#pragma unroll
        for (uint32_t k = 0; k <= UW; ++k)
          t[k] = base[r][p * UW + k];
#pragma unroll
        for (uint32_t k = 0; k < UW; ++k)
          w[r][k] = __funnelshift_r(t[k], t[k + 1], sh[r]);
      } else {
#pragma unroll
        for (uint32_t k = 0; k < UW; ++k)
          w[r][k] = base[r][p * UW + k];
      }
    }
    const bool second = U == 2 && 2 * p + 1 < nb;
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
      if (kCols > 1 && c >= static_cast<int>(ncols))
        break;
      AnyX<kFormat> x;
      if constexpr (kXReg)
        x = *xp;
      else
        any_load_x<kFormat>(x, xsm + static_cast<size_t>(c) * xcol_bytes, units, nbp, p);
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        float term[U], pr[U];
#pragma unroll
        for (uint32_t h = 0; h < U; ++h) {
          AnyBlock b;
          any_block<kFormat>(w[r], h, b);
          const float dw = half_bits_to_float(b.d);
          // (five-bit codes are merged for one column too: the words that their fifth bits would meet cost a
          // third of the rings on long rows, us: Q5_0 2048 x 49152 66 -> 126, or the kernel: 64 x 61440 14 -> 75)
          const float fs = strict_dot<kFormat, kCols == 1 && F::kQh == 0>(b.q, b.qh, x.y[h], x.y[h],
                                                           F::kBias == 0 ? kStrictMagicBits : x.s[h]);
          pr[h] = 0.0f;
          if constexpr (!kStrict) {
            const float next = kFormat == 5 ? __fmaf_rn(fs, __fmul_rn(dw, x.d[h]), acc[r][c])
                                            : __fmaf_rn(__fmul_rn(fs, dw), x.d[h], acc[r][c]);
            acc[r][c] = (h == 0 || second) ? next : acc[r][c];
          } else if constexpr (F::kFold == kFoldMin) {
            term[h] = __fmaf_rn(__fmul_rn(dw, x.d[h]), fs, __fmul_rn(half_bits_to_float(b.m), __uint_as_float(x.s[h])));
          } else if constexpr (F::kFold == kFoldProduct) {
            term[h] = fs;
            pr[h] = __fmul_rn(dw, x.d[h]);
          } else {
            term[h] = __fmul_rn(fs, dw);
          }
        }
        if constexpr (kStrict) {
          float *t = table + (static_cast<uint32_t>(c) * kRows + r) * pitch + U * p;
          float *q = prod + (static_cast<uint32_t>(c) * kRows + r) * pitch + U * p;
          if constexpr (U == 2) {
            *reinterpret_cast<float2 *>(t) = make_float2(term[0], second ? term[1] : 0.0f);
            if constexpr (A::kTwo)
              *reinterpret_cast<float2 *>(q) = make_float2(pr[0], second ? pr[1] : 0.0f);
          } else {
            *t = term[0];
            if constexpr (A::kTwo)
              *q = pr[0];
          }
        }
      }
    }
  };
  if constexpr (kXReg) {
#pragma unroll
    for (int i = 0; i < kAnyXItems<kFormat>; ++i)
      if (lane + 32u * i < units)
        one_item(lane + 32u * i, xr + i);
  } else {
    for (uint32_t p = lane; p < units; p += 32)
      one_item(p, nullptr);
  }
  if constexpr (!kStrict) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
#pragma unroll
      for (int r = 0; r < kRows; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c)
          acc[r][c] = __fadd_rn(acc[r][c], __shfl_xor_sync(0xffffffffu, acc[r][c], o));
    // lane (row, column) stores
    float mine = 0.0f;
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int c = 0; c < kCols; ++c)
        mine = lane == r * kCols + c ? acc[r][c] : mine;
    const uint32_t r = static_cast<uint32_t>(lane) / kCols, c = static_cast<uint32_t>(lane) % kCols;
    if (r < kRows && c < ncols)
      a.s[static_cast<size_t>(row + r) * a.bs + c] = mine;
  } else {
    // zero terms up to the padded block count
    for (uint32_t b = U * units + lane; b < nbp; b += 32)
      for (uint32_t i = 0; i < ncols * kRows; ++i) {
        table[i * pitch + b] = 0.0f;
        if constexpr (A::kTwo)
          prod[i * pitch + b] = 0.0f;
      }
    __syncwarp();
    if (static_cast<uint32_t>(lane) < ncols * kRows) {
      const uint32_t c = static_cast<uint32_t>(lane) / kRows, r = static_cast<uint32_t>(lane) % kRows;
      const float4 *t = reinterpret_cast<const float4 *>(table + static_cast<uint32_t>(lane) * pitch);
      const float4 *m = A::kTwo ? reinterpret_cast<const float4 *>(prod + static_cast<uint32_t>(lane) * pitch)
                                : reinterpret_cast<const float4 *>(xsm + static_cast<size_t>(c) * xcol_bytes + units * U * 32u);
      float sum = 0.0f;
#pragma unroll 4
      for (uint32_t i = 0; i < nbp / 4; ++i) {
        const float4 tv = t[i];
        if constexpr (F::kFold == kFoldMin) {
          sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, tv.x), tv.y), tv.z), tv.w);
        } else {
          const float4 mv = m[i];
          sum = __fmaf_rn(tv.x, mv.x, sum);
          sum = __fmaf_rn(tv.y, mv.y, sum);
          sum = __fmaf_rn(tv.z, mv.z, sum);
          sum = __fmaf_rn(tv.w, mv.w, sum);
        }
      }
      a.s[static_cast<size_t>(row + r) * a.bs + c] = sum;
    }
    __syncwarp();  // the table may be written again
  }
}

// CTA `cta` of the `nctas` that share the problem.  The block may have more warps than a.nwarps.
template <int kFormat, int kCols, bool kStrict, bool kMis, bool kXReg>
__device__ __forceinline__ void gemv_any_body(const GemvAnyArgs &a, uint32_t cta, uint32_t nctas, uint8_t *smem) {
  using F = StrictFormat<kFormat>;
  constexpr uint32_t U = AnyFormat<kFormat>::kUnit;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem);
  uint8_t *xsm = smem + kAnyBarrierBytes;
  const uint32_t nb = a.nb, units = any_units<kFormat>(nb), nbp = any_padded(nb);
  const uint32_t xcol_bytes = any_xcol_bytes<kFormat>(nb);
  const uint32_t ncols = kCols == 1 ? 1u : a.nc;
  uint8_t *tables = xsm + static_cast<size_t>(ncols) * xcol_bytes;
  uint8_t *slots = tables + static_cast<size_t>(a.nwarps) * a.table_bytes;
  const uint32_t warp = threadIdx.x >> 5, nwarps = a.nwarps, rps = a.rps;
  const int lane = threadIdx.x & 31;
  const bool spare = warp >= nwarps;
  const uint32_t r0 = static_cast<uint32_t>(static_cast<uint64_t>(a.nr) * cta / nctas);
  const uint32_t r1 = static_cast<uint32_t>(static_cast<uint64_t>(a.nr) * (cta + 1) / nctas);
  const uint32_t w0 = r0 + (r1 - r0) * warp / nwarps;
  const uint32_t wrows = spare ? 0 : r0 + (r1 - r0) * (warp + 1) / nwarps - w0;
  const uint32_t mine = (wrows + rps - 1) / rps;
  const uint32_t slot_rows = mine > 0 ? wrows / mine : 0, slot_extra = mine > 0 ? wrows % mine : 0;
  auto slot_row = [&](uint32_t t) { return w0 + t * slot_rows + min(t, slot_extra); };
  auto slot_count = [&](uint32_t t) { return slot_rows + (t < slot_extra ? 1u : 0u); };

  // Byte offsets from the 16-byte boundary at or below vx.  A range [first, last) of the matrix is
  // copied as [from, to): rounded outwards to 16 bytes, but never outside the matrix.
  const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(a.vx) & 15u);
  const uint8_t *base = a.vx - lead;
  const size_t low = (lead + 15u) & ~static_cast<size_t>(15), high = (lead + a.total) & ~static_cast<size_t>(15);
  auto clip = [&](size_t first, size_t last, size_t &from, size_t &to) {
    from = first & ~static_cast<size_t>(15);
    from = from < low ? low : from;
    to = (last + 15) & ~static_cast<size_t>(15);
    to = to > high ? high : to;
  };
  // pieces of a slot: one when rows are contiguous, else one per row
  auto piece = [&](uint32_t t, uint32_t i, size_t &first, size_t &last) {
    first = lead + (static_cast<size_t>(slot_row(t)) + i) * a.bx;
    last = a.contiguous ? lead + static_cast<size_t>(slot_row(t)) * a.bx + static_cast<size_t>(slot_count(t)) * a.row_bytes
                        : first + a.row_bytes;
  };
  auto issue = [&](uint32_t t) {  // one lane
    const uint32_t bar = warp * kAnyRing + t % kAnyRing;
    const uint32_t pieces = a.contiguous ? 1u : slot_count(t);
    uint32_t bytes = 0;
    for (uint32_t i = 0; i < pieces; ++i) {
      size_t first, last, from, to;
      piece(t, i, first, last);
      clip(first, last, from, to);
      bytes += to > from ? static_cast<uint32_t>(to - from) : 0u;
    }
    mbar_arrive_expect_tx(&full[bar], bytes);
    uint8_t *slot = slots + static_cast<size_t>(bar) * a.slot_bytes;
    for (uint32_t i = 0; i < pieces; ++i) {
      size_t first, last, from, to;
      piece(t, i, first, last);
      clip(first, last, from, to);
      if (to > from)
        bulk_copy_g2s(slot + i * a.row_pitch + (from - (first & ~static_cast<size_t>(15))), base + from,
                      static_cast<uint32_t>(to - from), &full[bar]);
    }
  };

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (!a.static_weights)
    asm volatile("griddepcontrol.wait;" ::: "memory");
  if (lane == 0 && !spare) {
    for (uint32_t i = 0; i < kAnyRing; ++i)
      mbar_init(&full[warp * kAnyRing + i], 1);
    mbar_fence_init();
    if (mine > 0)
      issue(0);
  }
  if (a.static_weights)
    asm volatile("griddepcontrol.wait;" ::: "memory");
  // the activation columns (2-byte aligned blocks) into planes; blocks past the end are zero
  for (uint32_t idx = threadIdx.x; idx < ncols * max(nbp, U * units); idx += blockDim.x) {
    const uint32_t per = max(nbp, U * units), col = idx / per, ib = idx - col * per;
    uint8_t *xcol = xsm + static_cast<size_t>(col) * xcol_bytes;
    uint32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint32_t third = 0;
    float d = 0.0f;
    if (ib < nb) {
      const unsigned short *h = reinterpret_cast<const unsigned short *>(a.vy + col * a.by + static_cast<size_t>(ib) * F::kA);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        q[j] = static_cast<uint32_t>(h[F::kAq / 2 + 2 * j]) | (static_cast<uint32_t>(h[F::kAq / 2 + 1 + 2 * j]) << 16);
      d = half_bits_to_float(h[0]);
      if constexpr (F::kFold == kFoldMin)
        third = __float_as_uint(half_bits_to_float(h[1]));
      else
        third = strict_start<kFormat>(F::kBias != 0 ? strict_ysum(q) : 0);
    }
    const uint32_t p = ib / U, h = ib % U;
    if (p < units) {
      uint4 *planes = reinterpret_cast<uint4 *>(xcol);
      planes[(2 * h) * units + p] = make_uint4(q[0], q[1], q[2], q[3]);
      planes[(2 * h + 1) * units + p] = make_uint4(q[4], q[5], q[6], q[7]);
    }
    reinterpret_cast<float *>(xcol + units * U * 32u)[ib] = d;
    reinterpret_cast<uint32_t *>(xcol + units * U * 32u + nbp * 4u)[ib] = third;
  }
  __syncthreads();
  if (spare)
    return;

  AnyX<kFormat> xr[kXReg ? kAnyXItems<kFormat> : 1];
  if constexpr (kXReg) {
#pragma unroll
    for (int i = 0; i < kAnyXItems<kFormat>; ++i)
      if (lane + 32u * i < units)
        any_load_x<kFormat>(xr[i], xsm, units, nbp, lane + 32u * i);
  }
  float *table = reinterpret_cast<float *>(tables + static_cast<size_t>(warp) * a.table_bytes);
  for (uint32_t t = 0; t < mine; ++t) {
    const uint32_t bar = warp * kAnyRing + t % kAnyRing;
    if (!mbar_wait_bounded(&full[bar], (t / kAnyRing) & 1)) {
      if (lane == 0)
        raise_device_error(kDevErrBarrierTimeout);
      return;  // (one copy in flight: nothing else is on its way into this CTA's memory)
    }
    if (lane == 0 && t + 1 < mine) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(t + 1);
    }
    uint8_t *slot = slots + static_cast<size_t>(bar) * a.slot_bytes;
    const uint32_t row = slot_row(t), rows = slot_count(t);
    // what the copy could not reach: bytes before the first or after the last whole 16 of the matrix
    const uint32_t pieces = a.contiguous ? 1u : rows;
    if (row == 0 || row + rows == a.nr) {
      for (uint32_t i = 0; i < pieces; ++i) {
        size_t first, last, from, to;
        piece(t, i, first, last);
        clip(first, last, from, to);
        if (to <= from)
          from = to = last;  // no copy at all
        uint8_t *dst = slot + i * a.row_pitch - (first & ~static_cast<size_t>(15));
        for (size_t k = first + lane; k < min(from, last); k += 32)
          dst[k] = base[k];
        for (size_t k = max(to, first) + lane; k < last; k += 32)
          dst[k] = base[k];
      }
      __syncwarp();
    }
    uint32_t off[4];
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
      const size_t at = lead + (static_cast<size_t>(row) + (a.contiguous ? 0u : r)) * a.bx;
      off[r] = static_cast<uint32_t>(at & 15u) + r * (a.contiguous ? a.row_bytes : a.row_pitch);
    }
    if (rows == 4) {
      if constexpr (kCols == 1)
        any_rows<kFormat, kCols, kStrict, kMis, kXReg, 4>(a, slot, off, xr, xsm, xcol_bytes, table, row, lane);
    } else if (rows == 3) {
      if constexpr (kCols == 1)
        any_rows<kFormat, kCols, kStrict, kMis, kXReg, 3>(a, slot, off, xr, xsm, xcol_bytes, table, row, lane);
    } else if (rows == 2) {
      if constexpr (kCols <= 4)
        any_rows<kFormat, kCols, kStrict, kMis, kXReg, 2>(a, slot, off, xr, xsm, xcol_bytes, table, row, lane);
    } else {
      any_rows<kFormat, kCols, kStrict, kMis, kXReg, 1>(a, slot, off, xr, xsm, xcol_bytes, table, row, lane);
    }
    __syncwarp();
  }
}

template <int kFormat, int kCols, bool kStrict, bool kMis, bool kXReg>
__global__ void __launch_bounds__(kAnyMaxWarps * 32, 1) gemv_any_kernel(const __grid_constant__ GemvAnyArgs a) {
  extern __shared__ __align__(128) uint8_t smem[];
  gemv_any_body<kFormat, kCols, kStrict, kMis, kXReg>(a, blockIdx.x, gridDim.x, smem);
}

// Several independent one-column problems in one launch (see gemv_stream_group_kernel).
constexpr int kAnyGroupMax = 16;
struct GemvAnyGroupArgs {
  GemvAnyArgs problem[kAnyGroupMax];
  uint32_t first[kAnyGroupMax + 1];
  uint32_t count;
};
template <int kFormat, bool kStrict>
__global__ void __launch_bounds__(kAnyMaxWarps * 32, 1) gemv_any_group_kernel(const __grid_constant__ GemvAnyGroupArgs g) {
  extern __shared__ __align__(128) uint8_t smem[];
  uint32_t i = 0;
  while (i + 1 < g.count && blockIdx.x >= g.first[i + 1])
    ++i;
  const GemvAnyArgs &a = g.problem[i];
  const uint32_t cta = blockIdx.x - g.first[i], nctas = g.first[i + 1] - g.first[i];
  if (any_units<kFormat>(a.nb) <= 32u * kAnyXItems<kFormat>)
    gemv_any_body<kFormat, 1, kStrict, true, true>(a, cta, nctas, smem);
  else
    gemv_any_body<kFormat, 1, kStrict, true, false>(a, cta, nctas, smem);
}

// ------------------------------------------------------------------------------ host side

constexpr size_t kAnySmemCap = 227 * 1024;

struct GemvAnyPlan {
  GemvAnyArgs args;
  size_t smem;
  int grid;
};

// Fills the plan; false when the operands rule the kernel out (odd addresses, a column layout or a
// row that does not fit in shared memory).
template <int kFormat>
bool plan_gemv_any(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t by, size_t nr, size_t nc, size_t bx,
                   size_t bs, bool strict, bool static_weights, int sms, GemvAnyPlan &plan) {
  using F = StrictFormat<kFormat>;
  const uint32_t nb = static_cast<uint32_t>(n / kQK);
  if (nb == 0 || nr == 0 || nc == 0 || nc > 8 || ((reinterpret_cast<uintptr_t>(vx) | reinterpret_cast<uintptr_t>(vy)) & 1u) != 0 ||
      (nr > 1 && (bx & 1u) != 0) || (nc > 1 && (by & 1u) != 0))
    return false;
  const size_t row_bytes = static_cast<size_t>(nb) * F::kW;
  if (row_bytes > kAnySmemCap)
    return false;
  const uint32_t cols = static_cast<uint32_t>(nc);
  // (a lane reads whole items, one word ahead: up to 60 bytes past the end of a row)
  const size_t pitch = (row_bytes + 15) / 16 * 16 + 64;
  const size_t fixed = kAnyBarrierBytes + nc * static_cast<size_t>(any_xcol_bytes<kFormat>(nb));
  // rows per slot as in gemv_stream.cuh: four chains side by side on short rows and one column,
  // two up to 4 columns, one beyond (registers); fewer when the slots do not fit
  size_t rps = nc == 1 ? (row_bytes <= 4096 ? 4 : 2) : (nc <= 4 ? 2 : 1);
  auto per_warp = [&](size_t rows) {
    const size_t table = strict ? any_table_bytes<kFormat>(nb, static_cast<uint32_t>(rows), cols) : 0;
    return kAnyRing * rows * pitch + table;
  };
  // every warp should have work: no more rows per slot than a warp has rows
  const size_t rows_per_warp = (nr + static_cast<size_t>(sms) * kAnyMaxWarps - 1) / (static_cast<size_t>(sms) * kAnyMaxWarps);
  while (rps > 1 && (fixed + per_warp(rps) * 8 > kAnySmemCap || rps > rows_per_warp))
    rps /= 2;
  if (fixed + per_warp(rps) > kAnySmemCap)
    return false;
  size_t nwarps = (kAnySmemCap - fixed) / per_warp(rps);
  nwarps = nwarps > kAnyMaxWarps ? kAnyMaxWarps : nwarps;
  GemvAnyArgs &a = plan.args;
  a.vx = vx, a.vy = vy, a.s = s;
  a.bx = nr > 1 ? bx : row_bytes, a.by = by, a.bs = bs;
  a.total = (nr - 1) * a.bx + row_bytes;
  a.nr = static_cast<uint32_t>(nr), a.nc = cols, a.nb = nb, a.row_bytes = static_cast<uint32_t>(row_bytes);
  a.nwarps = static_cast<uint32_t>(nwarps), a.rps = static_cast<uint32_t>(rps);
  a.row_pitch = static_cast<uint32_t>(pitch), a.slot_bytes = static_cast<uint32_t>(rps * pitch);
  a.table_bytes = strict ? any_table_bytes<kFormat>(nb, a.rps, cols) : 0;
  a.contiguous = a.bx == row_bytes ? 1u : 0u;
  a.static_weights = static_weights ? 1u : 0u;
  const size_t nslots = (nr + rps - 1) / rps;
  plan.grid = static_cast<int>(nslots < static_cast<size_t>(sms) ? nslots : static_cast<size_t>(sms));
  plan.smem = fixed + nwarps * (kAnyRing * static_cast<size_t>(a.slot_bytes) + a.table_bytes);
  return true;
}

// Matrices that are done before this kernel is set up stay on the general kernels, which ask for no shared
// memory: in the strict order rows of one pass of a warp there and no more than one round of its warps, in
// the lane-pair order rows of half as many blocks, and outputs for at least half of the SMs (with fewer only
// a few CTAs of this kernel start).  us, general / this one:
//   strict Q4_0   148 x 5 blocks 2.0 / 3.1, 600 x 25 2.6 / 3.2, 1200 x 9 2.6 / 3.1, 1200 x 25 3.5 / 3.3, 600 x 33 3.4 / 3.2
//   strict Q5_0   148 x 9 2.0 / 3.1, 600 x 25 2.7 / 3.3, 1200 x 25 3.5 / 3.4, 600 x 33 3.5 / 3.3
//   lane pairs    300 x 5 2.4 / 2.9, 600 x 12 2.7 / 2.8, 300 x 17 2.9 / 2.9, 1200 x 5 3.0 / 2.9, 40 x 5 2.4 / 2.1
inline bool any_tiny(uint32_t nb, size_t nr, size_t nc, bool strict, int sms) {
  const size_t outputs = nr * nc, n = static_cast<size_t>(sms);
  return strict ? nb <= 32 && outputs <= 8 * n : nb <= 16 && 2 * outputs >= n && outputs <= 4 * n;
}

template <typename Kernel>
int any_configure(Kernel kernel, std::atomic<bool> (&configured)[64]) {
  int dev = 0;
  TCRV_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    TCRV_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kAnySmemCap)));
    if (dev >= 0 && dev < 64)
      configured[dev] = true;
  }
  return TCRV_CUDA_OK;
}

template <int kFormat, int kCols, bool kStrict, bool kMis, bool kXReg>
int launch_any_instance(const GemvAnyPlan &plan, cudaStream_t stream) {
  static std::atomic<bool> configured[64];
  auto kernel = gemv_any_kernel<kFormat, kCols, kStrict, kMis, kXReg>;
  const int st = any_configure(kernel, configured);
  if (st != TCRV_CUDA_OK)
    return st;
  // All 16 warps whatever a.nwarps is: where long rows or many columns leave shared memory for one or
  // two rings, the spare warps still stage the activations (8 rows x 1001 blocks x 4 columns of Q4_0:
  // 51.5 us with the one warp that has a ring, 12.1 us; the general kernel takes 34).
  TCRV_CUDA_TRY(launch_pdl(kernel, plan.grid, kAnyMaxWarps * 32, plan.smem, stream, plan.args));
  TCRV_CUDA_TRY(cudaGetLastError());
  return TCRV_CUDA_OK;
}

// (column counts are served by the next larger of 1, 2, 4, 8: the loops stop at the real count)
template <int kFormat, bool kStrict, bool kMis>
int launch_any_columns(const GemvAnyPlan &plan, cudaStream_t stream) {
  if (plan.args.nc == 1) {
    if (any_units<kFormat>(plan.args.nb) <= 32u * kAnyXItems<kFormat>)
      return launch_any_instance<kFormat, 1, kStrict, kMis, true>(plan, stream);
    return launch_any_instance<kFormat, 1, kStrict, kMis, false>(plan, stream);
  }
  if (plan.args.nc == 2)
    return launch_any_instance<kFormat, 2, kStrict, kMis, false>(plan, stream);
  if (plan.args.nc <= 4)
    return launch_any_instance<kFormat, 4, kStrict, kMis, false>(plan, stream);
  return launch_any_instance<kFormat, 8, kStrict, kMis, false>(plan, stream);
}

template <int kFormat, bool kStrict>
int launch_gemv_any(const GemvAnyPlan &plan, cudaStream_t stream) {
  // The sibling formats have no other streaming kernel for one word-aligned row after another, so
  // they get an instance without the re-alignment; Q4_0 and Q8_0 rows of that kind go elsewhere.
  if constexpr (kFormat <= 3) {
    const GemvAnyArgs &a = plan.args;
    if (((reinterpret_cast<uintptr_t>(a.vx) | a.bx) & 3u) == 0)
      return launch_any_columns<kFormat, kStrict, false>(plan, stream);
  }
  return launch_any_columns<kFormat, kStrict, true>(plan, stream);
}

}  // namespace tcrv
