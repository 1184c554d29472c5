// Decode GEMV for several (4..8) activation columns on the tensor cores (legacy warp-level MMA,
// mma.sync.m16n8k32.s8: 16 weight rows x 32 K x 8 columns is exactly one ggml block of a
// 16-row group against all columns).  With several columns the dp4a kernel is issue-bound
// long before HBM is; here one MMA replaces 16 x 8 x 8 dp4a.  This is the form for rows of more than
// 4096 elements; shorter rows take the whole-row form in gemv_mma_rows.cuh (same arithmetic, same
// order).
//
// One persistent CTA per SM owns a contiguous range of 16-row groups, taken two at a time (one with Q8_0
// weights).  All 16 warps of the CTA work on the SAME rows and split K: the row's blocks are cut into
// chunks of 8 (144 bytes of Q4_0, 272 of Q8_0 per row) and warp w takes chunks w, w+16, ...: at most
// three, so the activation fragments of its chunks stay in registers for the whole kernel (the
// scales in shared memory).  A warp brings everything it needs itself, by 16-byte asynchronous copies: its
// columns' bytes once, its rows' bytes chunk by chunk through a ring of its own.  No warp waits for another
// before the K partials meet.  A unit of the ring is 16 rows of a chunk; its row pitch is 16 bytes times
// an odd number for both formats, so the 8 rows x 4 words an MMA fragment load touches fall into 32
// different banks.
//
// Before, a chunk was one tiled TMA box (144-byte rows cost the copy engine about 8 cycles each: 5.6 us for
// 32 x 11008 on an SM) and the CTA staged all columns in a fragment layout behind a barrier.  8 columns, us
// before / after: 64 x 11008 8.0 / 5.9, 4096 x 11008 13.0 / 11.0, 11008 x 11008 23.0 / 22.0, 16000 x 6400
// 20.4 / 19.2.  What is left of the third: 2 us of launch, 1.5 until the columns have arrived (148 copies
// of 94 KB out of L2), 3.5 for each wave of 16-row groups (2.3 at the copy rate; 1.5 of issue), 1 to combine.
//
// Fragments: thread (g = lane/4, t = lane%4) holds A = rows g and g+8, K bytes 4t..4t+3 and
// 16+4t.. -- for Q4_0 that is quant word t of the block (low nibbles -> first K half, high
// nibbles -> second half), B = column g, the same K bytes, C = rows g, g+8 x columns 2t, 2t+1.  The
// int32 tile of each block is folded into fp32 with that block's two scales before the next block.
//
// What surrounds an MMA is kept short, because instruction issue bounds these kernels:
// * A nibble moved to the top of its byte, its top bit flipped, is the int8 16 * (nibble - 8): no
//   offset to correct.  The tile is then 16 * S, and the activation scales are staged as d_x / 16.
// * The MMA's C input is 0x4B400000, the bits of the float 12582912 = 1.5 * 2^23, in every element: as long
//   as the sum stays below 2^22 in magnitude (16 * 32 * 8 * 128 = 2^19; 32 * 128 * 128 = 2^19) the result's bits
//   are those of the float 12582912 + sum, and the conversion costs nothing:
//     Q4_0: fma(12582912 + 16 S, d_w, -12582912 * d_w) == 16 * ((float)S * d_w), rounded once, as in the
//           reference order (-12582912 * d_w is exact: d_w has an 11-bit significand); times d_x / 16
//           that is the reference's second factor, since powers of two move through exactly
//     Q8_0: (12582912 + S) - 12582912 == (float)S exactly.
//
// fp32 order: partial w folds its chunks in ascending order (blocks ascending inside a chunk)
// with the fused fold, starting from 0.0f; the row value is ((p_0 + p_1) + ...) + p_15.
#pragma once

#include <type_traits>

#include "async_copy.cuh"
#include "gemv_stream.cuh"

namespace tcrv {

constexpr int kMmaWarps = 16;
constexpr int kMmaThreads = kMmaWarps * 32;
constexpr int kMmaRows = 16;        // rows of one MMA
constexpr int kMmaCols = 8;         // columns of one MMA
constexpr int kMmaMaxSlotGroups = 2;
constexpr int kMmaChunkBlocks = 8;
constexpr int kMmaPartialRing = 2;  // slots (pairs of row groups) whose K-partials may be waiting to be combined
constexpr int kMmaBarrierBytes = 128;  // a full/empty pair per partial buffer, an abort word
constexpr int kMmaPartialBytes = kMmaPartialRing * kMmaWarps * kMmaMaxSlotGroups * 32 * 16;  // a float4 per thread, group, buffer
constexpr int kMmaXColBytes = kMmaChunkBlocks * kQ8Block;   // 272: a chunk of one column
constexpr int kMmaXWarpBytes = kMmaCols * kMmaXColBytes;    // 2176
// the first chunk of every warp's columns is staged in the room the partial ring uses afterwards
constexpr int kMmaScratchBytes = kMmaWarps * kMmaXWarpBytes > kMmaPartialBytes ? kMmaWarps * kMmaXWarpBytes : kMmaPartialBytes;

// 16-row groups per slot, and chunks per row and warp, whose activation fragments stay in registers.  A ring
// position of a warp holds one chunk of one group; there are as many as fit.
template <bool kQ8W>
constexpr int kMmaGroups = kQ8W ? 1 : 2;
template <bool kQ8W>
constexpr int kMmaWarpChunks = kQ8W ? 2 : 3;
template <bool kQ8W>
constexpr int kMmaRing = kQ8W ? 2 : 5;
template <bool kQ8W>
constexpr int kMmaUnitBytes = kMmaRows * kMmaChunkBlocks * WeightFormat<kQ8W>::kBlockBytes;
static_assert(kMmaUnitBytes<false> >= kMmaXWarpBytes, "the other chunks' columns are staged in the last ring positions");
template <bool kQ8W>
constexpr uint32_t kMmaMaxBlocks = kMmaWarpChunks<kQ8W> * kMmaWarps * kMmaChunkBlocks;
template <bool kQ8W>
constexpr int kMmaSmemBytes = kMmaBarrierBytes + kMmaScratchBytes + kMmaMaxBlocks<kQ8W> * kMmaCols * 4 +
                              kMmaWarps * kMmaRing<kQ8W> * kMmaUnitBytes<kQ8W>;

struct GemvMmaArgs {
  const uint8_t *vx;
  const uint8_t *vy;
  float *s;
  size_t bx, by, bs;
  uint32_t nr, nc, nb;
  uint32_t static_weights;  // weights may be fetched before the preceding kernel has finished
  uint32_t x_aligned;       // vy and by are multiples of 16: the columns can be fetched in 16-byte pieces
};

constexpr uint32_t kMmaMagicBits = 0x4B400000u;
constexpr float kMmaMagic = 12582912.0f;

// f = (float)(a * b) + 12582912, exact (see above).
__device__ __forceinline__ void mma_m16n8k32_s8(float (&f)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  uint32_t c[4];
  asm(
      "mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%10, %10, %10, %10};"
      : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(kMmaMagicBits));
#pragma unroll
  for (int i = 0; i < 4; ++i)
    f[i] = __uint_as_float(c[i]);
}

// The quant words of a Q4_0 block as the A operand: 16 * (nibble - 8) per byte.
__device__ __forceinline__ uint32_t mma_low_nibbles(uint32_t qw) { return ((qw << 4) & 0xf0f0f0f0u) ^ 0x80808080u; }
__device__ __forceinline__ uint32_t mma_high_nibbles(uint32_t qw) { return (qw & 0xf0f0f0f0u) ^ 0x80808080u; }

// The activation scale that goes with it.
template <bool kQ8W>
__device__ __forceinline__ float mma_act_scale(float d) {
  return kQ8W ? d : __fmul_rn(d, 0.0625f);
}

// ---- packed fp32x2 helpers (two IEEE round-to-nearest operations per instruction)
__device__ __forceinline__ uint64_t mma_pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void mma_unpack2(uint64_t v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t mma_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mma_mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mma_add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The order-free part of the fold of two adjacent columns of one row: Q4_0 16 * ((float)S * d_w), Q8_0
// (float)S.  (Scalar operations where a packed one would first have to copy a scale into a pair.)
template <bool kQ8W>
__device__ __forceinline__ uint64_t mma_terms2(float f_even, float f_odd, float dw) {
  if constexpr (kQ8W) {
    return mma_add2(mma_pack2(f_even, f_odd), mma_pack2(-kMmaMagic, -kMmaMagic));
  } else {
    const float neg = __fmul_rn(-kMmaMagic, dw);
    return mma_pack2(__fmaf_rn(f_even, dw, neg), __fmaf_rn(f_odd, dw, neg));
  }
}

// acc (two adjacent columns of one row) += fold of the block's MMA results with the row's weight scale dw
// and the columns' activation scales dx2 (mma_act_scale), in the format's fold order.
template <bool kQ8W>
__device__ __forceinline__ uint64_t mma_fold2(uint64_t acc, float f_even, float f_odd, float dw, uint64_t dx2) {
  const uint64_t terms = mma_terms2<kQ8W>(f_even, f_odd, dw);
  if constexpr (kQ8W)
    return mma_fma2(terms, mma_mul2(mma_pack2(dw, dw), dx2), acc);
  else
    return mma_fma2(terms, dx2, acc);
}

__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ unsigned short lds_u16(uint32_t addr) {
  unsigned short v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}

// global -> shared, 16 bytes, past the L1 cache; the second form, when not `valid`, writes zeros and reads nothing.
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_16_or_zero(uint32_t dst, const void *src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// The four bytes at shared-window address `blk` + 2 + byte_off, where blk + 2 is 4-byte aligned for odd
// blocks of a chunk and off by two for even ones (`odd` is a constant after unrolling).
__device__ __forceinline__ uint32_t mma_quant_word(uint32_t blk, uint32_t byte_off, bool odd) {
  if (odd)
    return lds_u32(blk + 2 + byte_off);
  return __funnelshift_r(lds_u32(blk + byte_off), lds_u32(blk + byte_off + 4), 16);
}

// The MMA's A operand for block `bi` of a chunk: rows at shared-window addresses `row_lo` and
// `row_hi` (the chunk's first byte in each), thread column t; also the two rows' block scales.
template <bool kQ8W>
__device__ __forceinline__ void mma_load_a_fragment(uint32_t row_lo, uint32_t row_hi, int bi, int t,
                                                    uint32_t (&afrag)[4], float &dw_lo, float &dw_hi) {
  constexpr int WB = WeightFormat<kQ8W>::kBlockBytes;
  auto load_row = [&](uint32_t row, uint32_t &k_lo, uint32_t &k_hi, float &dw) {
    const uint32_t blk = row + bi * WB;
    dw = half_bits_to_float(lds_u16(blk));
    if constexpr (kQ8W) {
      k_lo = mma_quant_word(blk, 4 * t, (bi & 1) != 0);
      k_hi = mma_quant_word(blk, 16 + 4 * t, (bi & 1) != 0);
    } else {
      const uint32_t qw = mma_quant_word(blk, 4 * t, (bi & 1) != 0);
      k_lo = mma_low_nibbles(qw);
      k_hi = mma_high_nibbles(qw);
    }
  };
  load_row(row_lo, afrag[0], afrag[2], dw_lo);
  load_row(row_hi, afrag[1], afrag[3], dw_hi);
}

// kFar: the rows of a group are too far apart for 32-bit offsets.  (An instance of its own: with both kinds of
// offsets the kernel spills, 4096 x 11008 12.4 -> 12.7 us.)
constexpr size_t kMmaFarStride = size_t{1} << 27;
template <bool kQ8W, bool kFar>
__global__ void __launch_bounds__(kMmaThreads, 1) gemv_mma_kernel(const __grid_constant__ GemvMmaArgs a) {
  constexpr int CB = kMmaChunkBlocks * WeightFormat<kQ8W>::kBlockBytes;  // chunk bytes per row: 144 or 272
  constexpr int kGroups = kMmaGroups<kQ8W>, kSlotRows = kMmaRows * kGroups, kChunks = kMmaWarpChunks<kQ8W>;
  constexpr uint32_t kRing = kMmaRing<kQ8W>, kUnitBytes = kMmaUnitBytes<kQ8W>;
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t *pfull = reinterpret_cast<uint64_t *>(smem);  // partial buffer written by all 16 warps
  uint64_t *pempty = pfull + kMmaPartialRing;            // partial buffer consumed by its combining warp
  volatile uint32_t *abort_flag = reinterpret_cast<volatile uint32_t *>(pempty + kMmaPartialRing);
  float4 *partial = reinterpret_cast<float4 *>(smem + kMmaBarrierBytes);
  float *xd = reinterpret_cast<float *>(smem + kMmaBarrierBytes + kMmaScratchBytes);  // [nb][8] scales

  const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t ring = smem_addr(xd) + kMmaMaxBlocks<kQ8W> * kMmaCols * 4 + warp * (kRing * kUnitBytes);
  // this CTA's 16-row groups; the last slot may hold one group where others hold two
  const uint32_t groups = (a.nr + kMmaRows - 1) / kMmaRows;
  const uint32_t g0 = static_cast<uint32_t>(static_cast<uint64_t>(groups) * blockIdx.x / gridDim.x);
  const uint32_t g1 = static_cast<uint32_t>(static_cast<uint64_t>(groups) * (blockIdx.x + 1) / gridDim.x);
  const uint32_t nslots = (g1 - g0 + kGroups - 1) / kGroups;
  const uint32_t rows = min(a.nr, g1 * kMmaRows) - g0 * kMmaRows;
  const uint8_t *vx = a.vx + static_cast<size_t>(g0) * kMmaRows * a.bx;
  const uint32_t nchunks = a.nb / kMmaChunkBlocks;
  const uint32_t cnt = nchunks > warp ? (nchunks - warp + kMmaWarps - 1) / kMmaWarps : 0;  // chunks per slot

  // The units of this warp, in the order of their use: slot, chunk, group.  fetch_unit requests the next one
  // into the next ring position (rows past this CTA's as zeros) as one group of copies; past the last
  // unit an empty group, so that the count of groups stays the same.  Lane `lane` copies the pieces
  // lane, lane + 32, ... of a unit.
  constexpr uint32_t kPieces = CB / 16, kUnitPieces = kMmaRows * kPieces, kCopies = (kUnitPieces + 31) / 32;
  uint32_t offset[kCopies];
#pragma unroll
  for (uint32_t p = 0; p < kCopies; ++p) {
    const uint32_t idx = p * 32 + lane, r = idx / kPieces;
    offset[p] = r * static_cast<uint32_t>(a.bx) + (idx - r * kPieces) * 16;
  }
  const size_t group_bytes = kMmaRows * a.bx;
  const uint32_t ngroups = g1 - g0;
  uint32_t fetch_slot = 0, fetch_chunk = 0, fetch_group = 0, fetch_position = 0;  // of the next request
  auto fetch_unit = [&]() {
    const uint32_t group = fetch_slot * kGroups + fetch_group;
    if (group < ngroups && cnt > 0) {
      const uint8_t *src = vx + group * group_bytes + (warp + kMmaWarps * fetch_chunk) * CB;
      const uint32_t dst = ring + fetch_position * kUnitBytes + lane * 16, left = rows - group * kMmaRows;
      if (!kFar && left >= kMmaRows) {
#pragma unroll
        for (uint32_t p = 0; p < kCopies; ++p)
          if (kUnitPieces % 32 == 0 || p * 32 + lane < kUnitPieces)
            cp_async_16(dst + p * 512, src + offset[p]);
      } else {
#pragma unroll
        for (uint32_t p = 0; p < kCopies; ++p) {
          const uint32_t r = (p * 32 + lane) / kPieces;
          const bool valid = r < left;
          const size_t at = kFar ? r * a.bx + (p * 32 + lane - r * kPieces) * 16 : offset[p];
          if (kUnitPieces % 32 == 0 || p * 32 + lane < kUnitPieces)
            cp_async_16_or_zero(dst + p * 512, src + (valid ? at : 0), valid);
        }
      }
      fetch_position = fetch_position + 1 == kRing ? 0 : fetch_position + 1;
      if (++fetch_group == kGroups || group + 1 == ngroups) {
        fetch_group = 0;
        if (++fetch_chunk == cnt) {
          fetch_chunk = 0;
          ++fetch_slot;
        }
      }
    }
    cp_async_commit();
  };
  // Where the columns of the warp's chunk u are staged, and the copies that bring them (columns past the
  // last one as zeros).
  auto column_stage = [&](uint32_t u) {
    return u == 0 ? smem_addr(partial) + warp * kMmaXWarpBytes : ring + (kRing - kChunks + u) * kUnitBytes;
  };
  auto fetch_columns = [&]() {
    const uint8_t *src = a.vy + static_cast<size_t>(warp) * kMmaXColBytes;  // chunk u is kMmaWarps * u columns' chunks further
    if (a.x_aligned) {
      constexpr uint32_t kXPieces = kMmaXColBytes / 16;  // 17 per column
#pragma unroll
      for (uint32_t p = 0; p < kMmaCols * kXPieces; p += 32) {
        const uint32_t idx = p + lane, col = idx / kXPieces;
        const uint8_t *piece = src + (col < a.nc ? col : 0) * a.by + (idx - col * kXPieces) * 16;
#pragma unroll
        for (uint32_t u = 0; u < kChunks; ++u)
          if (u < cnt && idx < kMmaCols * kXPieces)
            cp_async_16_or_zero(column_stage(u) + idx * 16, piece + u * (kMmaWarps * kMmaXColBytes), col < a.nc);
      }
    } else {
      for (uint32_t u = 0; u < cnt; ++u) {
        for (uint32_t idx = lane; idx < kMmaXWarpBytes / 2; idx += 32) {
          const uint32_t col = idx / (kMmaXColBytes / 2), h = idx - col * (kMmaXColBytes / 2);
          const uint8_t *from = src + u * (kMmaWarps * kMmaXColBytes) + col * a.by;
          const unsigned short v = col < a.nc ? reinterpret_cast<const unsigned short *>(from)[h] : static_cast<unsigned short>(0);
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(column_stage(u) + 2 * idx), "h"(v) : "memory");
        }
      }
    }
    cp_async_commit();
  };

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (!a.static_weights)
    asm volatile("griddepcontrol.wait;" ::: "memory");
  constexpr uint32_t kFirst = kRing - (kChunks - 1);  // units requested at once
#pragma unroll
  for (uint32_t n = 0; n < kFirst; ++n)
    fetch_unit();
  if (threadIdx.x == 0) {
    for (int r = 0; r < kMmaPartialRing; ++r) {
      mbar_init(&pfull[r], kMmaWarps);
      mbar_init(&pempty[r], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
  }
  if (a.static_weights)
    asm volatile("griddepcontrol.wait;" ::: "memory");
  fetch_columns();
  cp_async_wait<0>();
  __syncwarp();
  // Activation fragments: the two quant words of column g in each block (the MMA's B operand).  The scales
  // (mma_act_scale) go to shared memory, where the fold reads those of columns 2t and 2t+1 as a pair.
  uint32_t b0[kChunks][kMmaChunkBlocks], b1[kChunks][kMmaChunkBlocks];
#pragma unroll
  for (uint32_t u = 0; u < kChunks; ++u) {
    if (u < cnt) {
      const uint32_t mine = column_stage(u) + g * kMmaXColBytes;
#pragma unroll
      for (int bi = 0; bi < kMmaChunkBlocks; ++bi) {
        b0[u][bi] = mma_quant_word(mine + bi * kQ8Block, 4 * t, (bi & 1) != 0);
        b1[u][bi] = mma_quant_word(mine + bi * kQ8Block, 16 + 4 * t, (bi & 1) != 0);
      }
#pragma unroll
      for (int bi = t; bi < kMmaChunkBlocks; bi += 4)
        xd[((warp + kMmaWarps * u) * kMmaChunkBlocks + bi) * kMmaCols + g] =
            mma_act_scale<kQ8W>(half_bits_to_float(lds_u16(mine + bi * kQ8Block)));
    }
  }
  __syncthreads();  // every warp has read its staged columns: the partial ring and the last ring positions are free
#pragma unroll
  for (uint32_t n = kFirst; n < kRing; ++n)
    fetch_unit();

  bool dead = false;  // a wait expired here or in another warp: do no more work
  uint32_t position = 0;
  for (uint32_t j = 0; j < nslots && !dead; ++j) {
    // per 16-row group of the slot: rows g and g+8, columns 2t and 2t+1
    uint64_t acc_lo[kGroups] = {}, acc_hi[kGroups] = {};
    const bool single = kGroups == 1 || j * kGroups + 1 == ngroups;
#pragma unroll
    for (uint32_t u = 0; u < kChunks; ++u) {
      if (u < cnt) {
        // kRing units have been requested from this chunk's first one on
        if (single)
          cp_async_wait<kRing - 1>();
        else
          cp_async_wait<kRing - kGroups>();
        __syncwarp();  // every lane's copies have landed
        const float *dx = xd + (warp + kMmaWarps * u) * (kMmaChunkBlocks * kMmaCols) + 2 * t;
        uint32_t unit[kGroups];
#pragma unroll
        for (int q = 0; q < kGroups; ++q)
          unit[q] = ring + (position + q < kRing ? position + q : position + q - kRing) * kUnitBytes + g * CB;
        auto fold_chunk = [&](auto count) {
#pragma unroll
          for (int bi = 0; bi < kMmaChunkBlocks; ++bi) {
            const uint64_t dx2 = *reinterpret_cast<const uint64_t *>(dx + bi * kMmaCols);
#pragma unroll
            for (int q = 0; q < decltype(count)::value; ++q) {
              uint32_t afrag[4];
              float dw_lo, dw_hi, c[4];
              mma_load_a_fragment<kQ8W>(unit[q], unit[q] + 8 * CB, bi, t, afrag, dw_lo, dw_hi);
              mma_m16n8k32_s8(c, afrag, b0[u][bi], b1[u][bi]);
              acc_lo[q] = mma_fold2<kQ8W>(acc_lo[q], c[0], c[1], dw_lo, dx2);
              acc_hi[q] = mma_fold2<kQ8W>(acc_hi[q], c[2], c[3], dw_hi, dx2);
            }
          }
        };
        if (single)
          fold_chunk(std::integral_constant<int, 1>());
        else
          fold_chunk(std::integral_constant<int, kGroups>());
        position += single ? 1 : kGroups;
        position -= position >= kRing ? kRing : 0;
        __syncwarp();  // every lane has read the chunk's units
        fetch_unit();
        if (!single && kGroups == 2)
          fetch_unit();
      }
    }
    // Combine the 16 K-partials of this slot in warp order.  No CTA-wide barrier: every warp
    // drops its partial into buffer j % ring and moves on; warp j % 16 waits until all 16 have
    // arrived, adds them up and hands the buffer back.
    const uint32_t r = j % kMmaPartialRing, rphase = (j / kMmaPartialRing) & 1;
    float4 *buf = partial + r * (kMmaWarps * kMmaMaxSlotGroups * 32);
    if (!mbar_wait_bounded(&pempty[r], rphase ^ 1, abort_flag)) {
      dead = true;
      break;
    }
#pragma unroll
    for (int q = 0; q < kGroups; ++q) {
      float4 mine;
      mma_unpack2(acc_lo[q], mine.x, mine.y);
      mma_unpack2(acc_hi[q], mine.z, mine.w);
      buf[(warp * kGroups + q) * 32 + lane] = mine;
    }
    __syncwarp();
    if (lane == 0)
      mbar_arrive(&pfull[r]);
    if (warp == (j & (kMmaWarps - 1))) {
      if (!mbar_wait_bounded(&pfull[r], rphase, abort_flag)) {
        dead = true;
        break;
      }
      float4 p[kGroups];
#pragma unroll
      for (int q = 0; q < kGroups; ++q) {
        p[q] = buf[q * 32 + lane];
#pragma unroll
        for (int w = 1; w < kMmaWarps; ++w) {
          const float4 o = buf[(w * kGroups + q) * 32 + lane];
          p[q].x = __fadd_rn(p[q].x, o.x);
          p[q].y = __fadd_rn(p[q].y, o.y);
          p[q].z = __fadd_rn(p[q].z, o.z);
          p[q].w = __fadd_rn(p[q].w, o.w);
        }
      }
      __syncwarp();
      if (lane == 0)
        mbar_arrive(&pempty[r]);
      const uint32_t col = 2 * t;
#pragma unroll
      for (int q = 0; q < kGroups; ++q) {
        const uint32_t local = j * kSlotRows + q * kMmaRows + g, row = g0 * kMmaRows + local;
        if (local < rows) {
          if (col < a.nc)
            a.s[static_cast<size_t>(row) * a.bs + col] = p[q].x;
          if (col + 1 < a.nc)
            a.s[static_cast<size_t>(row) * a.bs + col + 1] = p[q].y;
        }
        if (local + 8 < rows) {
          if (col < a.nc)
            a.s[static_cast<size_t>(row + 8) * a.bs + col] = p[q].z;
          if (col + 1 < a.nc)
            a.s[static_cast<size_t>(row + 8) * a.bs + col + 1] = p[q].w;
        }
      }
    }
  }
  if (dead) {
    if (lane == 0 && *abort_flag == 0)
      raise_device_error(kDevErrBarrierTimeout);
    *abort_flag = 1;
  }
  cp_async_wait<0>();  // no copy outlives the CTA's shared memory
}

}  // namespace tcrv
