// Prefill GEMM, Q4_0 weights x Q8_0 activations, on the 5th-generation tensor cores.
//
//   s[row*bs + col] = sum over blocks b of ((float)S_b[row,col] * d_w[row,b]) * d_x[col,b]
//   S_b[row,col]    = int32 dot of the 32 int8 weight values and 32 int8 activation values
//
// Every ggml block (32 elements of K) has its own pair of fp16 scales, so the contraction
// cannot accumulate across blocks inside the tensor core: each block gets fresh TMEM
// accumulator tiles (128 weight rows x up to 64 activation columns, K = 32), and the epilogue
// warps fold them into fp32 register accumulators with the two scales.  The fold runs in strict
// ascending block order per output element, in the fused form fma((float)S * d_w, d_x, acc).
//
// The fold on the CUDA cores, not the tensor pipe, bounds this kernel, so the tensor core is
// asked for the form that is cheapest to fold: the block sum arrives as an fp32 number.
// Weights (nibble - 8, in [-8, 7]) are stored as e4m3, where every such integer is exact; an
// int8 activation q is split as q = 16*h + l with h = q >> 4 in [-8, 7] and l = q & 15 in
// [0, 15], and the two e4m3 planes 16*h and l are both exact.  Two tcgen05.mma kind::f8f6f4 per
// block (the second accumulating) give S exactly: every product is an integer below 2^11, every
// partial sum an integer below 2^17, far inside fp32's 24-bit significand.  The fold is
// then two packed fp32 operations per pair of outputs and nothing else.  (int8 operands with
// kind::i8 need one MMA and an integer add per element.  That was 17 % slower on 128 x 128 items whose
// MMAs a single-lane branch issued; it has not been measured on the items below.)
//
// Work items.  256 weight rows x 64 columns: the two row tiles share their columns, so one broadcast
// load of activation scales serves two outputs of a thread (with 128 x 128 items those loads put 64 KB
// per block through the shared-memory pipe beside the operands: 305 us for 512 x 32000 x 4096, 640
// cycles per 128 x 128 x 32 of arithmetic that takes 276; what they still cost stands below).  8
// epilogue warps with 64 accumulators a thread: with 16 a hand-over's fixed cost is paid twice as often and
// registers run out (252 us and more instead of 231), with 4 nothing covers a warp's waits (267).
// Whole items are dealt round-robin to the CTAs; a last round that would leave more than half of
// them idle is cut into halves of 128 rows.  Few columns or rows: items of 128 rows x 32 or 16 columns, 4
// blocks to a hand-over (gemm.cu chooses).
//
// A second fold (kRepack) serves the consumer of the 16-row interleaved layouts: the same
// contraction with fma((float)S, d_w * d_x, acc) (the scales multiplied first, an exact
// product of two fp16 values) and the result stored token-major, s[col*bs + row].
//
// Operands come from a planar ("prepared") layout written by the unpack kernels: 8-bit
// matrices [rows][K] and fp32 scale matrices, all fetched with tiled TMA loads (128-byte
// swizzle for the 8-bit tiles, no multicast).  Warp roles in a CTA of 12 warps:
//   warps 0..7  epilogue: warp w reads TMEM lanes 32*(w%4).. (its weight rows) and half of the
//               columns of every accumulator tile
//   warp 8      TMA producer (one elected lane)
//   warps 9, 10 MMA issue (one elected lane each), by turns; warp 9 allocates TMEM.  Two of a block's MMAs share
//               A through the tensor core's operand buffer (without it 10 % slower on every shape), so the turns
//               are kept by the accumulators' barriers (0 to 1.5 % faster than without turns)
// Pipelines: shared-memory stages of 4 blocks each (full/empty mbarriers) and TMEM stages of
// several blocks each (full/empty mbarriers).  The epilogue warps wait on the accumulator barriers
// only: a stage's scale tiles have landed when its first accumulator has.
//
// What bounds it: per 256 x 64 block of outputs the fold's 128 packed operations a warp pair take about
// 320 cycles of a scheduler's FMA pipe (a packed FMA of three different register pairs takes 3 cycles, not
// 2), and the scale loads' 256 and the MMA operands' 128 cycles share the shared-memory pipe: without
// the scale loads 210, without MMAs 206 of 230 us (512 x 32000 x 4096, operands in L2, before the turns).  With one MMA warp,
// 16-register chunks and a single-lane producer it was 250; 512 x 11008 x 4096 92.7 -> 88.2 us, 77 x 4096 x
// 11008 41.6 -> 32.5 us (there the producer's 780 cycles per stage were the limit).  32-register chunks need
// more than the 168 registers a thread starts with; without setmaxnreg, 16-register chunks: 244 us.
// Every wait is bounded; a failed wait raises the device error word and the CTA winds down.
#pragma once

#include "tcgen05.cuh"
#include "tcrv_common.cuh"

namespace tcrv {

constexpr int kGemmTileRows = 128;      // weight rows of one MMA (M, TMEM lanes)
constexpr int kGemmStageBlocks = 4;     // ggml blocks per shared-memory stage (128 bytes of K)
constexpr int kGemmTmemCols = 512;      // all of TMEM
constexpr int kGemmEpilogueWarps = 8;  // 4 lane quarters x 2 column groups
constexpr int kGemmMmaWarps = 2;
constexpr int kGemmThreads = (kGemmEpilogueWarps + 4) * 32;  // TMA, MMA and one warp that fills the third warpgroup
// The block starts with 384 x 168 registers; the third warpgroup keeps 128 x 40 of them and the epilogue's
// two take 256 x 216 (60416 of 64512 in all).
constexpr int kGemmEpilogueRegs = 216, kGemmOtherRegs = 40;
constexpr int kGemmSplitRegs = 32 * (kGemmEpilogueWarps * kGemmEpilogueRegs + 4 * kGemmOtherRegs);
static_assert(kGemmSplitRegs <= kGemmThreads * 168, "the launch's registers");
constexpr int kGemmCtrlBytes = 1024;  // barriers, TMEM base, abort flag

// The shape of a work item: kRowTiles x 128 weight rows, kCols activation columns.
template <int kRowTiles_, int kCols_>
struct GemmShape {
  static constexpr int kRowTiles = kRowTiles_, kCols = kCols_;
  static constexpr int kRows = kRowTiles * kGemmTileRows;
  static constexpr int kCpw = kCols / (kGemmEpilogueWarps / 4);  // columns of an epilogue warp
  static constexpr int kBlockCols = kRowTiles * kCols;           // TMEM columns of one block's accumulators
  // A chunk is what a thread loads from TMEM at a time, 32 registers (16 in halves and where a stage is no more than that):
  // kChunkCols columns of its rows of kChunkBlocks blocks.
  static constexpr bool kHalf = kRowTiles == 1 && kCols == 64;
  static constexpr int kChunkRegs = kRowTiles * kCpw * kGemmStageBlocks > 32 && !kHalf ? 32 : 16;
  static constexpr int kChunkCols = kCpw < kChunkRegs / kRowTiles ? kCpw : kChunkRegs / kRowTiles;
  static constexpr int kChunkBlocks = kChunkRegs / (kRowTiles * kChunkCols);
  static constexpr int kBlockChunks = kCpw / kChunkCols;  // chunks of one block, where it has several
  static_assert(kCpw % kChunkCols == 0 && (kChunkBlocks == 1 || kBlockChunks == 1), "part of a block or whole blocks");
  __host__ __device__ static constexpr uint32_t chunk_block(uint32_t i) { return i / kBlockChunks * kChunkBlocks; }
  __host__ __device__ static constexpr uint32_t chunk_col(uint32_t i) { return i % kBlockChunks * kChunkCols; }
  // Blocks per accumulator hand-over.  A hand-over costs a barrier test, a release and a commit
  // whatever it carries, so it carries what leaves two TMEM stages.
  static constexpr int kHandover = 256 / kBlockCols < kGemmStageBlocks ? 256 / kBlockCols : kGemmStageBlocks;
  static constexpr int kChunks = kGemmStageBlocks * kBlockChunks / kChunkBlocks;  // of a shared-memory stage
  static constexpr int kHandoverChunks = kHandover * kBlockChunks / kChunkBlocks;
  static_assert(kChunks % 2 == 0 && kChunks % kHandoverChunks == 0, "two chunk buffers, whole hand-overs");
};

// What one launch works on: whole items of 256 x 64 and halves of those (kNarrow 0), or items of 128 rows x
// kNarrow columns.
template <int kNarrow>
struct GemmPlan {
  using Full = GemmShape<kNarrow != 0 ? 1 : 2, kNarrow != 0 ? kNarrow : 64>;
  using Half = GemmShape<1, kNarrow != 0 ? kNarrow : 64>;
  static constexpr uint32_t kColParts = Full::kCols / Half::kCols;
  static constexpr uint32_t kParts = Full::kRowTiles * kColParts;
  static constexpr int kTmemStages = kNarrow != 0 ? 4 : 2;
  static_assert(kTmemStages % kGemmMmaWarps == 0, "the MMA warps take turns");
  static constexpr int kTmemStageCols = kGemmTmemCols / kTmemStages;
  static_assert(Full::kBlockCols * Full::kHandover <= kTmemStageCols, "a hand-over fits a TMEM stage");
  static_assert(Half::kBlockCols * Half::kHandover <= kTmemStageCols, "a hand-over fits a TMEM stage");
  // one shared-memory stage; activations and their scales come in boxes of kBoxCols columns
  static constexpr int kBoxCols = Half::kCols;
  static constexpr int kATileBytes = kGemmTileRows * kGemmStageBlocks * kQK;  // 16384
  static constexpr int kBoxBytes = kBoxCols * kGemmStageBlocks * kQK;
  static constexpr int kPlaneBytes = Full::kCols * kGemmStageBlocks * kQK;    // one activation plane
  static constexpr int kDwTileBytes = kGemmTileRows * kGemmStageBlocks * 4;   // [128][4] fp32
  static constexpr int kDxBoxBytes = kGemmStageBlocks * kBoxCols * 4;         // [4][kBoxCols] fp32
  static constexpr int kOffB = Full::kRowTiles * kATileBytes;                 // low plane, then high plane
  static constexpr int kOffDw = kOffB + 2 * kPlaneBytes;
  static constexpr int kOffDx = kOffDw + Full::kRowTiles * kDwTileBytes;
  static constexpr int kStageBytes = (kOffDx + Full::kCols / kBoxCols * kDxBoxBytes + 1023) / 1024 * 1024;
};

// Several output copies: a finished 128-row tile is staged in shared memory (16 bytes of padding
// per row keep the staging stores conflict-free) and leaves through bulk shared->global copies of
// whole rows.
constexpr int kGemmOutRowBytes = 64 * 4 + 16;
constexpr int kGemmOutBytes = kGemmTileRows * kGemmOutRowBytes;  // 34816

template <bool kMulti, int kNarrow>
struct GemmSmem {
  static constexpr int kStages = kNarrow != 0 ? 8 : kMulti ? 3 : 4;
  static constexpr size_t kBytes = kGemmCtrlBytes + 1024 +
                                   static_cast<size_t>(kStages) * GemmPlan<kNarrow>::kStageBytes +
                                   (kMulti ? kGemmOutBytes : 0);
};

constexpr int kGemmMaxDst = 8;  // copies of the output written by the epilogue (this GPU's and its peers')

struct GemmArgs {
  // Output bases, all with row stride bs.  dst[0] is normally this GPU's buffer; further
  // entries may be peers' buffers: the N-sharded GEMM delivers each finished tile to every
  // rank's copy of the full matrix, so the all-gather overlaps the remaining tiles instead of
  // following the kernel.
  float *dst[kGemmMaxDst];
  uint32_t ndst;
  size_t bs;
  uint32_t nr, nc, nb;
  uint32_t tiles_m;     // column tiles
  uint32_t full_items;  // items [0, full_items) are whole ones
  uint32_t items;       // items [full_items, items) are halves: half j % 2 of whole item full_items + j / 2
  DeviceErrorWords errors;
};

struct GemmItem {
  uint32_t n0, m0;
  bool whole;
};

template <int kNarrow>
__device__ __forceinline__ GemmItem gemm_item(const GemmArgs &a, uint32_t idx) {
  using Plan = GemmPlan<kNarrow>;
  GemmItem it;
  it.whole = idx < a.full_items;
  const uint32_t j = it.whole ? 0u : idx - a.full_items;
  const uint32_t tile = it.whole ? idx : a.full_items + j / Plan::kParts, part = j % Plan::kParts;
  it.n0 = (tile / a.tiles_m) * Plan::Full::kRows + part / Plan::kColParts * Plan::Half::kRows;
  it.m0 = (tile % a.tiles_m) * Plan::Full::kCols + part % Plan::kColParts * Plan::Half::kCols;
  return it;
}

// ---- packed fp32x2 arithmetic (two IEEE round-to-nearest operations per instruction)
__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// 256-bit store of four packed fp32 pairs (address 32-byte aligned).
__device__ __forceinline__ void st_global_v4_b64(float *p, uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
  asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

struct PipeState {
  uint32_t stage = 0, phase = 0;
  __device__ __forceinline__ void advance(uint32_t nstages) {
    if (++stage == nstages) {
      stage = 0;
      phase ^= 1;
    }
  }
};

// shared -> global bulk copy (this GPU's or a peer's memory); both addresses 16-byte aligned,
// bytes a multiple of 16.  Completion is tracked per thread in bulk groups.
__device__ __forceinline__ void bulk_store_s2g(void *dst_gmem, const void *src_smem, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst_gmem), "r"(smem_addr(src_smem)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the sources of all this thread's bulk stores have been read (the shared memory may be rewritten)
__device__ __forceinline__ void bulk_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// A chunk (this thread's kRowTiles rows of one block, kChunkCols columns of each) folded into
// acc[.][col0 / 2 ..].
//   plain:  acc = fma((float)S * d_w, d_x, acc)      repack: acc = fma((float)S, d_w * d_x, acc)
// `dx2` holds the activation scales of this block and these columns; a scale that has been loaded
// serves the rows of all row tiles.
template <typename Shape, bool kRepack>
__device__ __forceinline__ void fold_part(const uint32_t *v, uint64_t (&acc)[Shape::kRowTiles][Shape::kCpw / 2],
                                          int col0, const float (&dw)[Shape::kRowTiles],
                                          const ulonglong2 *dx2) {
#pragma unroll
  for (int j = 0; j < Shape::kChunkCols / 4; ++j) {
    const ulonglong2 d = dx2[j];
    const int at = col0 / 2 + 2 * j;
#pragma unroll
    for (int r = 0; r < Shape::kRowTiles; ++r) {
      const uint64_t dw2 = pack_f32x2(dw[r], dw[r]);
      const uint32_t *s = v + r * Shape::kChunkCols + 4 * j;
      const uint64_t s0 = pack_f32x2(__uint_as_float(s[0]), __uint_as_float(s[1]));
      const uint64_t s1 = pack_f32x2(__uint_as_float(s[2]), __uint_as_float(s[3]));
      if constexpr (kRepack) {
        acc[r][at] = fma_f32x2(s0, mul_f32x2(dw2, d.x), acc[r][at]);
        acc[r][at + 1] = fma_f32x2(s1, mul_f32x2(dw2, d.y), acc[r][at + 1]);
      } else {
        acc[r][at] = fma_f32x2(mul_f32x2(s0, dw2), d.x, acc[r][at]);
        acc[r][at + 1] = fma_f32x2(mul_f32x2(s1, dw2), d.y, acc[r][at + 1]);
      }
    }
  }
}

struct GemmEpilogueCtx {
  uint8_t *stages;
  uint8_t *out_stage;
  uint64_t *smem_full, *smem_empty, *tmem_full, *tmem_empty, *store_bar;
  volatile uint32_t *abort_flag;
  uint32_t tmem_base;
  uint32_t store_syncs;  // syncs of the epilogue warps done so far (parity of the next one)
  uint32_t mma_warp;     // an MMA warp fills the TMEM stages of its parity
  PipeState ps, ts;
};

// Sync of the epilogue warps on an mbarrier (bounded, unlike a named barrier).
__device__ __forceinline__ bool epilogue_sync(GemmEpilogueCtx &c, int lane) {
  __syncwarp();
  if (lane == 0)
    mbar_arrive(c.store_bar);
  const bool ok = mbar_wait_bounded(c.store_bar, c.store_syncs & 1u, c.abort_flag);
  ++c.store_syncs;
  return ok;
}

// kCpw consecutive outputs of one weight row, columns m0.., to every destination (token-major: to
// the one destination's column vectors).
template <int kCpw, bool kRepack>
__device__ __forceinline__ void store_outputs(const GemmArgs &a, const uint64_t (&acc)[kCpw / 2], uint32_t row,
                                              uint32_t m0) {
  if (row >= a.nr)
    return;
  if constexpr (kRepack) {
    // for one column the 32 lanes of the warp write 32 consecutive floats
    float *dst = a.dst[0] + row;
#pragma unroll
    for (int j = 0; j < kCpw / 2; ++j) {
      float lo, hi;
      unpack_f32x2(acc[j], lo, hi);
      if (m0 + 2 * j < a.nc)
        dst[static_cast<size_t>(m0 + 2 * j) * a.bs] = lo;
      if (m0 + 2 * j + 1 < a.nc)
        dst[static_cast<size_t>(m0 + 2 * j + 1) * a.bs] = hi;
    }
    return;
  }
  bool vec = (a.bs % 4 == 0) && (m0 + kCpw <= a.nc);  // warp-uniform
  for (uint32_t d = 0; d < a.ndst; ++d)
    vec = vec && ((reinterpret_cast<uintptr_t>(a.dst[d]) & 15u) == 0);
  const size_t off = static_cast<size_t>(row) * a.bs + m0;
  for (uint32_t d = 0; d < a.ndst; ++d) {
    float *dst = a.dst[d] + off;
    if (vec && (a.bs % 8 == 0) && ((reinterpret_cast<uintptr_t>(a.dst[d]) & 31u) == 0)) {
      // 32-byte stores: every lane writes whole sectors of its row
#pragma unroll
      for (int j = 0; j < kCpw / 8; ++j)
        st_global_v4_b64(dst + 8 * j, acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
    } else if (vec) {
#pragma unroll
      for (int j = 0; j < kCpw / 4; ++j) {
        float4 o;
        unpack_f32x2(acc[2 * j], o.x, o.y);
        unpack_f32x2(acc[2 * j + 1], o.z, o.w);
        reinterpret_cast<float4 *>(dst)[j] = o;
      }
    } else {
      // ragged columns or unaligned bases: element by element
#pragma unroll
      for (int j = 0; j < kCpw / 2; ++j) {
        float lo, hi;
        unpack_f32x2(acc[j], lo, hi);
        if (m0 + 2 * j < a.nc)
          dst[2 * j] = lo;
        if (m0 + 2 * j + 1 < a.nc)
          dst[2 * j + 1] = hi;
      }
    }
  }
}

// One work item for one epilogue warp: fold all blocks, then store.  Returns false after a failed
// wait.
template <typename Plan, typename Shape, bool kMulti, bool kRepack, int kStages>
__device__ __forceinline__ bool gemm_epilogue_item(const GemmArgs &a, GemmEpilogueCtx &c, const GemmItem it, int warp,
                                                   int lane) {
  constexpr int kCpw = Shape::kCpw, kRt = Shape::kRowTiles;
  const int quarter = warp & 3, colgroup = warp >> 2;
  const int row_local = quarter * 32 + lane;
  const uint32_t nkb = (a.nb + kGemmStageBlocks - 1) / kGemmStageBlocks;
  const uint32_t tmem_lane = c.tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + colgroup * kCpw;
  constexpr int kScaleVecs = Shape::kChunkCols / 4;  // activation scales of one block of a chunk
  uint64_t acc[kRt][kCpw / 2];
#pragma unroll
  for (int r = 0; r < kRt; ++r)
#pragma unroll
    for (int j = 0; j < kCpw / 2; ++j)
      acc[r][j] = 0ull;
  uint32_t v[2][Shape::kChunkRegs];
  ulonglong2 xd[2][Shape::kChunkBlocks * kScaleVecs];
  float4 dw[kRt];
  const uint8_t *st = nullptr;
  uint32_t tmem_at = 0;
  bool ready = false;
  // Whether the next hand-over is there already, asked one chunk before the answer is needed.
  auto peek_handover = [&]() {
    PipeState next = c.ts;
    next.advance(Plan::kTmemStages);
    ready = mbar_test(&c.tmem_full[next.stage], next.phase);
  };
  auto open_handover = [&]() -> bool {
    if (!ready && !mbar_wait_bounded(&c.tmem_full[c.ts.stage], c.ts.phase, c.abort_flag))
      return false;
    tcgen05_fence_after_thread_sync();
    tmem_at = tmem_lane + c.ts.stage * Plan::kTmemStageCols;
    return true;
  };
  auto release_handover = [&]() {  // its last chunk is in registers: the TMEM stage goes back
    tcgen05_fence_before_thread_sync();
    __syncwarp();
    mbar_arrive_if(&c.tmem_empty[c.ts.stage], lane == 0);
    c.ts.advance(Plan::kTmemStages);
  };
  // The stage's scale tiles arrive with its operands (same transaction barrier), and an MMA warp
  // issues a block's MMAs only after that barrier has completed; so when an accumulator barrier of
  // this stage has completed, the scale tiles are in shared memory.  The epilogue therefore does not
  // wait on the stage's own barrier and reads no scale before its first accumulator wait of the stage.
  float4 dw_next[kRt];
  auto open_stage = [&]() {
    st = c.stages + static_cast<size_t>(c.ps.stage) * Plan::kStageBytes;
#pragma unroll
    for (int r = 0; r < kRt; ++r)
      dw_next[r] = reinterpret_cast<const float4 *>(st + Plan::kOffDw)[r * kGemmTileRows + row_local];
  };
  // All accumulators of the stage have been waited for, so its MMAs have read its operands, and this
  // warp has requested its last scales (reads that an arrive is ordered behind).
  auto close_stage = [&]() {
    __syncwarp();
    mbar_arrive_if(&c.smem_empty[c.ps.stage], lane == 0);
    c.ps.advance(kStages);
  };
  // chunk i of the stage, from TMEM into a buffer
  auto load_chunk = [&](uint32_t i, uint32_t buffer) {
#pragma unroll
    for (int b = 0; b < Shape::kChunkBlocks; ++b) {
      const uint32_t at =
          (Shape::chunk_block(i) + b) % Shape::kHandover * Shape::kBlockCols + Shape::chunk_col(i);
#pragma unroll
      for (int r = 0; r < kRt; ++r)
        tmem_ld_32x32b<Shape::kChunkCols>(tmem_at + at + r * Shape::kCols, v[buffer] + (b * kRt + r) * Shape::kChunkCols);
    }
  };
  // the activation scales of chunk i into a buffer: column c of an item is column c % kBoxCols of box
  // c / kBoxCols
  auto load_scales = [&](uint32_t i, uint32_t buffer) {
    const uint32_t col = colgroup * kCpw + Shape::chunk_col(i);
    const uint8_t *dx = st + Plan::kOffDx + col / Plan::kBoxCols * Plan::kDxBoxBytes + col % Plan::kBoxCols * 4;
#pragma unroll
    for (int b = 0; b < Shape::kChunkBlocks; ++b)
#pragma unroll
      for (int j = 0; j < kScaleVecs; ++j)
        xd[buffer][b * kScaleVecs + j] =
            reinterpret_cast<const ulonglong2 *>(dx + (Shape::chunk_block(i) + b) * (Plan::kBoxCols * 4))[j];
  };
  auto fold_chunk = [&](uint32_t i, uint32_t buffer) {
#pragma unroll
    for (int b = 0; b < Shape::kChunkBlocks; ++b) {
      const uint32_t block = Shape::chunk_block(i) + b;
      float d[kRt];
#pragma unroll
      for (int r = 0; r < kRt; ++r)
        d[r] = block == 0 ? dw[r].x : block == 1 ? dw[r].y : block == 2 ? dw[r].z : dw[r].w;
      fold_part<Shape, kRepack>(v[buffer] + b * kRt * Shape::kChunkCols, acc, Shape::chunk_col(i), d,
                                xd[buffer] + b * kScaleVecs);
    }
  };
  // The chunks are software-pipelined: while one is folded the next, and its scales, are on their
  // way, across hand-overs and stages, so neither the barrier test nor the loads' latency stands
  // between two folds.  A stage is always folded whole: blocks past the last one were read as zeros and
  // add +0 (an accumulator is never -0: it starts as +0 and x + -x is +0).
  // (A scale serves one row in a half item: twice the registers per chunk, and fetched with their own chunk
  // they leave more for the rest.  200 x 4096 x 4096 23.1 -> 21.8 us, 150 x 4096 x 11008 60.1 -> 56.1.)
  constexpr bool kLate = Shape::kHalf;
  if (!open_handover())
    return false;
  open_stage();
  load_chunk(0, 0);
  load_scales(0, 0);
  for (uint32_t kb = 0; kb < nkb; ++kb) {
#pragma unroll
    for (int r = 0; r < kRt; ++r)
      dw[r] = dw_next[r];
#pragma unroll
    for (uint32_t i = 0; i < Shape::kChunks; ++i) {
      const bool last_of_handover = (i + 1) % Shape::kHandoverChunks == 0;
      if (last_of_handover)
        peek_handover();
      if (kLate)
        load_scales(i, i & 1);
      else if (i + 1 < Shape::kChunks)
        load_scales(i + 1, (i + 1) & 1);
      tmem_ld_wait();
      if (last_of_handover)
        release_handover();
      if (i + 1 < Shape::kChunks) {
        if (last_of_handover && !open_handover())
          return false;
        load_chunk(i + 1, (i + 1) & 1);
      } else {
        close_stage();
        if (kb + 1 < nkb) {
          if (!open_handover())
            return false;
          open_stage();
          load_chunk(0, 0);
          if (!kLate)
            load_scales(0, 0);
        }
      }
      fold_chunk(i, i & 1);
    }
  }

  // ---- store: this thread owns kCpw consecutive outputs of kRt weight rows
  if constexpr (kMulti) {
    // whole item inside the matrix and every base 16-byte aligned: rows leave as bulk copies
    bool bulk = (a.bs % 4 == 0) && (it.m0 + Shape::kCols <= a.nc);
    for (uint32_t d = 0; d < a.ndst; ++d)
      bulk = bulk && ((reinterpret_cast<uintptr_t>(a.dst[d]) & 15u) == 0);
    if (bulk) {
#pragma unroll
      for (int r = 0; r < kRt; ++r) {
        // the previous tile's copies must have read the staging tile before it is rewritten
        bulk_store_wait_read();
        if (!epilogue_sync(c, lane))
          return false;
        float4 *mine = reinterpret_cast<float4 *>(c.out_stage + static_cast<size_t>(row_local) * kGemmOutRowBytes +
                                                  static_cast<size_t>(colgroup) * kCpw * 4);
#pragma unroll
        for (int j = 0; j < kCpw / 4; ++j) {
          float4 o;
          unpack_f32x2(acc[r][2 * j], o.x, o.y);
          unpack_f32x2(acc[r][2 * j + 1], o.z, o.w);
          mine[j] = o;
        }
        fence_proxy_async_smem();
        if (!epilogue_sync(c, lane))
          return false;
        // thread t sends row t%128 to destinations t/128, t/128 + 2, ...
        const uint32_t t = static_cast<uint32_t>(warp * 32 + lane);
        const uint32_t lr = t & 127u, grow = it.n0 + r * kGemmTileRows + lr;
        if (grow < a.nr) {
          const uint8_t *src = c.out_stage + static_cast<size_t>(lr) * kGemmOutRowBytes;
          for (uint32_t d = t >> 7; d < a.ndst; d += kGemmEpilogueWarps / 4)
            bulk_store_s2g(a.dst[d] + static_cast<size_t>(grow) * a.bs + it.m0, src, Shape::kCols * 4u);
        }
        bulk_store_commit();
      }
      return true;
    }
  }
#pragma unroll
  for (int r = 0; r < kRt; ++r)
    store_outputs<kCpw, kRepack>(a, acc[r], it.n0 + r * kGemmTileRows + row_local, it.m0 + colgroup * kCpw);
  return true;
}

// One work item for a (converged) MMA warp.  Returns false after a failed wait.
template <typename Plan, typename Shape, int kStages>
__device__ __forceinline__ bool gemm_mma_item(const GemmArgs &a, GemmEpilogueCtx &c, uint32_t stage_base_addr,
                                              bool leader) {
  constexpr uint32_t idesc = umma_idesc_e4m3(kGemmTileRows, Shape::kCols);
  const uint32_t nkb = (a.nb + kGemmStageBlocks - 1) / kGemmStageBlocks;
  for (uint32_t kb = 0; kb < nkb; ++kb) {
    // Operand descriptors of the stage's first block; a block further along K is 32 bytes
    // further inside the 128-byte swizzled rows, i.e. +2 in the descriptor's 16-byte
    // address field.
    const uint32_t a_addr = stage_base_addr + c.ps.stage * Plan::kStageBytes;
    const uint64_t da0 = umma_desc_k_major_sw128(a_addr);
    const uint64_t dl0 = umma_desc_k_major_sw128(a_addr + Plan::kOffB);
    const uint64_t dh0 = umma_desc_k_major_sw128(a_addr + Plan::kOffB + Plan::kPlaneBytes);
#pragma unroll
    for (uint32_t kk = 0; kk < kGemmStageBlocks; kk += Shape::kHandover) {
      if (c.ts.stage % kGemmMmaWarps == c.mma_warp) {
        // Only the operands that this warp issues from are waited for: the epilogue hands a stage back when
        // its accumulators have come, so it holds a stage for the warp that makes those and for no other.
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&c.smem_full[c.ps.stage], c.ps.phase, c.abort_flag)))
          return false;
        // The accumulators are free, and it is this warp's turn: an MMA that takes A from the operand buffer has
        // to follow the one that put it there, with no MMA of the other warp between.  So a hand-over's MMAs
        // are issued after those of the one before, whose warp is the ninth to arrive here.
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&c.tmem_empty[c.ts.stage], c.ts.phase, c.abort_flag)))
          return false;
        tcgen05_fence_after_thread_sync();
        constexpr uint64_t kStep = (kQK >> 4);  // 32 bytes in 16-byte units
        if (leader) {
#pragma unroll
          for (uint32_t h = 0; h < Shape::kHandover; ++h) {
            const uint64_t off = (kk + h) * kStep;
#pragma unroll
            for (uint32_t r = 0; r < Shape::kRowTiles; ++r) {
              const uint32_t d_tmem = c.tmem_base + c.ts.stage * Plan::kTmemStageCols +
                                      (h * Shape::kRowTiles + r) * Shape::kCols;
              const uint64_t da = da0 + off + r * (Plan::kATileBytes >> 4);
              umma_f8_first(d_tmem, da, dl0 + off, idesc);
              umma_f8_again(d_tmem, da, dh0 + off, idesc);
            }
          }
          umma_commit(&c.tmem_full[c.ts.stage]);
          tcgen05_fence_before_thread_sync();
          mbar_arrive(&c.tmem_empty[c.ts.stage + 1 == Plan::kTmemStages ? 0 : c.ts.stage + 1]);
        }
        __syncwarp();
      }
      c.ts.advance(Plan::kTmemStages);
    }
    c.ps.advance(kStages);
  }
  return true;
}

// kMulti: the result goes to several output copies (peers) through a shared-memory staging tile.
// kRepack (single destination only): scales multiplied first, token-major output.
// kNarrow: see GemmPlan.
template <bool kMulti, bool kRepack, int kNarrow>
__global__ void __launch_bounds__(kGemmThreads, 1)
    gemm_q4_0_q8_0_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                             const __grid_constant__ CUtensorMap map_xhi, const __grid_constant__ CUtensorMap map_dw,
                             const __grid_constant__ CUtensorMap map_dx, const __grid_constant__ GemmArgs a) {
  using Plan = GemmPlan<kNarrow>;
  using Full = typename Plan::Full;
  using Half = typename Plan::Half;
  constexpr int kStages = GemmSmem<kMulti, kNarrow>::kStages;
  extern __shared__ uint8_t smem_raw[];
  // control block first, then stages on a 1024-byte boundary (required by the 128B swizzle)
  GemmEpilogueCtx c;
  c.smem_full = reinterpret_cast<uint64_t *>(smem_raw);
  c.smem_empty = c.smem_full + kStages;
  c.tmem_full = c.smem_empty + kStages;
  c.tmem_empty = c.tmem_full + Plan::kTmemStages;
  uint64_t *drain_bar = c.tmem_empty + Plan::kTmemStages;
  c.store_bar = drain_bar + 1;
  uint32_t *tmem_base_slot = reinterpret_cast<uint32_t *>(c.store_bar + 1);
  c.abort_flag = tmem_base_slot + 1;
  const uint32_t stage_base_addr = (smem_addr(smem_raw) + kGemmCtrlBytes + 1023u) & ~1023u;
  c.stages = smem_raw + (stage_base_addr - smem_addr(smem_raw));
  c.out_stage = c.stages + static_cast<size_t>(kStages) * Plan::kStageBytes;  // 1024-byte aligned
  c.store_syncs = 0;

  // (shuffled, so that the compiler knows them to be the same for the whole warp)
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t nkb = (a.nb + kGemmStageBlocks - 1) / kGemmStageBlocks;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&c.smem_full[i], 1);
      mbar_init(&c.smem_empty[i], kGemmEpilogueWarps);
    }
    for (int i = 0; i < Plan::kTmemStages; ++i) {
      mbar_init(&c.tmem_full[i], 1);
      mbar_init(&c.tmem_empty[i], kGemmEpilogueWarps + 1);
    }
    mbar_init(drain_bar, kGemmMmaWarps);
    mbar_init(c.store_bar, kGemmEpilogueWarps);
    *c.abort_flag = 0;
    mbar_fence_init();
  }
  if (warp == kGemmEpilogueWarps + 1) {
    tmem_alloc(tmem_base_slot, kGemmTmemCols);
    tmem_relinquish_alloc_permit();
  }
  tcgen05_fence_before_thread_sync();
  __syncthreads();
  tcgen05_fence_after_thread_sync();
  c.tmem_base = __shfl_sync(0xffffffffu, *tmem_base_slot, 0);
  // Programmatic dependent launch: everything above touched only this CTA's shared memory and
  // TMEM, so it may overlap the tail of the preceding kernel (the activation unpack); operands
  // are read and outputs written only after that kernel has completed.
  asm volatile("griddepcontrol.wait;" ::: "memory");

  bool ok = true;
  if (warp >= kGemmEpilogueWarps) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kGemmOtherRegs));
    // In these roles the whole warp walks the loop and one elected lane issues.  Coordinates and operand
    // descriptors live in uniform registers; computed in code that the compiler knows to be converged
    // they are there already, while a single-lane branch had to move them across: 85 cycles per MMA,
    // 340 per commit and 780 for the five copies of a 128 x 32 stage.
    const bool leader = elect_one();
    if (warp == kGemmEpilogueWarps) {
      // ------------------------------ TMA producer ------------------------------
      if (leader) {
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_x);
        prefetch_tensormap(&map_xhi);
        prefetch_tensormap(&map_dw);
        prefetch_tensormap(&map_dx);
      }
      __syncwarp();
      PipeState ps;
      uint32_t issued = 0;
      for (uint32_t idx = blockIdx.x; idx < a.items && ok; idx += gridDim.x) {
        const GemmItem it = gemm_item<kNarrow>(a, idx);
        if (it.n0 >= a.nr || it.m0 >= a.nc)
          continue;
        const int n0 = static_cast<int>(it.n0), m0 = static_cast<int>(it.m0);
        const int row_tiles = it.whole ? Full::kRowTiles : Half::kRowTiles;
        const int boxes = it.whole ? Full::kCols / Plan::kBoxCols : 1;
        const uint32_t tx = row_tiles * (Plan::kATileBytes + Plan::kDwTileBytes) +
                            boxes * (2 * Plan::kBoxBytes + Plan::kDxBoxBytes);
        for (uint32_t kb = 0; kb < nkb; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait_bounded(&c.smem_empty[ps.stage], ps.phase ^ 1, c.abort_flag));
          if (!ok)
            break;
          if (leader) {
            uint8_t *st = c.stages + static_cast<size_t>(ps.stage) * Plan::kStageBytes;
            uint64_t *bar = &c.smem_full[ps.stage];
            mbar_arrive_expect_tx(bar, tx);
            const int kbyte = static_cast<int>(kb) * kGemmStageBlocks * kQK;
            const int kblk = static_cast<int>(kb) * kGemmStageBlocks;
            for (int r = 0; r < row_tiles; ++r) {
              // (a second tile that starts past the last row reads as zeros)
              tma_load_2d(st + r * Plan::kATileBytes, &map_w, kbyte, n0 + r * kGemmTileRows, bar);
              tma_load_2d(st + Plan::kOffDw + r * Plan::kDwTileBytes, &map_dw, kblk, n0 + r * kGemmTileRows, bar);
            }
            for (int b = 0; b < boxes; ++b) {
              const int mb = m0 + b * Plan::kBoxCols;
              tma_load_2d(st + Plan::kOffB + b * Plan::kBoxBytes, &map_x, kbyte, mb, bar);
              tma_load_2d(st + Plan::kOffB + Plan::kPlaneBytes + b * Plan::kBoxBytes, &map_xhi, kbyte, mb, bar);
              tma_load_2d(st + Plan::kOffDx + b * Plan::kDxBoxBytes, &map_dx, mb, kblk, bar);
            }
          }
          __syncwarp();
          ps.advance(kStages);
          ++issued;
        }
      }
      if (!ok && leader) {
        *c.abort_flag = 1;
        raise_device_error(a.errors, kDevErrBarrierTimeout);
      }
      __syncwarp();
      if (*c.abort_flag != 0) {
        // winding down after a failed wait: let this CTA's own copies land before it exits
        const uint32_t first = issued > kStages ? issued - kStages : 0;
        for (uint32_t i = first; i < issued; ++i)
          (void)mbar_wait_bounded(&c.smem_full[i % kStages], (i / kStages) & 1, nullptr);
      }
    } else if (warp <= kGemmEpilogueWarps + kGemmMmaWarps) {
      // ------------------------------ MMA issuers ------------------------------
      // Two warps take turns at the TMEM stages: one warp's wait, wait, issue and commit for a hand-over
      // (640 cycles) is longer than what eight MMAs take (240 to 300).
      c.mma_warp = static_cast<uint32_t>(warp - kGemmEpilogueWarps - 1);
      mbar_arrive_if(&c.tmem_empty[0], c.mma_warp == 0 && leader);  // the first turn
      for (uint32_t idx = blockIdx.x; idx < a.items && ok; idx += gridDim.x) {
        const GemmItem it = gemm_item<kNarrow>(a, idx);
        if (it.n0 >= a.nr || it.m0 >= a.nc)
          continue;
        ok = it.whole ? gemm_mma_item<Plan, Full, kStages>(a, c, stage_base_addr, leader)
                      : gemm_mma_item<Plan, Half, kStages>(a, c, stage_base_addr, leader);
      }
      if (!ok && leader) {
        *c.abort_flag = 1;
        raise_device_error(a.errors, kDevErrBarrierTimeout);
      }
      // every MMA issued above must have finished before TMEM is released
      if (leader)
        umma_commit(drain_bar);
      __syncwarp();
      (void)mbar_wait_bounded(drain_bar, 0, nullptr);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kGemmEpilogueRegs));
    for (int i = 0; i < Plan::kTmemStages; ++i)  // all TMEM stages are free
      mbar_arrive_if(&c.tmem_empty[i], lane == 0);
    // ------------------------------ epilogue warps ------------------------------
    for (uint32_t idx = blockIdx.x; idx < a.items && ok; idx += gridDim.x) {
      const GemmItem it = gemm_item<kNarrow>(a, idx);
      if (it.n0 >= a.nr || it.m0 >= a.nc)
        continue;
      if (it.whole)
        ok = gemm_epilogue_item<Plan, Full, kMulti, kRepack, kStages>(a, c, it, warp, lane);
      else
        ok = gemm_epilogue_item<Plan, Half, kMulti, kRepack, kStages>(a, c, it, warp, lane);
    }
    if (kMulti)
      bulk_store_wait_all();  // the staging tile must outlive the copies that read it
    if (!ok && lane == 0) {
      *c.abort_flag = 1;
      raise_device_error(a.errors, kDevErrBarrierTimeout);
    }
  }

  tcgen05_fence_before_thread_sync();
  __syncthreads();
  if (warp == kGemmEpilogueWarps + 1) {
    tcgen05_fence_after_thread_sync();
    tmem_dealloc(c.tmem_base, kGemmTmemCols);
  }
}

}  // namespace tcrv
