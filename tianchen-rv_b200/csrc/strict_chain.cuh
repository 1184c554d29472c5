// The sequential half of the reference's fold, for one output: a chain of one dependent operation per
// block over the block terms that other lanes have left in shared memory.
//
// What bounds it is latency: 4 cycles per block is what the dependent operation takes.  So the terms come
// in batches of kBatch groups of four blocks by 16-byte loads, and the next batch is on its way while one is
// folded.
#pragma once

#include <stdint.h>

namespace tcrv {

// acc = fma(t[b], m[b], acc) over the blocks b = 0 .. 4 * groups - 1, or, kAdd, acc = acc + t[b]; from +0.
template <bool kAdd, uint32_t kBatch>
__device__ __forceinline__ float strict_chain(const float4 *t, [[maybe_unused]] const float4 *m, uint32_t groups) {
  struct Batch {
    float4 t[kBatch], m[kAdd ? 1 : kBatch];
  };
  float acc = 0.0f;
  auto load = [&](Batch &b, uint32_t i) {
#pragma unroll
    for (uint32_t u = 0; u < kBatch; ++u) {
      b.t[u] = t[i + u];
      if constexpr (!kAdd)
        b.m[u] = m[i + u];
    }
  };
  auto fold4 = [&](const float4 &x, const float4 &y) {
    if constexpr (kAdd) {
      acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, x.x), x.y), x.z), x.w);
    } else {
      acc = __fmaf_rn(x.x, y.x, acc);
      acc = __fmaf_rn(x.y, y.y, acc);
      acc = __fmaf_rn(x.z, y.z, acc);
      acc = __fmaf_rn(x.w, y.w, acc);
    }
  };
  auto fold = [&](const Batch &b) {
#pragma unroll
    for (uint32_t u = 0; u < kBatch; ++u)
      fold4(b.t[u], b.m[kAdd ? 0 : u]);
  };
  uint32_t i = 0;
  if (groups >= 2 * kBatch) {
    Batch even, odd;
    load(even, 0);
    for (; i + 3 * kBatch <= groups; i += 2 * kBatch) {
      load(odd, i + kBatch);
      fold(even);
      load(even, i + 2 * kBatch);
      fold(odd);
    }
    fold(even);  // i + kBatch .. has not been loaded
    i += kBatch;
  }
  for (; i < groups; ++i)
    fold4(t[i], kAdd ? t[i] : m[i]);
  return acc;
}

}  // namespace tcrv
