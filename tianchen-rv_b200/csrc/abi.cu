// extern "C" surface of the provider: argument validation, status codes, error text and the
// device-side error word.  Every function here takes device pointers and launches on the
// caller's stream; none allocates, and none has a CPU fallback.
#include <atomic>
#include <cstring>
#include <stdio.h>
#include <string.h>

#include "launchers.h"
#include "tcrv_common.cuh"

namespace tcrv {

__device__ int g_device_error = 0;
__device__ int *g_host_error_mirror = nullptr;

namespace {
thread_local char t_error_text[256] = "";
}

int record_cuda_error(cudaError_t err, const char *what) {
  snprintf(t_error_text, sizeof t_error_text, "%s: %s (%s)", what, cudaGetErrorName(err), cudaGetErrorString(err));
  (void)cudaGetLastError();  // clear the sticky-free error state
  return TCRV_CUDA_ERR_CUDA;
}

int sm_count() {
  static std::atomic<int> cached[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return kNumSMsB200;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = kNumSMsB200;
    cached[dev] = n;
  }
  return cached[dev];
}

int device_error_words(DeviceErrorWords *out) {
  static std::atomic<int *> word[64];
  static std::atomic<int **> mirror[64];
  int dev = 0;
  TCRV_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64)
    return TCRV_CUDA_ERR_UNSUPPORTED;
  if (mirror[dev].load() == nullptr) {  // host threads may race to fill these with the same values
    void *w = nullptr, *m = nullptr;
    TCRV_CUDA_TRY(cudaGetSymbolAddress(&w, g_device_error));
    TCRV_CUDA_TRY(cudaGetSymbolAddress(&m, g_host_error_mirror));
    word[dev] = static_cast<int *>(w);
    mirror[dev] = static_cast<int **>(m);
  }
  out->word = word[dev];
  out->mirror = mirror[dev];
  return TCRV_CUDA_OK;
}

namespace {

inline cudaStream_t as_stream(tcrv_cuda_stream s) { return static_cast<cudaStream_t>(s); }

// Shared checks of the GEMV/GEMM-shaped entry points.
int check_matrix_args(size_t n, const void *out, const void *vx, const void *vy, size_t by, size_t nr, size_t nc,
                      size_t bx, size_t out_stride, size_t weight_block_bytes) {
  if (n % TCRV_QK != 0)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nr == 0 || nc == 0)
    return TCRV_CUDA_OK;
  if (!out || !vx || !vy)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  const size_t nb = n / TCRV_QK;
  if (nb > 0xffffffffull / 64 || nr > 0xffffffffull || nc > 0xffffffffull)
    return TCRV_CUDA_ERR_UNSUPPORTED;
  if (nr > 1 && bx < nb * weight_block_bytes)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nc > 1 && by < nb * TCRV_Q8_0_BLOCK_BYTES)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nr > 1 && out_stride < nc)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return TCRV_CUDA_OK;
}

}  // namespace
}  // namespace tcrv

using namespace tcrv;

extern "C" {

const char *tcrv_cuda_status_string(int status) {
  switch (status) {
    case TCRV_CUDA_OK:
      return "ok";
    case TCRV_CUDA_ERR_INVALID_ARGUMENT:
      return "invalid argument";
    case TCRV_CUDA_ERR_UNSUPPORTED:
      return "unsupported facts";
    case TCRV_CUDA_ERR_CUDA:
      return "CUDA runtime error";
    case TCRV_CUDA_ERR_DEVICE_TIMEOUT:
      return "device-side wait timed out";
    case TCRV_CUDA_ERR_WORKSPACE:
      return "workspace missing or too small";
    default:
      return "unknown status";
  }
}

const char *tcrv_cuda_last_error_text(void) { return t_error_text; }

int tcrv_cuda_abi_version(void) { return 1; }

int tcrv_cuda_check_device_errors(tcrv_cuda_stream stream) {
  TCRV_CUDA_TRY(cudaStreamSynchronize(as_stream(stream)));
  int word = 0;
  TCRV_CUDA_TRY(cudaMemcpyFromSymbol(&word, g_device_error, sizeof word));
  if (word != 0) {
    const int zero = 0;
    TCRV_CUDA_TRY(cudaMemcpyToSymbol(g_device_error, &zero, sizeof zero));
    host_error_mirror_reset();
    return TCRV_CUDA_ERR_DEVICE_TIMEOUT;
  }
  return TCRV_CUDA_OK;
}

int tcrv_cuda_add_f32(const float *lhs, const float *rhs, float *out, size_t n, tcrv_cuda_stream stream) {
  if (n != 0 && (!lhs || !rhs || !out))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_add_f32(lhs, rhs, out, n, as_stream(stream));
}

int tcrv_cuda_add_i32(const int32_t *lhs, const int32_t *rhs, int32_t *out, size_t n, tcrv_cuda_stream stream) {
  if (n != 0 && (!lhs || !rhs || !out))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_add_i32(lhs, rhs, out, n, as_stream(stream));
}

int tcrv_cuda_dequantize_i32_f32(const int32_t *lhs, float scale, float *out, size_t n, tcrv_cuda_stream stream) {
  if (n != 0 && (!lhs || !out))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_dequantize_i32_f32(lhs, scale, out, n, as_stream(stream));
}

int tcrv_cuda_dequantize_row_q8_0(const uint8_t *vx, float *y, size_t n, tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || (n != 0 && (!vx || !y)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_dequantize_row_q8_0(vx, y, n, as_stream(stream));
}

int tcrv_cuda_dequantize_row_q4_0(const uint8_t *vx, float *y, size_t n, tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || (n != 0 && (!vx || !y)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_dequantize_row_q4_0(vx, y, n, as_stream(stream));
}

int tcrv_cuda_quantize_row_q8_0(size_t n, const float *x, uint8_t *vy, tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || (n != 0 && (!x || !vy)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_quantize_row_q8_0(n, x, vy, as_stream(stream));
}

int tcrv_cuda_quantize_row_q4_0(size_t n, const float *x, uint8_t *vx, tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || (n != 0 && (!x || !vx)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_quantize_row_q4_0(n, x, vx, as_stream(stream));
}

int tcrv_cuda_vec_dot_q4_0_q8_0(size_t n, float *s, size_t bs, const uint8_t *vx, size_t bx, const uint8_t *vy,
                                size_t by, int32_t nrc, tcrv_cuda_stream stream) {
  (void)bs;
  (void)bx;
  (void)by;
  (void)nrc;  // as in the reference kernel, only n, s, vx, vy are consumed
  if (n % TCRV_QK != 0 || !s || (n != 0 && (!vx || !vy)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_gemv<false>(n, s, vx, vy, 0, 1, 1, 0, 1, TCRV_CUDA_FLAG_STRICT_ORDER, as_stream(stream));
}

int tcrv_cuda_vec_dot_q8_0_q8_0(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || !s || (n != 0 && (!vx || !vy)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_gemv<true>(n, s, vx, vy, 0, 1, 1, 0, 1, TCRV_CUDA_FLAG_STRICT_ORDER, as_stream(stream));
}

int tcrv_cuda_gemv_q4_0_q8_0(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t by, size_t nr,
                             size_t nc, size_t bx, size_t bs, unsigned flags, tcrv_cuda_stream stream) {
  const int st = check_matrix_args(n, s, vx, vy, by, nr, nc, bx, bs, TCRV_Q4_0_BLOCK_BYTES);
  if (st != TCRV_CUDA_OK)
    return st;
  return launch_gemv<false>(n, s, vx, vy, by, nr, nc, bx, bs, flags, as_stream(stream));
}

int tcrv_cuda_gemv_q8_0_q8_0(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t by, size_t nr,
                             size_t nc, size_t bx, size_t bs, unsigned flags, tcrv_cuda_stream stream) {
  const int st = check_matrix_args(n, s, vx, vy, by, nr, nc, bx, bs, TCRV_Q8_0_BLOCK_BYTES);
  if (st != TCRV_CUDA_OK)
    return st;
  return launch_gemv<true>(n, s, vx, vy, by, nr, nc, bx, bs, flags, as_stream(stream));
}

namespace {
int gemv_group(bool q8_weights, const tcrv_cuda_gemv_call *calls, size_t count, unsigned flags, tcrv_cuda_stream stream) {
  if (count == 0)
    return TCRV_CUDA_OK;
  if (!calls || count > 16)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  GemvGroupItem items[16];
  for (size_t i = 0; i < count; ++i) {
    const tcrv_cuda_gemv_call &c = calls[i];
    const int st = check_matrix_args(c.n, c.s, c.vx, c.vy, c.by, c.nr, c.nc, c.bx, c.bs,
                                     q8_weights ? TCRV_Q8_0_BLOCK_BYTES : TCRV_Q4_0_BLOCK_BYTES);
    if (st != TCRV_CUDA_OK)
      return st;
    items[i] = GemvGroupItem{c.n, c.s, c.vx, c.vy, c.by, c.nr, c.nc, c.bx, c.bs, flags};
  }
  const int st = launch_gemv_group(q8_weights, items, count, as_stream(stream));
  if (st != TCRV_CUDA_ERR_UNSUPPORTED)
    return st;
  // not one launch (several columns, tuning bits, operands the bulk copies refuse): one after the other
  for (size_t i = 0; i < count; ++i) {
    const GemvGroupItem &g = items[i];
    const int each = q8_weights ? launch_gemv<true>(g.n, g.s, g.vx, g.vy, g.by, g.nr, g.nc, g.bx, g.bs, g.flags, as_stream(stream))
                                : launch_gemv<false>(g.n, g.s, g.vx, g.vy, g.by, g.nr, g.nc, g.bx, g.bs, g.flags, as_stream(stream));
    if (each != TCRV_CUDA_OK)
      return each;
  }
  return TCRV_CUDA_OK;
}
}  // namespace

int tcrv_cuda_gemv_group_q4_0_q8_0(const tcrv_cuda_gemv_call *calls, size_t count, unsigned flags,
                                   tcrv_cuda_stream stream) {
  return gemv_group(false, calls, count, flags, stream);
}

int tcrv_cuda_gemv_group_q8_0_q8_0(const tcrv_cuda_gemv_call *calls, size_t count, unsigned flags,
                                   tcrv_cuda_stream stream) {
  return gemv_group(true, calls, count, flags, stream);
}

int tcrv_cuda_gemv_fold_order(int q8_weights, size_t n, size_t nc, const void *vx, size_t bx, const void *vy,
                              size_t by, unsigned flags) {
  return q8_weights ? gemv_fold_order<true>(n, nc, vx, bx, vy, by, flags)
                    : gemv_fold_order<false>(n, nc, vx, bx, vy, by, flags);
}

int tcrv_cuda_block_sums_q4_0_q8_0(size_t n, int32_t *sumi, const uint8_t *vx, const uint8_t *vy, size_t by,
                                   size_t nr, size_t nc, size_t bx, tcrv_cuda_stream stream) {
  const int st = check_matrix_args(n, sumi, vx, vy, by, nr, nc, bx, nc, TCRV_Q4_0_BLOCK_BYTES);
  if (st != TCRV_CUDA_OK)
    return st;
  return launch_block_sums<false>(n, sumi, vx, vy, by, nr, nc, bx, as_stream(stream));
}

int tcrv_cuda_block_sums_q8_0_q8_0(size_t n, int32_t *sumi, const uint8_t *vx, const uint8_t *vy, size_t by,
                                   size_t nr, size_t nc, size_t bx, tcrv_cuda_stream stream) {
  const int st = check_matrix_args(n, sumi, vx, vy, by, nr, nc, bx, nc, TCRV_Q8_0_BLOCK_BYTES);
  if (st != TCRV_CUDA_OK)
    return st;
  return launch_block_sums<true>(n, sumi, vx, vy, by, nr, nc, bx, as_stream(stream));
}

size_t tcrv_cuda_gemm_weights_bytes(size_t n, size_t nr) { return gemm_weights_bytes(n, nr); }

size_t tcrv_cuda_gemm_acts_workspace_bytes(size_t n, size_t nc) { return gemm_acts_bytes(n, nc); }

size_t tcrv_cuda_gemm_workspace_bytes(size_t n, size_t nr, size_t nc) {
  return gemm_weights_bytes(n, nr) + gemm_acts_bytes(n, nc);
}

int tcrv_cuda_gemm_prepare_weights_q4_0(size_t n, const uint8_t *vx, size_t bx, size_t nr, void *prepared,
                                        size_t prepared_bytes, tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || (nr != 0 && n != 0 && (!vx || !prepared)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nr > 1 && bx < n / TCRV_QK * TCRV_Q4_0_BLOCK_BYTES)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (prepared_bytes < gemm_weights_bytes(n, nr) || reinterpret_cast<uintptr_t>(prepared) % 256 != 0)
    return TCRV_CUDA_ERR_WORKSPACE;
  return launch_gemm_prepare_weights_q4_0(n, vx, bx, nr, static_cast<uint8_t *>(prepared), as_stream(stream));
}

int tcrv_cuda_gemm_q4_0_q8_0_prepared(size_t n, float *s, const void *prepared_weights, const uint8_t *vy,
                                      size_t by, size_t nr, size_t nc, size_t bs, void *workspace,
                                      size_t workspace_bytes, unsigned flags, tcrv_cuda_stream stream) {
  (void)flags;  // the GEMM always folds in strict ascending block order
  const int st = check_matrix_args(n, s, prepared_weights, vy, by, nr, nc, static_cast<size_t>(-1), bs, 0);
  if (st != TCRV_CUDA_OK)
    return st;
  if (nr == 0 || nc == 0 || n == 0) {
    if (n == 0)
      for (size_t r = 0; r < nr; ++r)
        TCRV_CUDA_TRY(cudaMemsetAsync(s + r * bs, 0, nc * sizeof(float), as_stream(stream)));
    return TCRV_CUDA_OK;
  }
  if (!workspace || workspace_bytes < gemm_acts_bytes(n, nc) || reinterpret_cast<uintptr_t>(workspace) % 256 != 0 ||
      reinterpret_cast<uintptr_t>(prepared_weights) % 256 != 0)
    return TCRV_CUDA_ERR_WORKSPACE;
  uint8_t *acts = static_cast<uint8_t *>(workspace);
  int rc = launch_gemm_prepare_acts_q8_0(n, vy, by, nc, acts, as_stream(stream));
  if (rc != TCRV_CUDA_OK)
    return rc;
  return launch_gemm_prepared(n, s, static_cast<const uint8_t *>(prepared_weights), acts, nr, nc, bs,
                              as_stream(stream));
}

int tcrv_cuda_gemm_q4_0_q8_0_prepared_multi(size_t n, float *const *dst, size_t ndst, const void *prepared_weights,
                                            const uint8_t *vy, size_t by, size_t nr, size_t nc, size_t bs,
                                            void *workspace, size_t workspace_bytes, unsigned flags,
                                            tcrv_cuda_stream stream) {
  (void)flags;  // the GEMM always folds in strict ascending block order
  if (!dst || ndst == 0 || ndst > 8)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  for (size_t d = 0; d < ndst; ++d) {
    const int st = check_matrix_args(n, dst[d], prepared_weights, vy, by, nr, nc, static_cast<size_t>(-1), bs, 0);
    if (st != TCRV_CUDA_OK)
      return st;
  }
  if (nr == 0 || nc == 0 || n == 0) {
    if (n == 0)
      for (size_t d = 0; d < ndst; ++d)
        for (size_t r = 0; r < nr; ++r)
          TCRV_CUDA_TRY(cudaMemsetAsync(dst[d] + r * bs, 0, nc * sizeof(float), as_stream(stream)));
    return TCRV_CUDA_OK;
  }
  if (!workspace || workspace_bytes < gemm_acts_bytes(n, nc) || reinterpret_cast<uintptr_t>(workspace) % 256 != 0 ||
      reinterpret_cast<uintptr_t>(prepared_weights) % 256 != 0)
    return TCRV_CUDA_ERR_WORKSPACE;
  uint8_t *acts = static_cast<uint8_t *>(workspace);
  int rc = launch_gemm_prepare_acts_q8_0(n, vy, by, nc, acts, as_stream(stream));
  if (rc != TCRV_CUDA_OK)
    return rc;
  return launch_gemm_prepared_multi(n, dst, ndst, static_cast<const uint8_t *>(prepared_weights), acts, nr, nc, bs,
                                    as_stream(stream));
}

int tcrv_cuda_vec_scale_f32(size_t n, float *y, float v, tcrv_cuda_stream stream) {
  if (n != 0 && !y)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_vec_scale_f32(n, y, v, as_stream(stream));
}

int tcrv_cuda_vec_silu_f32(size_t n, const float *x, float *y, tcrv_cuda_stream stream) {
  if (n != 0 && (!x || !y))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_vec_silu_f32(n, x, y, as_stream(stream));
}

int tcrv_cuda_rms_norm_f32(size_t ne00, const float *x, float *y, float eps, size_t nrows, size_t x_stride,
                           size_t y_stride, tcrv_cuda_stream stream) {
  if (ne00 == 0 || nrows == 0)
    return TCRV_CUDA_OK;
  if (!x || !y || (nrows > 1 && (x_stride < ne00 || y_stride < ne00)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_rms_norm_f32(ne00, x, y, eps, nrows, x_stride, y_stride, TCRV_CUDA_FLAG_NONE, as_stream(stream));
}

int tcrv_cuda_rms_norm_f32_flags(size_t ne00, const float *x, float *y, float eps, size_t nrows, size_t x_stride,
                                 size_t y_stride, unsigned flags, tcrv_cuda_stream stream) {
  if (ne00 == 0 || nrows == 0)
    return TCRV_CUDA_OK;
  if (!x || !y || (nrows > 1 && (x_stride < ne00 || y_stride < ne00)) || (flags & ~TCRV_CUDA_FLAG_STRICT_ORDER) != 0)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_rms_norm_f32(ne00, x, y, eps, nrows, x_stride, y_stride, flags, as_stream(stream));
}

int tcrv_cuda_vec_soft_max_f32(size_t n, float *y, const float *x, float max, double *sum, tcrv_cuda_stream stream) {
  if (n != 0 && (!x || !y))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_vec_soft_max_f32(n, y, x, max, sum, as_stream(stream));
}

int tcrv_cuda_rope_cache_f32(size_t n_dims, float theta_base, float theta_scale, float *cache, float *thetas,
                             tcrv_cuda_stream stream) {
  if (n_dims % 2 != 0 || n_dims > 0xffffffffull)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (n_dims != 0 && (!cache || reinterpret_cast<uintptr_t>(cache) % 8 != 0))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_rope_cache_f32(n_dims, theta_base, theta_scale, cache, thetas, as_stream(stream));
}

int tcrv_cuda_rope_apply_f32(size_t n_dims, const float *x, float *y, const float *cache, size_t nrows, size_t x_stride,
                             size_t y_stride, tcrv_cuda_stream stream) {
  if (n_dims % 2 != 0 || n_dims > 0xffffffffull)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (n_dims == 0 || nrows == 0)
    return TCRV_CUDA_OK;
  if (!x || !y || !cache || reinterpret_cast<uintptr_t>(cache) % 8 != 0 ||
      (nrows > 1 && (x_stride < n_dims || y_stride < n_dims)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_rope_apply_f32(n_dims, x, y, cache, nrows, x_stride, y_stride, as_stream(stream));
}

int tcrv_cuda_pack_q4_0_to_q4_0x16(size_t nblocks, const uint8_t *src, uint8_t *dst, tcrv_cuda_stream stream) {
  if (nblocks != 0 && (!src || !dst || src == dst))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_pack_q4_0_to_q4_0x16(nblocks, src, dst, as_stream(stream));
}

int tcrv_cuda_unpack_q4_0x16_to_q4_0(size_t nblocks, const uint8_t *src, uint8_t *dst, tcrv_cuda_stream stream) {
  if (nblocks != 0 && (!src || !dst || src == dst))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_unpack_q4_0x16_to_q4_0(nblocks, src, dst, as_stream(stream));
}

namespace {
int check_sibling_args(int format, size_t n, const void *out, const void *vx, const void *vy, size_t by, size_t nr,
                       size_t nc, size_t bx, size_t out_stride) {
  size_t wb = 0, ab = 0;
  if (sibling_block_bytes(format, &wb, &ab) != TCRV_CUDA_OK || n % TCRV_QK != 0)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nr == 0 || nc == 0)
    return TCRV_CUDA_OK;
  if (!out || !vx || !vy)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  const size_t nb = n / TCRV_QK;
  if (nb > 0xffffffffull / 64 || nr > 0xffffffffull || nc > 0xffffffffull)
    return TCRV_CUDA_ERR_UNSUPPORTED;
  if ((nr > 1 && bx < nb * wb) || (nc > 1 && by < nb * ab) || (nr > 1 && out_stride < nc))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return TCRV_CUDA_OK;
}
}  // namespace

int tcrv_cuda_sibling_dot_rows(int format, size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t by,
                               size_t nr, size_t nc, size_t bx, size_t bs, tcrv_cuda_stream stream) {
  const int st = check_sibling_args(format, n, s, vx, vy, by, nr, nc, bx, bs);
  if (st != TCRV_CUDA_OK)
    return st;
  return launch_sibling_dot(format, n, s, nullptr, vx, vy, by, nr, nc, bx, bs, as_stream(stream));
}

int tcrv_cuda_sibling_block_sums(int format, size_t n, int32_t *sumi, const uint8_t *vx, const uint8_t *vy, size_t by,
                                 size_t nr, size_t nc, size_t bx, tcrv_cuda_stream stream) {
  const int st = check_sibling_args(format, n, sumi, vx, vy, by, nr, nc, bx, nc);
  if (st != TCRV_CUDA_OK)
    return st;
  return launch_sibling_dot(format, n, nullptr, sumi, vx, vy, by, nr, nc, bx, nc, as_stream(stream));
}

int tcrv_cuda_vec_dot_q4_1_q8_1(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, tcrv_cuda_stream stream) {
  return tcrv_cuda_sibling_dot_rows(TCRV_CUDA_FORMAT_Q4_1_Q8_1, n, s, vx, vy, 0, 1, 1, 0, 1, stream);
}

int tcrv_cuda_vec_dot_q5_0_q8_0(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, tcrv_cuda_stream stream) {
  return tcrv_cuda_sibling_dot_rows(TCRV_CUDA_FORMAT_Q5_0_Q8_0, n, s, vx, vy, 0, 1, 1, 0, 1, stream);
}

int tcrv_cuda_vec_dot_q5_1_q8_1(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, tcrv_cuda_stream stream) {
  return tcrv_cuda_sibling_dot_rows(TCRV_CUDA_FORMAT_Q5_1_Q8_1, n, s, vx, vy, 0, 1, 1, 0, 1, stream);
}

size_t tcrv_cuda_repack_gemv_parts(size_t n) { return repack_gemv_parts(n); }

namespace {
int check_repack_gemv_args(size_t n, const float *s, const uint8_t *vx, const uint8_t *vy, size_t nc) {
  if (n % TCRV_QK != 0 || nc % 16 != 0)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nc != 0 && (!s || (reinterpret_cast<uintptr_t>(s) & 3u) != 0))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nc != 0 && n != 0 && (!vx || !vy))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return TCRV_CUDA_OK;
}
}  // namespace

int tcrv_cuda_repack_gemv_q4_0_q8_0(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t nc,
                                    unsigned flags, tcrv_cuda_stream stream) {
  const int st = check_repack_gemv_args(n, s, vx, vy, nc);
  if (st != TCRV_CUDA_OK)
    return st;
  if (n == 0 && nc != 0)
    TCRV_CUDA_TRY(cudaMemsetAsync(s, 0, nc * sizeof(float), as_stream(stream)));  // empty sums
  return launch_repack_gemv_q4_0_q8_0(n, s, vx, vy, nc, flags, as_stream(stream));
}

int tcrv_cuda_repack_gemv_q8_0_q8_0(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t nc,
                                    unsigned flags, tcrv_cuda_stream stream) {
  const int st = check_repack_gemv_args(n, s, vx, vy, nc);
  if (st != TCRV_CUDA_OK)
    return st;
  if (n == 0 && nc != 0)
    TCRV_CUDA_TRY(cudaMemsetAsync(s, 0, nc * sizeof(float), as_stream(stream)));
  return launch_repack_gemv_q8_0_q8_0(n, s, vx, vy, nc, flags, as_stream(stream));
}

size_t tcrv_cuda_repack_gemm_workspace_bytes(size_t n, size_t nr, size_t nc) {
  return gemm_weights_bytes(n, nc) + gemm_acts_bytes(n, nr);
}

int tcrv_cuda_repack_gemm_prepare_weights_q4_0x16(size_t n, const uint8_t *vx, size_t nc, void *prepared,
                                                  size_t prepared_bytes, tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || nc % 16 != 0 || (nc != 0 && n != 0 && (!vx || !prepared)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (prepared_bytes < gemm_weights_bytes(n, nc) || reinterpret_cast<uintptr_t>(prepared) % 256 != 0)
    return TCRV_CUDA_ERR_WORKSPACE;
  return launch_repack_gemm_prepare_weights_q4_0x16(n, vx, nc, static_cast<uint8_t *>(prepared), as_stream(stream));
}

int tcrv_cuda_repack_gemm_q4_0_q8_0_prepared(size_t n, float *s, const void *prepared_weights, const uint8_t *vy,
                                             size_t nr, size_t nc, size_t bs, void *workspace, size_t workspace_bytes,
                                             tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || nr % 4 != 0 || nc % 16 != 0 || (nr > 1 && bs < nc))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nr != 0 && nc != 0 && (!s || (reinterpret_cast<uintptr_t>(s) & 3u) != 0))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nr == 0 || nc == 0)
    return TCRV_CUDA_OK;
  if (n == 0) {
    for (size_t r = 0; r < nr; ++r)
      TCRV_CUDA_TRY(cudaMemsetAsync(s + r * bs, 0, nc * sizeof(float), as_stream(stream)));
    return TCRV_CUDA_OK;
  }
  if (!prepared_weights || !vy)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (!workspace || workspace_bytes < gemm_acts_bytes(n, nr) || reinterpret_cast<uintptr_t>(workspace) % 256 != 0 ||
      reinterpret_cast<uintptr_t>(prepared_weights) % 256 != 0)
    return TCRV_CUDA_ERR_WORKSPACE;
  return launch_repack_gemm_prepared(n, s, static_cast<const uint8_t *>(prepared_weights), vy, nr, nc, bs,
                                     static_cast<uint8_t *>(workspace), as_stream(stream));
}

int tcrv_cuda_repack_gemm_q4_0_q8_0(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t nr, size_t nc,
                                    size_t bs, void *workspace, size_t workspace_bytes, tcrv_cuda_stream stream) {
  if (n % TCRV_QK != 0 || nr % 4 != 0 || nc % 16 != 0)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  if (nr == 0 || nc == 0 || n == 0)
    return tcrv_cuda_repack_gemm_q4_0_q8_0_prepared(n, s, nullptr, vy, nr, nc, bs, nullptr, 0, stream);
  if (!vx)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  const size_t wbytes = gemm_weights_bytes(n, nc);
  if (!workspace || workspace_bytes < wbytes + gemm_acts_bytes(n, nr) ||
      reinterpret_cast<uintptr_t>(workspace) % 256 != 0)
    return TCRV_CUDA_ERR_WORKSPACE;
  uint8_t *ws = static_cast<uint8_t *>(workspace);
  const int st = launch_repack_gemm_prepare_weights_q4_0x16(n, vx, nc, ws, as_stream(stream));
  if (st != TCRV_CUDA_OK)
    return st;
  return tcrv_cuda_repack_gemm_q4_0_q8_0_prepared(n, s, ws, vy, nr, nc, bs, ws + wbytes, workspace_bytes - wbytes,
                                                  stream);
}

int tcrv_cuda_q4_0_q8_0_integer_core(const int8_t *w, const int8_t *qlo, const int8_t *qhi, const int32_t *acc,
                                     int32_t *out, size_t n, tcrv_cuda_stream stream) {
  if (!acc || !out || (n != 0 && (!w || !qlo || !qhi)))
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  return launch_q4_0_q8_0_integer_core(w, qlo, qhi, acc, out, n, as_stream(stream));
}

int tcrv_cuda_peer_alloc(size_t bytes, void **ptr) {
  if (!ptr || bytes == 0)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  TCRV_CUDA_TRY(cudaMalloc(ptr, bytes));
  return TCRV_CUDA_OK;
}

int tcrv_cuda_peer_free(void *ptr) {
  if (ptr)
    TCRV_CUDA_TRY(cudaFree(ptr));
  return TCRV_CUDA_OK;
}

int tcrv_cuda_peer_export(const void *ptr, unsigned char *handle) {
  static_assert(sizeof(cudaIpcMemHandle_t) == TCRV_CUDA_PEER_HANDLE_BYTES, "handle size");
  if (!ptr || !handle)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  cudaIpcMemHandle_t h;
  TCRV_CUDA_TRY(cudaIpcGetMemHandle(&h, const_cast<void *>(ptr)));
  memcpy(handle, &h, sizeof h);
  return TCRV_CUDA_OK;
}

int tcrv_cuda_peer_open(const unsigned char *handle, void **ptr) {
  if (!ptr || !handle)
    return TCRV_CUDA_ERR_INVALID_ARGUMENT;
  cudaIpcMemHandle_t h;
  memcpy(&h, handle, sizeof h);
  TCRV_CUDA_TRY(cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess));
  return TCRV_CUDA_OK;
}

int tcrv_cuda_peer_close(void *ptr) {
  if (ptr)
    TCRV_CUDA_TRY(cudaIpcCloseMemHandle(ptr));
  return TCRV_CUDA_OK;
}

int tcrv_cuda_gemm_q4_0_q8_0(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t by, size_t nr,
                             size_t nc, size_t bx, size_t bs, void *workspace, size_t workspace_bytes,
                             unsigned flags, tcrv_cuda_stream stream) {
  const int st = check_matrix_args(n, s, vx, vy, by, nr, nc, bx, bs, TCRV_Q4_0_BLOCK_BYTES);
  if (st != TCRV_CUDA_OK)
    return st;
  if (nr == 0 || nc == 0)
    return TCRV_CUDA_OK;
  const size_t wbytes = gemm_weights_bytes(n, nr);
  if (n != 0 && (!workspace || workspace_bytes < wbytes + gemm_acts_bytes(n, nc) ||
                 reinterpret_cast<uintptr_t>(workspace) % 256 != 0))
    return TCRV_CUDA_ERR_WORKSPACE;
  uint8_t *ws = static_cast<uint8_t *>(workspace);
  if (n != 0) {
    const int rc = launch_gemm_prepare_weights_q4_0(n, vx, bx, nr, ws, as_stream(stream));
    if (rc != TCRV_CUDA_OK)
      return rc;
  }
  return tcrv_cuda_gemm_q4_0_q8_0_prepared(n, s, ws, vy, by, nr, nc, bs, ws + wbytes, workspace_bytes - wbytes, flags,
                                           stream);
}

int tcrv_cuda_gemm_q4_0_q8_0_static_scratch(size_t n, float *s, const uint8_t *vx, const uint8_t *vy, size_t by,
                                            size_t nr, size_t nc, size_t bx, size_t bs, unsigned flags,
                                            tcrv_cuda_stream stream) {
  (void)flags;
  const int st = check_matrix_args(n, s, vx, vy, by, nr, nc, bx, bs, TCRV_Q4_0_BLOCK_BYTES);
  if (st != TCRV_CUDA_OK)
    return st;
  if (n == 0) {
    for (size_t r = 0; r < nr; ++r)
      TCRV_CUDA_TRY(cudaMemsetAsync(s + r * bs, 0, nc * sizeof(float), as_stream(stream)));
    return TCRV_CUDA_OK;
  }
  return launch_gemm_static_scratch(n, s, vx, bx, vy, by, nr, nc, bs, as_stream(stream));
}

}  // extern "C"
