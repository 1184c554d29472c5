"""GPU parity, several columns against rows beyond 4096 elements (the chunk-wise tensor-core kernel): ragged
groups, CTAs with an odd number of them, warps with one to three chunks, columns that 16-byte copies cannot
take and wide row strides give the oracle's restatement of the 16-way order bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q8w,nr,k,nc,pad,shift", [
    (False, 1, 4352, 8, 0, 0), (False, 17, 8448, 5, 0, 0), (False, 33, 12288, 4, 16, 0), (False, 40, 4608, 7, 0, 2),
    (False, 148 * 32 + 9, 4352, 4, 0, 0), (True, 31, 4352, 8, 0, 0), (True, 18, 5888, 6, 48, 6), (True, 148 * 16 + 3, 4352, 4, 0, 0),
])
def test_long_rows_several_columns(cuda, pkg, O, q8w, nr, k, nc, pad, shift):
    w = (O.quantize_q8_0 if q8w else O.quantize_q4_0)(O.fill_normal(nr * k, 61, 0, 0.02).reshape(nr, k))
    x = O.quantize_q8_0(O.fill_normal(nc * k, 62).reshape(nc, k))
    wd = cuda.zeros((nr, w.shape[1] + pad), dtype=cuda.uint8, device="cuda")[:, :w.shape[1]]
    wd.copy_(cuda.from_numpy(w))
    xd = cuda.zeros((nc, x.shape[1] + shift + 2), dtype=cuda.uint8, device="cuda")[:, shift:shift + x.shape[1]] \
        if shift else cuda.zeros((nc, x.shape[1]), dtype=cuda.uint8, device="cuda")
    xd.copy_(cuda.from_numpy(x))
    L = pkg.lib()
    out = cuda.full((nr + 1, nc + 1), -1.0, dtype=cuda.float32, device="cuda")
    fn = L.tcrv_cuda_gemv_q8_0_q8_0 if q8w else L.tcrv_cuda_gemv_q4_0_q8_0
    assert fn(k, out.data_ptr(), wd.data_ptr(), xd.data_ptr(), xd.stride(0), nr, nc, wd.stride(0), nc + 1, 0,
              cuda.cuda.current_stream().cuda_stream) == 0
    pkg.check_device_errors()
    got = out.cpu().numpy()
    assert np.array_equal(np.ascontiguousarray(got[:nr, :nc]).view(np.uint32),
                          O.gemv_ksplit_order(w, x, q8w).view(np.uint32))
    assert np.all(got[nr] == -1.0) and np.all(got[:, nc] == -1.0)


@pytest.mark.parametrize("q8w,nr,k,nc,stride", [(False, 18, 4352, 5, 1 << 27), (True, 17, 4352, 4, (1 << 28) + 16)])
def test_rows_far_apart_keep_the_order_of_near_ones(cuda, pkg, O, q8w, nr, k, nc, stride):
    w = (O.quantize_q8_0 if q8w else O.quantize_q4_0)(O.fill_normal(nr * k, 63, 0, 0.02).reshape(nr, k))
    x = O.quantize_q8_0(O.fill_normal(nc * k, 64).reshape(nc, k))
    room = cuda.empty((nr - 1) * stride + w.shape[1], dtype=cuda.uint8, device="cuda")  # 2.3 and 4.3 GB
    wd = room.as_strided(w.shape, (stride, 1))
    wd.copy_(cuda.from_numpy(w))
    xd = cuda.from_numpy(x).cuda()
    assert pkg.gemv_fold_order(wd, xd, q8_weights=q8w) == 2
    got = pkg.gemv(wd, xd, q8_weights=q8w)
    pkg.check_device_errors()
    assert np.array_equal(got.cpu().numpy().view(np.uint32), O.gemv_ksplit_order(w, x, q8w).view(np.uint32))
