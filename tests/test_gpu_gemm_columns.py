"""GPU parity, activations prepared in tiles of 8 columns x 32 blocks: ragged columns and blocks, rows whose bytes
end inside a 16-byte piece, and the padding the GEMM's scale boxes read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,nb,pad", [(1, 1, 0), (7, 8, 0), (9, 33, 14), (13, 32, 0), (16, 71, 10), (70, 65, 6), (3, 40, 2)])
def test_prepared_columns_give_the_same_product(cuda, pkg, O, nc, nb, pad):
    k, nr = nb * 32, 40  # (pad 2 leaves the 16-byte boundaries: the kernel for any alignment)
    w = O.quantize_q4_0(O.fill_normal(nr * k, 91, 0, 0.02).reshape(nr, k))
    x = O.quantize_q8_0(O.fill_normal(nc * k, 92).reshape(nc, k))
    xd = cuda.zeros((nc, x.shape[1] + pad), dtype=cuda.uint8, device="cuda")[:, :x.shape[1]]
    xd.copy_(cuda.from_numpy(x))
    L = pkg.lib()
    pw = pkg.PreparedWeights(cuda.from_numpy(w).cuda())
    ws = cuda.full((L.tcrv_cuda_gemm_acts_workspace_bytes(k, nc),), 0x7F, dtype=cuda.uint8, device="cuda")  # NaNs where nothing is written
    out = cuda.full((nr, nc), -1.0, dtype=cuda.float32, device="cuda")
    assert L.tcrv_cuda_gemm_q4_0_q8_0_prepared(k, out.data_ptr(), pw.buffer.data_ptr(), xd.data_ptr(), xd.stride(0), nr, nc, nc,
                                               ws.data_ptr(), ws.numel(), 0, cuda.cuda.current_stream().cuda_stream) == 0
    pkg.check_device_errors()
    assert np.array_equal(out.cpu().numpy().view(np.uint32), O.gemm(w, x, fold=O.FOLD_FMA).view(np.uint32))
