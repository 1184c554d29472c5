"""GPU parity, operand preparation of the prefill GEMM: every kernel that unpacks Q4_0 rows gives the
GEMM the same operands, whatever the rows' alignment, stride and block count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# block counts with and without padding to 4 blocks, odd totals (a pair of blocks that is half
# there, rows that change inside a pair), and column counts with and without padding to 4
@pytest.mark.parametrize("nr,k,nc", [(1, 32, 1), (3, 32, 5), (129, 96, 9), (257, 544, 33), (515, 1024, 66)])
@pytest.mark.parametrize("offset,pad", [(0, 0), (2, 0), (1, 0), (0, 18), (0, 1)])
def test_prepared_rows_of_any_alignment_and_stride(cuda, pkg, O, nr, k, nc, offset, pad):
    w = O.quantize_q4_0(O.fill_normal(nr * k, 41, 0, 0.02).reshape(nr, k))
    x = O.quantize_q8_0(O.fill_normal(nc * k, 42).reshape(nc, k))
    bx = w.shape[1] + pad
    host = np.zeros(offset + nr * bx, dtype=np.uint8)
    rows = host[offset:].reshape(nr, bx)
    rows[:, :w.shape[1]] = w
    wd, xd = cuda.from_numpy(host).cuda(), cuda.from_numpy(np.ascontiguousarray(x)).cuda()
    L = pkg.lib()
    # 0xff everywhere first: what is not written must not reach a result
    ws = cuda.full((L.tcrv_cuda_gemm_workspace_bytes(k, nr, nc),), 255, dtype=cuda.uint8, device="cuda")
    out = cuda.empty((nr, nc), dtype=cuda.float32, device="cuda")
    st = L.tcrv_cuda_gemm_q4_0_q8_0(k, out.data_ptr(), wd.data_ptr() + offset, xd.data_ptr(), xd.stride(0), nr, nc, bx,
                                    nc, ws.data_ptr(), ws.numel(), 0, cuda.cuda.current_stream().cuda_stream)
    assert st == 0
    pkg.check_device_errors()
    want = O.gemm(w, x, fold=O.FOLD_FMA, threads=8)
    assert np.array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32))
