"""GPU parity, work items of the prefill GEMM: whole items, halves and narrow ones of 32 columns at their edges
(ragged rows and columns, block counts that end a stage early) equal the sequential oracle bit for bit, with both
folds and with several destinations.  (test_gpu_gemm_narrow_items.py has those of 16 columns.)"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,k,nc", [
    (127, 32, 31), (129, 96, 33), (255, 160, 63), (257, 224, 65),  # 128 x 16
    (4096, 416, 77), (4001, 32, 77), (4081, 160, 95), (3900, 96, 97), (4111, 288, 65), (2049, 128, 160),  # 128 x 32
    (4000, 160, 200), (3969, 32, 193), (4097, 224, 161),  # 256 x 64, all of them cut into halves
    (4864, 160, 512),   # 152 whole items: one round and four items cut into halves
    (4737, 96, 481),    # the same with a second row tile that does not exist and ragged columns
    (20480, 32, 128),   # 160 whole items of one block
])
def test_items_at_their_edges_are_bit_exact(cuda, pkg, O, nr, k, nc):
    w = O.quantize_q4_0(O.fill_normal(nr * k, 51, 0, 0.02).reshape(nr, k))
    x = O.quantize_q8_0(O.fill_normal(nc * k, 52).reshape(nc, k))
    want = O.gemm(w, x, fold=O.FOLD_FMA, threads=8).view(np.uint32)
    wd, xd = cuda.from_numpy(w).cuda(), cuda.from_numpy(x).cuda()
    pw = pkg.PreparedWeights(wd)
    assert np.array_equal(pkg.gemm(pw, xd).cpu().numpy().view(np.uint32), want)
    # two destinations: the staging tile of the fused gather
    L = pkg.lib()
    ws = cuda.empty(L.tcrv_cuda_gemm_acts_workspace_bytes(k, nc), dtype=cuda.uint8, device="cuda")
    bs = (nc + 3) // 4 * 4
    outs = [cuda.full((nr, bs), -1.0, dtype=cuda.float32, device="cuda") for _ in range(2)]
    dst = (ctypes.c_void_p * 2)(*[o.data_ptr() for o in outs])
    st = L.tcrv_cuda_gemm_q4_0_q8_0_prepared_multi(k, dst, 2, pw.buffer.data_ptr(), xd.data_ptr(), xd.stride(0), nr, nc,
                                                   bs, ws.data_ptr(), ws.numel(), 0,
                                                   cuda.cuda.current_stream().cuda_stream)
    assert st == 0
    pkg.check_device_errors()
    for o in outs:
        res = o.cpu().numpy()
        assert np.array_equal(np.ascontiguousarray(res[:, :nc]).view(np.uint32), want) and np.all(res[:, nc:] == -1.0)


# (tokens, weight rows, K): whole items with halves in the last round, a row tile that does not exist with
# ragged columns, items of one block; halves only; items of 128 x 32
@pytest.mark.parametrize("tokens,rows,k", [(512, 4864, 160), (484, 4752, 96), (128, 20480, 32), (200, 4000, 160), (76, 4016, 96), (80, 4112, 32),
                                           (96, 4208, 288)])
def test_items_of_the_repacked_gemm_are_bit_exact(cuda, pkg, O, tokens, rows, k):
    w = O.quantize_q4_0(O.fill_normal(rows * k, 53, 0, 0.02).reshape(rows, k))
    x = O.quantize_q8_0(O.fill_normal(tokens * k, 54).reshape(tokens, k))
    wx, xx = O.rows_to_q4_0x16(w), O.rows_to_q8_0x4(x)
    got = pkg.repack_gemm(cuda.from_numpy(wx).cuda(), cuda.from_numpy(xx).cuda(), k, tokens, rows).cpu().numpy()
    pkg.check_device_errors()
    assert np.array_equal(got.view(np.uint32), O.repack_gemm(wx, xx, k, tokens, rows).view(np.uint32))
