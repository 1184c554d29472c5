"""GPU parity, the narrowest work items of the prefill GEMM (128 rows x 16 columns): ragged rows and columns, block
counts that end a stage early, one and two rounds, both folds, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,k,nc", [(127, 32, 15), (128, 128, 16), (300, 160, 17), (513, 4128, 33), (2048, 224, 143), (32000, 64, 9)])
def test_narrowest_items_are_bit_exact(cuda, pkg, O, nr, k, nc):
    w = O.quantize_q4_0(O.fill_normal(nr * k, 55, 0, 0.02).reshape(nr, k))
    x = O.quantize_q8_0(O.fill_normal(nc * k, 56).reshape(nc, k))
    got = pkg.gemm(pkg.PreparedWeights(cuda.from_numpy(w).cuda()), cuda.from_numpy(x).cuda()).cpu().numpy()
    pkg.check_device_errors()
    assert np.array_equal(got.view(np.uint32), O.gemm(w, x, fold=O.FOLD_FMA, threads=8).view(np.uint32))


@pytest.mark.parametrize("tokens,rows,k", [(16, 128, 96), (36, 528, 160)])
def test_narrowest_items_of_the_repacked_gemm_are_bit_exact(cuda, pkg, O, tokens, rows, k):
    w = O.quantize_q4_0(O.fill_normal(rows * k, 57, 0, 0.02).reshape(rows, k))
    x = O.quantize_q8_0(O.fill_normal(tokens * k, 58).reshape(tokens, k))
    wx, xx = O.rows_to_q4_0x16(w), O.rows_to_q8_0x4(x)
    got = pkg.repack_gemm(cuda.from_numpy(wx).cuda(), cuda.from_numpy(xx).cuda(), k, tokens, rows).cpu().numpy()
    pkg.check_device_errors()
    assert np.array_equal(got.view(np.uint32), O.repack_gemm(wx, xx, k, tokens, rows).view(np.uint32))
