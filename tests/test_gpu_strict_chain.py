"""GPU parity, the table per CTA: folds of a few blocks up to several batches with every remainder, items that
do not divide the 512 workers, and five-bit codes of every pattern give the sequential fold bit for bit."""
import numpy as np
import pytest
import sibling_data as sd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [1, 2, 3])
@pytest.mark.parametrize("nr,nb,nc", [(2048, 8, 1), (2051, 24, 1), (2048, 40, 1), (2049, 104, 1), (2060, 344, 1), (6001, 56, 2)])
def test_sibling_formats(cuda, pkg, O, fmt, nr, nb, nc):
    w, x = sd.make(fmt, nr, nc, nb, 970 + fmt + nb)
    wd, xd = cuda.from_numpy(w).cuda(), cuda.from_numpy(x).cuda()
    got = pkg.sibling_dot_rows(fmt, wd, xd).cpu().numpy()
    pkg.check_device_errors()
    rows = np.unique(np.concatenate([np.arange(0, nr, 41), np.arange(nr - 40, nr)]))
    assert np.array_equal(got[rows].view(np.uint32), O.sibling_dot_rows(fmt, w[rows], x).view(np.uint32))


@pytest.mark.parametrize("q8w,nb,nc", [(False, 136, 4), (False, 168, 8), (True, 152, 3), (True, 344, 5)])
def test_long_rows_in_the_reference_order(cuda, pkg, O, q8w, nb, nc):
    nr = 131
    w = (O.quantize_q8_0 if q8w else O.quantize_q4_0)(O.fill_normal(nr * nb * 32, 71, 0, 0.02).reshape(nr, nb * 32))
    x = O.quantize_q8_0(O.fill_normal(nc * nb * 32, 72).reshape(nc, nb * 32))
    got = pkg.gemv(cuda.from_numpy(w).cuda(), cuda.from_numpy(x).cuda(), q8_weights=q8w, flags=pkg.FLAG_STRICT_ORDER).cpu().numpy()
    pkg.check_device_errors()
    assert np.array_equal(got.view(np.uint32), O.gemm(w, x, q8_weights=q8w, fold=O.FOLD_FMA).view(np.uint32))
