"""GPU parity of the sibling block formats (Q4_1 x Q8_1, Q5_0 x Q8_0, Q5_1 x Q8_1) against the
oracle: per-block int32 sums and fp32 rows, both bit-exact (strict ascending fold)."""
import numpy as np
import pytest

import graph_time
import sibling_data as sd

pytestmark = pytest.mark.gpu


def dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("fmt", [1, 2, 3])
@pytest.mark.parametrize("nr,nc,nb", [(1, 1, 1), (5, 3, 33), (64, 2, 128), (300, 1, 344)])
def test_sibling_rows_bit_exact(cuda, pkg, O, fmt, nr, nc, nb):
    w, x = sd.make(fmt, nr, nc, nb, 700 + 10 * fmt + nr)
    wd, xd = dev(cuda, w), dev(cuda, x)
    sums = pkg.sibling_block_sums(fmt, wd, xd).cpu().numpy()
    for r in range(0, nr, max(1, nr // 7)):
        for c in range(nc):
            assert np.array_equal(sums[r, c], O.sibling_block_sums(fmt, w[r], x[c]))
    got = pkg.sibling_dot_rows(fmt, wd, xd).cpu().numpy()
    rows = np.unique(np.concatenate([np.arange(0, nr, max(1, nr // 40)), [nr - 1]]))
    want = O.sibling_dot_rows(fmt, w[rows], x)
    assert np.array_equal(got[rows].view(np.uint32), want.view(np.uint32))
    pkg.check_device_errors()


@pytest.mark.parametrize("fmt,entry", [(1, "tcrv_cuda_vec_dot_q4_1_q8_1"), (2, "tcrv_cuda_vec_dot_q5_0_q8_0"),
                                       (3, "tcrv_cuda_vec_dot_q5_1_q8_1")])
def test_sibling_vec_dot_entries_padded_and_unaligned(cuda, pkg, O, fmt, entry):
    w, x = sd.make(fmt, 1, 1, 96, 800 + fmt)
    L = pkg.lib()
    # one byte of offset: nothing in these formats is aligned anyway
    wb = cuda.zeros(w.size + 1, dtype=cuda.uint8, device="cuda")
    wb[1:] = dev(cuda, w[0])
    xd = dev(cuda, x[0])
    out = cuda.zeros(1, dtype=cuda.float32, device="cuda")
    assert getattr(L, entry)(96 * 32, out.data_ptr(), wb.data_ptr() + 1, xd.data_ptr(), None) == 0
    cuda.cuda.synchronize()
    assert out.cpu().numpy()[0] == O.sibling_dot_rows(fmt, w, x)[0, 0]
    # argument checks
    assert getattr(L, entry)(33, out.data_ptr(), wb.data_ptr(), xd.data_ptr(), None) == -1
    assert getattr(L, entry)(64, None, wb.data_ptr(), xd.data_ptr(), None) == -1
    assert L.tcrv_cuda_sibling_dot_rows(9, 64, out.data_ptr(), wb.data_ptr(), xd.data_ptr(), 0, 1, 1, 0, 1, None) == -1
    assert L.tcrv_cuda_sibling_dot_rows(fmt, 64, out.data_ptr(), wb.data_ptr(), xd.data_ptr(), 10, 1, 2, 100, 2, None) == -1


@pytest.mark.parametrize("fmt", [1, 2, 3])
@pytest.mark.parametrize("nr,nb,pad", [(2000, 128, 0), (777, 8, 0), (130, 40, 48), (4099, 64, 16)])
def test_sibling_streaming_rows_bit_exact(cuda, pkg, O, fmt, nr, nb, pad):
    # One column against many rows takes a streaming kernel: contiguous rows, rows with a stride, ragged last
    # slots; the one with a table per CTA at any address of the activation column, the one with a table per warp
    # where the weights are off 16-byte boundaries, by whole words or not.
    w, x = sd.make(fmt, nr, 1, nb, 900 + fmt + nr)
    wb = w.shape[1]
    padded = np.zeros((nr, wb + pad), dtype=np.uint8)
    padded[:, :wb] = w
    wd = dev(cuda, padded)
    xd = dev(cuda, x)
    L = pkg.lib()
    rows = np.unique(np.concatenate([np.arange(0, nr, max(1, nr // 60)), np.arange(max(0, nr - 40), nr)]))
    want = O.sibling_dot_rows(fmt, w[rows], x)

    def run(x_ptr, w_ptr=wd.data_ptr()):
        out = cuda.full((nr, 1), float("nan"), dtype=cuda.float32, device="cuda")
        assert L.tcrv_cuda_sibling_dot_rows(fmt, nb * 32, out.data_ptr(), w_ptr, x_ptr, x.shape[1], nr, 1,
                                            wb + pad, 1, None) == 0
        return out.cpu().numpy()

    assert np.array_equal(run(xd.data_ptr())[rows].view(np.uint32), want.view(np.uint32))
    # the same column one byte further on
    flat = cuda.zeros(x.shape[1] + 1, dtype=cuda.uint8, device="cuda")
    flat[1:] = xd[0]
    assert np.array_equal(run(flat.data_ptr() + 1)[rows].view(np.uint32), want.view(np.uint32))
    for shift in (4, 2):
        moved = cuda.zeros(padded.size + shift, dtype=cuda.uint8, device="cuda")
        moved[shift:] = wd.reshape(-1)
        assert np.array_equal(run(xd.data_ptr(), moved.data_ptr() + shift)[rows].view(np.uint32), want.view(np.uint32))
    pkg.check_device_errors()


# the calls that the table per CTA takes at any address: ragged slots, rows with a stride
@pytest.mark.parametrize("fmt,nr,nb,nc,pad", [(2, 8192, 128, 1, 0), (2, 11009, 64, 1, 16), (3, 20003, 8, 1, 0), (1, 6001, 16, 4, 0),
                                              (2, 9001, 24, 2, 32), (3, 8195, 40, 8, 0), (1, 2049, 344, 7, 16)])
def test_sibling_table_per_cta_bit_exact(cuda, pkg, O, fmt, nr, nb, nc, pad):
    w, x = sd.make(fmt, nr, nc, nb, 950 + fmt + nb)
    padded = np.zeros((nr, w.shape[1] + pad), dtype=np.uint8)
    padded[:, :w.shape[1]] = w
    wd, xd = dev(cuda, padded), dev(cuda, x)
    out = cuda.full((nr, nc), float("nan"), dtype=cuda.float32, device="cuda")
    assert pkg.lib().tcrv_cuda_sibling_dot_rows(fmt, nb * 32, out.data_ptr(), wd.data_ptr(), xd.data_ptr(), xd.stride(0), nr, nc,
                                                padded.shape[1], nc, cuda.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(out.cpu().numpy().view(np.uint32), O.sibling_dot_rows(fmt, w, x).view(np.uint32))
    pkg.check_device_errors()


@pytest.mark.parametrize("fmt,nr,nb,nc", [(1, 4096, 128, 1), (2, 4096, 344, 2), (3, 11008, 128, 8), (1, 32000, 8, 6), (2, 32000, 16, 3),
                                          (3, 5120, 448, 4), (3, 4096, 344, 6)])
def test_sibling_calls_take_the_faster_streaming_kernel(cuda, pkg, fmt, nr, nb, nc):
    # activations at an odd address leave only the table per CTA: a call at an even one is no slower, and
    # one at an odd address streams as well (the general kernel takes 2.4 to 9 times as long)
    wb, ab = sd.STRIDES[fmt]
    w = cuda.randint(0, 60, (nr * nb * wb,), dtype=cuda.uint8, device="cuda")
    x = cuda.randint(0, 60, (nc * nb * ab + 1,), dtype=cuda.uint8, device="cuda")
    out = cuda.empty(nr * nc, device="cuda")
    fn = pkg.lib().tcrv_cuda_sibling_dot_rows
    even, odd = (graph_time.us(cuda, lambda st: fn(fmt, nb * 32, out.data_ptr(), w.data_ptr(), x.data_ptr() + o, nb * ab, nr, nc,
                                                   nb * wb, nc, st)) for o in (0, 1))
    assert even < 1.1 * odd and odd < 1.6 * even, f"{even:.2f} us at an even address, {odd:.2f} at an odd one"
    pkg.check_device_errors()


# calls on both sides of the lines between the two streaming kernels, the shapes whose route was wrong among them
@pytest.mark.parametrize("fmt,nr,nb,nc", [(1, 11008, 128, 4), (3, 11008, 128, 4), (1, 4096, 128, 3), (2, 1536, 128, 8), (1, 4096, 344, 1), (2, 512, 256, 1),
                                          (1, 2048, 128, 1), (2, 100, 16, 8), (3, 32000, 128, 1), (2, 11008, 200, 2), (3, 11008, 344, 4), (3, 11008, 128, 8), (2, 512, 128, 8)])
def test_the_rule_takes_the_faster_of_both(cuda, pkg, fmt, nr, nb, nc):
    # weights off 16-byte boundaries leave only the table per warp, activations at an odd address only the one per CTA
    wb, ab = sd.STRIDES[fmt]
    w = cuda.randint(0, 60, (nr * nb * wb + 4,), dtype=cuda.uint8, device="cuda")
    x = cuda.randint(0, 60, (nc * nb * ab + 1,), dtype=cuda.uint8, device="cuda")
    out = cuda.empty(nr * nc, device="cuda")
    fn = pkg.lib().tcrv_cuda_sibling_dot_rows
    rule, warp, cta = (graph_time.us(cuda, lambda st: fn(fmt, nb * 32, out.data_ptr(), w.data_ptr() + wo, x.data_ptr() + xo, nb * ab, nr, nc,
                                                         nb * wb, nc, st)) for wo, xo in ((0, 0), (4, 0), (0, 1)))
    assert rule < 1.12 * min(warp, cta), f"{rule:.2f} us by the rule, {warp:.2f} with the table per warp, {cta:.2f} per CTA"
    pkg.check_device_errors()


@pytest.mark.parametrize("nr", [300, 1000, 4096])
def test_one_ring_is_not_for_many_rows(cuda, pkg, nr):
    # rows of 1920 blocks leave a ring to one warp only; weights at an odd address leave only the general kernel
    w = cuda.randint(0, 60, (nr * 1920 * 24 + 1,), dtype=cuda.uint8, device="cuda")
    x = cuda.randint(0, 60, (1920 * 36,), dtype=cuda.uint8, device="cuda")
    out = cuda.empty(nr, device="cuda")
    fn = pkg.lib().tcrv_cuda_sibling_dot_rows
    rule, general = (graph_time.us(cuda, lambda st: fn(3, 61440, out.data_ptr(), w.data_ptr() + o, x.data_ptr(), 1920 * 36, nr, 1, 1920 * 24, 1, st))
                     for o in (0, 1))
    assert rule < 1.1 * general, f"{rule:.1f} us by the rule, {general:.1f} on the general kernel"
    pkg.check_device_errors()
