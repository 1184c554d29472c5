"""GPU parity of the streaming GEMV for rows of any block count: rows that start off 16-byte
boundaries, odd block counts, matrices that begin or end off a boundary, padded strides, every
column count; all bit-exact against the oracle (lane-pair order or the sequential fold)."""
import numpy as np
import pytest

import graph_time
import sibling_data as sd
from test_gpu_gemv import dev, make, restated

pytestmark = pytest.mark.gpu


def place(torch, w, lead, pad):
    """The rows of `w` in device memory, `lead` bytes into an allocation and `pad` bytes apart."""
    nr, rb = w.shape
    flat = np.full(lead + nr * (rb + pad) - pad, 0xA5, dtype=np.uint8)
    for r in range(nr):
        flat[lead + r * (rb + pad):lead + r * (rb + pad) + rb] = w[r]
    return dev(torch, flat)


# odd and even block counts around the 32 pairs of a warp's pass, one block, 4n+1..4n+3; a row per
# warp or several; the last two at the smallest row count the kernel takes and with long rows
@pytest.mark.parametrize("q8w", [False, True])
@pytest.mark.parametrize("nr,nb,nc,lead,pad", [(64, 1, 1, 0, 0), (257, 3, 2, 2, 0), (300, 63, 1, 14, 0), (300, 65, 3, 0, 2),
                                               (4000, 91, 1, 0, 0), (2500, 66, 1, 6, 0), (97, 130, 8, 0, 14),
                                               (97, 129, 5, 4, 0), (8, 341, 1, 2, 0), (40, 343, 6, 0, 0),
                                               # shared memory for one or two of the sixteen rings
                                               (8, 1001, 4, 0, 0), (33, 563, 8, 2, 0), (300, 1501, 2, 0, 2),
                                               # the smallest rows that do not stay on the general kernel
                                               (2500, 1, 1, 0, 0), (1250, 3, 2, 2, 0), (3000, 5, 1, 0, 4),
                                               # slots of 3 and 4 rows, then three slots to a warp and more
                                               # (a ring slot is used again), in equal and unequal parts
                                               (7500, 91, 1, 0, 0), (20001, 65, 1, 2, 0), (32000, 91, 1, 0, 0),
                                               (9000, 35, 3, 0, 2), (20000, 33, 8, 6, 0)])
def test_any_rows_match_the_oracle(cuda, pkg, O, q8w, nr, nb, nc, lead, pad):
    k = nb * 32
    w, x = make(O, nr, k, nc, q8w, 40 + nr + nb)
    buf, xd = place(cuda, w, lead, pad), dev(cuda, x)
    L, stream = pkg.lib(), cuda.cuda.current_stream().cuda_stream
    fn = L.tcrv_cuda_gemv_q8_0_q8_0 if q8w else L.tcrv_cuda_gemv_q4_0_q8_0
    bx = w.shape[1] + pad
    for flags in (0, pkg.FLAG_STATIC_WEIGHTS, pkg.FLAG_STRICT_ORDER):
        order = L.tcrv_cuda_gemv_fold_order(int(q8w), k, nc, buf.data_ptr() + lead, bx, xd.data_ptr(), xd.stride(0), flags)
        assert order == (0 if flags & pkg.FLAG_STRICT_ORDER else 1)
        out = cuda.full((nr, nc + 1), -1.0, dtype=cuda.float32, device="cuda")
        assert fn(k, out.data_ptr(), buf.data_ptr() + lead, xd.data_ptr(), xd.stride(0), nr, nc, bx, nc + 1, flags, stream) == 0
        got = out.cpu().numpy()
        assert np.array_equal(got[:, :nc].view(np.uint32), restated(O, w, x, q8w, order).view(np.uint32))
        assert np.all(got[:, nc:] == -1.0)
    pkg.check_device_errors()


@pytest.mark.parametrize("fmt", [1, 2, 3])
@pytest.mark.parametrize("nr,nb,nc,lead,pad", [(64, 1, 1, 0, 0), (300, 33, 2, 2, 0), (2500, 91, 1, 0, 0), (130, 127, 4, 8, 2),
                                               (70, 346, 8, 0, 0), (2500, 1, 1, 0, 0), (7500, 61, 1, 0, 0),
                                               (20001, 67, 1, 4, 0), (9000, 35, 3, 0, 2), (12000, 17, 6, 2, 0)])
def test_any_sibling_rows_match_the_oracle(cuda, pkg, O, fmt, nr, nb, nc, lead, pad):
    w, x = sd.make(fmt, nr, nc, nb, 500 + fmt + nb)
    buf, xd = place(cuda, w, lead, pad), dev(cuda, x)
    out = cuda.full((nr, nc), -1.0, dtype=cuda.float32, device="cuda")
    assert pkg.lib().tcrv_cuda_sibling_dot_rows(fmt, nb * 32, out.data_ptr(), buf.data_ptr() + lead, xd.data_ptr(), xd.stride(0),
                                                nr, nc, w.shape[1] + pad, nc, cuda.cuda.current_stream().cuda_stream) == 0
    assert np.array_equal(out.cpu().numpy().view(np.uint32), O.sibling_dot_rows(fmt, w, x).view(np.uint32))
    pkg.check_device_errors()


@pytest.mark.parametrize("q8w", [False, True])
@pytest.mark.parametrize("strict", [False, True])
@pytest.mark.parametrize("shapes", [
    # rows of more than 128 blocks (activations not in registers) and several slots to a warp among them
    [(1000, 91), (300, 64), (64, 3), (2000, 90), (700, 131), (9000, 33)],
    [(33, 1001), (300, 1401)],  # shared memory for two to five rings
])
def test_a_group_with_such_rows_has_the_bits_of_the_single_calls(cuda, pkg, O, q8w, strict, shapes):
    flags = pkg.FLAG_STRICT_ORDER if strict else 0
    problems, want = [], []
    for i, (nr, nb) in enumerate(shapes):
        w, x = make(O, nr, nb * 32, 1, q8w, 80 + i)
        wd, xd = dev(cuda, w), dev(cuda, x)
        problems.append((wd, xd, cuda.empty((nr, 1), dtype=cuda.float32, device="cuda")))
        want.append(restated(O, w, x, q8w, 0 if strict else 1))
    pkg.gemv_group(pkg.gemv_group_calls(problems, q8_weights=q8w), q8_weights=q8w, flags=flags)
    for (_, _, out), ref in zip(problems, want):
        assert np.array_equal(out.cpu().numpy().view(np.uint32), ref.view(np.uint32))
    pkg.check_device_errors()


def gemv_times(cuda, pkg, q8w, nr, nb, nc, flags):
    """us of a call on the streaming kernel's route and on the general kernel (activations at an odd address)."""
    row = nb * (34 if q8w else 18)
    w = cuda.randint(0, 60, (nr * row,), dtype=cuda.uint8, device="cuda")
    x = cuda.randint(0, 60, (nc * nb * 34 + 1,), dtype=cuda.uint8, device="cuda")
    out = cuda.empty(nr * nc, device="cuda")
    fn = pkg.lib().tcrv_cuda_gemv_q8_0_q8_0 if q8w else pkg.lib().tcrv_cuda_gemv_q4_0_q8_0
    return [graph_time.us(cuda, lambda st: fn(nb * 32, out.data_ptr(), w.data_ptr(), x.data_ptr() + odd, nb * 34, nr, nc, row, nc,
                                              flags, st)) for odd in (0, 1)]


@pytest.mark.parametrize("q8w,nr,nb,nc,flags", [(False, 8, 1001, 4, 0), (False, 64, 1001, 4, 1), (True, 16, 343, 8, 1),  # few rings
                                                  (False, 148, 5, 8, 1), (True, 300, 5, 1, 1), (False, 300, 1, 1, 0)])  # tiny
def test_few_rings_and_tiny_matrices_are_no_slower_than_the_general_kernel(cuda, pkg, q8w, nr, nb, nc, flags):
    streaming, general = gemv_times(cuda, pkg, q8w, nr, nb, nc, flags)
    assert streaming < 1.15 * general, f"{streaming:.2f} us against {general:.2f}"
