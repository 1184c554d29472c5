"""GPU parity, Q8_0 quantiser: blocks whose 1/d is not finite share passes with plain ones, and products that lie
halfway between integers round to even, as the oracle has it byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 15, 17, 148 * 8 * 16 * 8 + 5])  # a warp's pass is 16 blocks
def test_plain_and_awkward_blocks(cuda, pkg, O, blocks):
    x = O.fill_normal(blocks * 32, 81).reshape(blocks, 32)
    half = (np.arange(32, dtype=np.float32) - 15.5) * np.float32(127 / 15.5)
    half[:31] = np.arange(31, dtype=np.float32) - 15.5  # with 127 among them d is 1: every other value is a half
    half[31] = 127.0
    x[0::3] = half
    x[1::7] = 0.0
    x[2::11] *= np.float32(1e-41)  # d rounds to a subnormal, 1/d overflows
    x[3::13] *= np.float32(1e30)   # d beyond fp16
    got = pkg.quantize_q8_0(cuda.from_numpy(x.reshape(1, -1)).cuda()).cpu().numpy()
    pkg.check_device_errors()
    assert np.array_equal(got, O.quantize_q8_0(x.reshape(1, -1)))


@pytest.mark.parametrize("spread", [1, 5, 16])  # such blocks make up whole passes, share them or stand alone
def test_nan_and_infinity_keep_their_bytes(cuda, pkg, O, spread):
    # a NaN is 0xff and does not count for the maximum; beside an infinity 1/d is 0: the block is plain, its values
    # are 0 and the infinity itself, inf * 0, is 0xff; a block of nothing but NaNs has a NaN for its scale
    n = np.float32("nan")
    odd = O.fill_normal(6 * 32, 83).reshape(6, 32)
    odd[0, ::5] = n
    odd[1, 31] = np.float32("inf")
    odd[2, 0], odd[2, 1] = -np.float32("inf"), n
    odd[3] = n
    odd[4, 1:] = n
    odd[5, 1:], odd[5, 0] = 0.0, n
    odd.view(np.uint32)[0, 0] = 0xFF800123  # another sign and payload
    x = O.fill_normal(16 * 37 * 32, 84).reshape(-1, 32)
    at = np.arange(0, len(x), spread)
    x[at] = odd[at % 6]
    with np.errstate(all="ignore"):
        top = np.fmax.reduce(np.abs(x), axis=1)
        d = (top / np.float32(127)).astype(np.float32)
        inverse = np.where(d != 0, np.float32(1) / d, np.float32(0)).astype(np.float32)
        q = x * inverse[:, None]
        q = np.where(np.isnan(q), 0xFF, np.rint(np.nan_to_num(q)).astype(np.int64) & 0xFF).astype(np.uint8)
        scale = d.astype(np.float16).view(np.uint16)
    scale[np.isnan(d)] = 0x7FFF
    want = np.concatenate([scale.view(np.uint8).reshape(-1, 2), q], axis=1)
    got = pkg.quantize_q8_0(cuda.from_numpy(x.reshape(1, -1)).cuda()).cpu().numpy().reshape(-1, 34)
    pkg.check_device_errors()
    assert np.array_equal(got, want)
