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
