"""The package's native call path (csrc/torch_calls.cpp): what a call does with operands that it
cannot take."""
import pytest

pytestmark = pytest.mark.gpu


def test_an_operand_without_storage_is_an_error(cuda, pkg):
    # torch refuses the data pointer of a vmap wrapper while the call runs without the interpreter lock
    x = cuda.randn(3, 64, device="cuda")
    calls = [lambda r: pkg.vec_silu(r), lambda r: pkg.add(r, r), lambda r: pkg.quantize_q8_0(r)]
    for call in calls:
        with pytest.raises(RuntimeError):
            cuda.func.vmap(call)(x)
    out = pkg.vec_silu(x)  # the interpreter and the device go on
    cuda.cuda.synchronize()
    assert bool(cuda.isfinite(out).all())
