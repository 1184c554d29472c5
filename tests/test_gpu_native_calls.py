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


def test_running_out_of_device_memory_keeps_its_class(cuda, pkg):
    # 2**34 rows that share one row's memory: the output would take 4 TB, which the allocator refuses
    x = cuda.ones(1, 64, device="cuda").expand(1 << 34, 64)
    with pytest.raises(cuda.OutOfMemoryError):
        pkg.rms_norm(x, 1e-5)


def test_errors_of_torch_keep_their_class(cuda, pkg):
    w = cuda.zeros(16, 18 * 4, dtype=cuda.uint8, device="cuda")
    x = cuda.zeros(1, 34 * 4, dtype=cuda.uint8, device="cuda")
    with pytest.raises(IndexError):  # an output without dimensions has no row stride
        pkg.gemv(w, x, out=cuda.zeros((), device="cuda"))
