"""The package's native call path (csrc/torch_calls.cpp): what a call does with operands that it
cannot take."""
import pytest

import sibling_data as sd

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


@pytest.fixture(scope="module")
def operands(cuda, pkg):
    """Small operands of every call: 48 weight rows of 4 blocks, 3 columns, 8 rows of 128 floats."""
    f = cuda.randn(48, 128, device="cuda")
    x = cuda.randn(8, 128, device="cuda")
    wq, xq = pkg.quantize_q4_0(f), pkg.quantize_q8_0(x[:3].contiguous())
    sw, sx = sd.make(2, 48, 3, 4, 5)
    return {"f": f, "x": x, "wq": wq, "xq": xq, "pw": pkg.PreparedWeights(wq), "w16": cuda.zeros(3 * 4 * 288, dtype=cuda.uint8, device="cuda"),
            "sw": cuda.from_numpy(sw).cuda(), "sx": cuda.from_numpy(sx).cuda(), "cache": pkg.rope_cache(128, 1.0, 0.9)}


# every call with an output: the call, the output's type, the fewest elements that it can take
OUTPUTS = {
    "add": (lambda p, o, out: p.add(o["x"], o["x"], out=out), "float32", 1024),
    "dequantize_q4_0": (lambda p, o, out: p.dequantize_q4_0(o["wq"], out=out), "float32", None),
    "quantize_q8_0": (lambda p, o, out: p.quantize_q8_0(o["x"], out=out), "uint8", 8 * 136),
    "quantize_q4_0": (lambda p, o, out: p.quantize_q4_0(o["x"], out=out), "uint8", 8 * 72),
    "gemv": (lambda p, o, out: p.gemv(o["wq"], o["xq"], out=out.view(-1, 3)), "float32", 144),
    "gemv_group_calls": (lambda p, o, out: p.gemv_group_calls([(o["wq"], o["xq"], out.view(-1, 3))]), "float32", 144),
    "gemm": (lambda p, o, out: p.gemm(o["wq"], o["xq"], out=out.view(-1, 3)), "float32", 144),
    "gemm_prepared": (lambda p, o, out: p.gemm(o["pw"], o["xq"], out=out.view(-1, 3)), "float32", 144),
    "sibling_dot_rows": (lambda p, o, out: p.sibling_dot_rows(2, o["sw"], o["sx"], out=out.view(-1, 3)), "float32", 144),
    "rms_norm": (lambda p, o, out: p.rms_norm(o["x"], 1e-5, out=out.view(-1, 128)), "float32", 1024),
    "rope_apply": (lambda p, o, out: p.rope_apply(o["x"], o["cache"], out=out.view(-1, 128)), "float32", 1024),
    "vec_silu": (lambda p, o, out: p.vec_silu(o["x"], out=out), "float32", 1024),
    "repack_gemv": (lambda p, o, out: p.repack_gemv(o["w16"], o["xq"][0], 48, out=out), "float32", 48),
}


@pytest.mark.parametrize("name", sorted(OUTPUTS))
def test_an_output_that_is_too_small_is_refused(cuda, pkg, operands, name):
    call, dtype, least = OUTPUTS[name]
    if least is None:  # as many elements as the output has: more than the blocks hold
        big = cuda.empty(48 * 128 + 32, dtype=cuda.float32, device="cuda")
        with pytest.raises(ValueError):
            call(pkg, operands, big)
        call(pkg, operands, big[:64])
        return
    row = 3 if least == 144 else 128 if name in ("rms_norm", "rope_apply") else 1  # elements of a row of `out`
    room = cuda.empty(least, dtype=getattr(cuda, dtype), device="cuda")
    with pytest.raises(ValueError):
        call(pkg, operands, room[:least - row])
    call(pkg, operands, room)
    pkg.check_device_errors()


def test_inputs_that_end_early_are_refused(cuda, pkg, operands):
    with pytest.raises(ValueError):
        pkg.add(operands["x"], operands["x"][:7])
    with pytest.raises(ValueError):
        pkg.rope_apply(operands["x"], operands["cache"][:126])


@pytest.mark.parametrize("call", [lambda p, o, out: p.rms_norm(o["x"], 1e-5, out=out),
                                  lambda p, o, out: p.rope_apply(o["x"], o["cache"], out=out)])
def test_row_outputs_are_float32_with_contiguous_rows(cuda, pkg, operands, call):
    with pytest.raises(TypeError):
        call(pkg, operands, cuda.empty(8, 128, dtype=cuda.int32, device="cuda"))
    with pytest.raises(ValueError):
        call(pkg, operands, cuda.empty(8, 256, device="cuda")[:, ::2])
    call(pkg, operands, cuda.empty(8, 256, device="cuda")[:, 3:131])  # a row stride is fine
    pkg.check_device_errors()


def test_operands_in_page_locked_memory_are_read_where_they_lie(cuda, pkg, operands):
    o = operands
    wq, xq = o["wq"].cpu().pin_memory(), o["xq"].cpu().pin_memory()
    out = cuda.full((48, 3), -1.0, device="cuda")
    assert cuda.equal(pkg.gemv(o["wq"], xq), pkg.gemv(o["wq"], o["xq"]))
    want = pkg.gemm(o["wq"], o["xq"])
    assert cuda.equal(pkg.gemm(o["wq"], xq), want)
    assert cuda.equal(pkg.gemm(wq, xq, out=out), want)
    assert cuda.equal(pkg.gemm(o["pw"], xq, out=out.fill_(-1.0)), want)
    rows = cuda.zeros(8, 128).pin_memory()
    normed, rotated = pkg.rms_norm(o["x"], 1e-5), pkg.rope_apply(o["x"], o["cache"])
    pkg.rms_norm(o["x"], 1e-5, out=rows)
    cuda.cuda.synchronize()
    assert cuda.equal(rows, normed.cpu())
    pkg.rope_apply(o["x"], o["cache"], out=rows)
    cuda.cuda.synchronize()
    assert cuda.equal(rows, rotated.cpu())
    # a result without a place of its own needs an operand on the device to lie beside; pageable memory is refused
    for call in (lambda: pkg.gemv(wq, xq), lambda: pkg.gemm(wq, xq), lambda: pkg.gemm(o["pw"], xq),
                 lambda: pkg.gemv(o["wq"], o["xq"].cpu()), lambda: pkg.gemm(o["wq"].cpu(), o["xq"]),
                 lambda: pkg.rms_norm(o["x"], 1e-5, out=cuda.zeros(8, 128))):
        with pytest.raises(TypeError):
            call()
    pkg.check_device_errors()


def test_a_package_under_a_second_name_raises_its_own_errors(cuda, pkg, operands):
    import importlib

    other = importlib.import_module("tianchen-rv_b200")
    assert other is not pkg and other.TcrvCudaError is not pkg.TcrvCudaError
    narrow = cuda.empty(144, device="cuda")  # one dimension: a row stride of 1 for rows of 3 floats
    for p in (pkg, other, pkg):
        with pytest.raises(p.TcrvCudaError) as e:
            p.gemv(operands["wq"], operands["xq"], out=narrow)
        assert e.value.status == -1


# (what is wrong, the call, the error): every check that a call makes before it launches
REFUSED = [
    ("not a tensor", lambda p, c, o: p.vec_silu([1.0]), TypeError),
    ("host memory", lambda p, c, o: p.vec_silu(o["x"].cpu()), TypeError),
    ("element type", lambda p, c, o: p.vec_silu(o["x"].double()), TypeError),
    ("element type of the output", lambda p, c, o: p.gemv(o["wq"], o["xq"], out=c.empty(48, 3, dtype=c.int32, device="cuda")), TypeError),
    ("strided input", lambda p, c, o: p.vec_silu(o["x"][:, ::2]), ValueError),
    ("strided output", lambda p, c, o: p.gemv(o["wq"], o["xq"], out=c.empty(48, 6, device="cuda")[:, ::2]), ValueError),
    ("types of the addends", lambda p, c, o: p.add(o["x"], o["x"].int()), TypeError),
    ("a type without a sum", lambda p, c, o: p.add(o["x"].half(), o["x"].half()), TypeError),
    ("bytes that are no whole blocks", lambda p, c, o: p.dequantize_q8_0(o["xq"][:, :35].contiguous()), ValueError),
    ("blocks without rows", lambda p, c, o: p.dequantize_q8_0(o["xq"][0, 0]), ValueError),
    ("floats that are no whole blocks", lambda p, c, o: p.quantize_q8_0(o["x"][:, :33].contiguous()), ValueError),
    ("weights of one dimension", lambda p, c, o: p.gemv(o["wq"][0], o["xq"]), ValueError),
    ("row lengths", lambda p, c, o: p.gemv(o["wq"][:, :54], o["xq"]), ValueError),
    ("weight format", lambda p, c, o: p.gemv(o["wq"], o["xq"], q8_weights=True), ValueError),
    ("row lengths", lambda p, c, o: p.gemm(o["wq"][:, :54], o["xq"]), ValueError),
    ("activations of one dimension", lambda p, c, o: p.gemm(o["wq"], o["xq"][0]), ValueError),
    ("prepared row lengths", lambda p, c, o: p.gemm(o["pw"], o["xq"][:, :102]), ValueError),
    ("activations of one dimension", lambda p, c, o: p.gemm(o["pw"], o["xq"][0]), ValueError),
    ("row lengths", lambda p, c, o: p.sibling_dot_rows(2, o["sw"], o["sx"][:, :102].contiguous()), ValueError),
    ("rows that are not contiguous", lambda p, c, o: p.rms_norm(o["x"].t(), 1e-5), ValueError),
    ("rows of another type", lambda p, c, o: p.rope_apply(o["x"].double(), o["cache"]), ValueError),
    ("type of the angles", lambda p, c, o: p.rope_apply(o["x"], o["cache"].double()), TypeError),
    ("rows of the interleaved layout", lambda p, c, o: p.repack_gemv(o["w16"], o["xq"][0], 47), ValueError),
    ("scale that is no number", lambda p, c, o: p.vec_scale_(o["x"].clone(), "2"), TypeError),
    ("flags that are no number", lambda p, c, o: p.gemv(o["wq"], o["xq"], flags="strict"), TypeError),
]


@pytest.mark.parametrize("what,call,error", REFUSED, ids=[f"{i}: {r[0]}" for i, r in enumerate(REFUSED)])
def test_operands_that_do_not_fit_are_refused(cuda, pkg, operands, what, call, error):
    with pytest.raises(error):
        call(pkg, cuda, operands)


def test_statuses_of_the_c_entries_become_errors(cuda, pkg, operands):
    o = operands
    small = cuda.empty(256, dtype=cuda.uint8, device="cuda")
    for call, status in [(lambda: pkg.gemm(o["wq"], o["xq"], workspace=small), -5), (lambda: pkg.gemm(o["pw"], o["xq"], workspace=small), -5),
                         (lambda: pkg.rms_norm(o["x"], 1e-5, flags=64), -1), (lambda: pkg.rope_apply(o["x"][:, :127], o["cache"]), -1)]:
        with pytest.raises(pkg.TcrvCudaError) as e:
            call()
        assert e.value.status == status
    # (a native function has a fixed number of arguments)
    with pytest.raises(TypeError):
        pkg._native.vec_silu(o["x"])
