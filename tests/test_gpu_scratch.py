"""The scratch of FP64 contractions on the tensor cores: a stream that is held up does not hold up
another one's contraction, and a size that cannot be had leaves the buffer of smaller ones alone."""
import ctypes
import time

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import einsums_gb300
    from einsums_gb300 import build
    build.build()
    einsums_gb300.trim_memory()  # buffers of other tests
    return einsums_gb300


def operands(dtype, m, n, k):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m + n)
    A, B = (torch.randn(s, generator=gen, dtype=dtype, device="cuda") for s in ((m, k), (k, n)))
    return A, B, A @ B


@pytest.mark.parametrize("dtype,m,n,k", [(torch.float64, 700, 500, 600), (torch.complex128, 300, 170, 257),
                                         (torch.complex128, 40, 30, 50)])
def test_streams_apart(eg, dtype, m, n, k):
    A, B, want = operands(dtype, m, n, k)
    streams = [torch.cuda.Stream() for _ in range(3)]
    Cs = [torch.zeros_like(want) for _ in streams]
    for C, s in zip(Cs, streams):  # every stream has run a call before
        eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B, stream=s)
        torch.cuda.synchronize()
        C.zero_()
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(3_000_000_000)  # about 1.5 s at the highest clock
    start = time.perf_counter()
    for C, s in zip(Cs, streams):
        eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B, stream=s)
    streams[1].synchronize()
    streams[2].synchronize()
    apart = time.perf_counter() - start
    held = not streams[0].query()
    for C in Cs[1:]:
        assert torch.allclose(C, want, rtol=0, atol=1e-10)
    torch.cuda.synchronize()
    assert torch.allclose(Cs[0], want, rtol=0, atol=1e-10)
    assert held and apart < 1.0


def test_small_buffers_stay(eg):
    """A stream's larger contraction while another stream is held up, with smaller buffers held: none of
    them is freed, which would wait for the device."""
    small, large = operands(torch.float64, 600, 500, 400), operands(torch.float64, 2500, 2000, 600)
    s, t = torch.cuda.Stream(), torch.cuda.Stream()
    eg.trim_memory()
    C, D = torch.zeros_like(small[2]), torch.zeros_like(large[2])
    eg.einsum(0.0, "ij", C, 1.0, "ik", small[0], "kj", small[1], stream=s)
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        torch.cuda._sleep(3_000_000_000)
    start = time.perf_counter()
    eg.einsum(0.0, "ij", D, 1.0, "ik", large[0], "kj", large[1], stream=t)
    t.synchronize()
    apart, held = time.perf_counter() - start, not s.query()
    torch.cuda.synchronize()
    assert torch.allclose(D, large[2], rtol=0, atol=1e-10)
    assert held and apart < 1.0


def test_too_large_a_size_takes_nothing_away(eg):
    from einsums_gb300 import _lib
    lib = _lib.load()
    small, large = operands(torch.float64, 600, 500, 400), operands(torch.float64, 6000, 5000, 900)
    used, p = ctypes.c_size_t(), ctypes.c_void_p()

    def run(x):
        A, B, want = x
        C = torch.zeros_like(want)
        eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B)
        torch.cuda.synchronize()
        assert torch.allclose(C, want, rtol=0, atol=1e-10)
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        return used.value

    _lib.check(lib.eg_set_memory_budget(1))
    assert lib.eg_device_alloc(1 << 20, ctypes.byref(p)) != 0  # what was held is given back
    _lib.check(lib.eg_set_memory_budget(0))
    before = run(small)
    try:
        _lib.check(lib.eg_set_memory_budget(before + (32 << 20)))
        assert run(large) == before  # on the FMA kernel
        assert run(small) == before
    finally:
        _lib.check(lib.eg_set_memory_budget(0))
    after = run(large)
    assert after > before
    assert run(small) == after


def test_trim_gives_back_scratch_and_kept_plans(eg):
    from einsums_gb300 import _lib
    lib = _lib.load()
    A, B, want = operands(torch.float64, 900, 800, 700)
    C = torch.zeros_like(want)
    As = [A[:, 10 * q:10 * q + 60 + q % 9].contiguous() for q in range(60)] * 6
    Bs = [A[:, 5 * q:5 * q + 50 + q % 7].contiguous() for q in range(60)] * 6
    Cs = [torch.zeros((a.shape[1], b.shape[1]), dtype=torch.float64, device="cuda") for a, b in zip(As, Bs)]
    used = ctypes.c_size_t()

    def in_use():
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        return used.value

    eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B)  # (the workspace of this stream, which stays, is there)
    eg.trim_memory()
    before = in_use()
    for _ in range(2):
        C.zero_()
        eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B)
        scratch = in_use()
        assert scratch >= before + (64 << 20)
        plan = eg.compile_plan("ab", "ka", "kb")
        plan.execute(0.0, Cs, 1.0, As, Bs)
        assert in_use() > scratch + (16 << 20)
        eg.trim_memory()  # with both still under way
        assert in_use() == before
        assert torch.allclose(C, want, rtol=0, atol=1e-10)
        for a, b, c in zip(As, Bs, Cs):
            assert torch.allclose(c, a.T @ b, rtol=0, atol=1e-10)
            c.zero_()


def test_kept_plans_make_room(eg):
    """An allocation that fails while list plans are kept gets their memory."""
    from einsums_gb300 import _lib
    lib = _lib.load()
    A, _, _ = operands(torch.float64, 900, 800, 700)
    As = [A[:, 10 * q:10 * q + 60].contiguous() for q in range(60)] * 6
    Cs = [torch.zeros((60, 60), dtype=torch.float64, device="cuda") for _ in As]
    eg.trim_memory()
    used, p = ctypes.c_size_t(), ctypes.c_void_p()
    _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
    before = used.value
    eg.compile_plan("ab", "ka", "kb").execute(0.0, Cs, 1.0, As, As)
    try:
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        assert used.value > before + (16 << 20)
        _lib.check(lib.eg_set_memory_budget(used.value + 4096))
        _lib.check(lib.eg_device_alloc(16 << 20, ctypes.byref(p)))
        _lib.check(lib.eg_device_free(p))
    finally:
        _lib.check(lib.eg_set_memory_budget(0))
    for a, c in zip(As, Cs):
        assert torch.allclose(c, a.T @ a, rtol=0, atol=1e-10)


def test_plans_do_not_push_scratch_out(eg):
    """An FP64 list plan that does not fit beside the scratch takes the FMA kernel, whatever is held."""
    from einsums_gb300 import _lib
    lib = _lib.load()
    A, B, want = operands(torch.float64, 3000, 2500, 900)
    C = torch.zeros_like(want)
    As = [A[:, 10 * q:10 * q + 60].contiguous() for q in range(60)] * 6
    Cs = [torch.zeros((60, 60), dtype=torch.float64, device="cuda") for _ in As]
    used, n = ctypes.c_size_t(), ctypes.c_uint64()
    eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B)  # some scratch
    torch.cuda.synchronize()
    _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
    before = used.value
    try:
        _lib.check(lib.eg_set_memory_budget(before + (16 << 20)))
        plan = eg.GroupedPlan(0.0, "ab", Cs, 1.0, "ka", As, "kb", As)
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        assert before < used.value < before + (16 << 20)
        _lib.check(lib.eg_kernel_launches(ctypes.byref(n)))
        start = n.value
        plan.execute()
        _lib.check(lib.eg_kernel_launches(ctypes.byref(n)))
        assert n.value - start == 1
    finally:
        _lib.check(lib.eg_set_memory_budget(0))
    torch.cuda.synchronize()
    for a, c in zip(As, Cs):
        assert torch.allclose(c, a.T @ a, rtol=0, atol=1e-9)
    plan.close()
