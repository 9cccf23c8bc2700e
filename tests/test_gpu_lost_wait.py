"""What follows a device wait of the tensor kernel that gave up, made on the host (eg_selftest_lose_next
sets the call's record, the kernels run undisturbed): FP64 outputs are NaN throughout, the split form
adds up no slices, the record reaches the stream that ran the call, and the next call is right again."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
TIMEOUT = 7


@pytest.fixture(scope="module")
def eg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import einsums_gb300
    from einsums_gb300 import build
    build.build()
    return einsums_gb300


@pytest.fixture(scope="module")
def lib():
    from einsums_gb300 import _lib, build
    build.build()
    return _lib.load()


def status(lib, stream):
    code = ctypes.c_int32(-1)
    st = lib.eg_stream_status(ctypes.c_void_p(stream.cuda_stream), ctypes.byref(code))
    assert st == (TIMEOUT if code.value else 0)
    return code.value


def normal(seed, *shape, dtype=torch.float64):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, dtype=dtype, device="cuda")


def test_codes(lib):
    assert lib.eg_selftest_lose_next(-1) == 1 and lib.eg_selftest_lose_next(128) == 1
    assert lib.eg_selftest_lose_next(5) == 0 and lib.eg_selftest_lose_next(0) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,m,n,k", [(torch.float64, 2000, 1300, 300), (torch.float64, 256, 200, 4100),
                                         (torch.float64, 70, 5000, 200), (torch.complex128, 300, 170, 257)])
def test_fp64(eg, lib, dtype, m, n, k):
    A, B = normal(1, m, k, dtype=dtype), normal(2, k, n, dtype=dtype)
    s = torch.cuda.Stream()
    C = torch.zeros((m, 2 * n), dtype=dtype, device="cuda")[:, ::2]
    torch.cuda.synchronize()
    assert lib.eg_selftest_lose_next(9) == 0
    eg.einsum(1.0, "ij", C, 1.0, "ik", A, "kj", B, stream=s)
    s.synchronize()
    parts = torch.view_as_real(C) if dtype == torch.complex128 else C
    assert bool(torch.isnan(parts).all())
    assert status(lib, torch.cuda.current_stream()) == 0
    assert status(lib, s) == 9
    eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B, stream=s)
    s.synchronize()
    assert status(lib, s) == 0
    assert torch.allclose(C, A @ B, rtol=0, atol=1e-10)


@pytest.mark.gpu
def test_split_adds_up_no_slices(eg, lib):
    A, B, C0 = normal(3, 256, 4096), normal(4, 4096, 256), normal(5, 256, 256)
    C = C0.clone()
    assert lib.eg_selftest_lose_next(11) == 0
    eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B, precision="split_bf16")
    torch.cuda.synchronize()
    assert torch.equal(C, C0)  # every tile is cut along K here
    assert status(lib, torch.cuda.current_stream()) == 11
    eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B, precision="split_bf16")
    torch.cuda.synchronize()
    assert torch.allclose(C, A @ B, rtol=0, atol=1e-7)


@pytest.mark.gpu
def test_lists(eg, lib):
    As = [normal(q, 200 + q % 7, 60 + q % 50) for q in range(400)]
    Bs = [normal(1000 + q, 200 + q % 7, 40 + q % 90) for q in range(400)]
    Cs = [torch.zeros((A.shape[1], B.shape[1]), dtype=torch.float64, device="cuda") for A, B in zip(As, Bs)]
    assert lib.eg_selftest_lose_next(13) == 0
    plan = eg.GroupedPlan(0.0, "ab", Cs, 1.0, "ka", As, "kb", Bs)  # every replay of this plan loses
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for s in streams + streams:
        for C in Cs:
            C.zero_()
        torch.cuda.synchronize()
        plan.execute(stream=s)
        s.synchronize()
        assert all(bool(torch.isnan(C).all()) for C in Cs)
        assert [status(lib, t) for t in streams] == [13 if t is s else 0 for t in streams]
        assert status(lib, torch.cuda.current_stream()) == 0
    plan.close()
    plan = eg.GroupedPlan(0.0, "ab", Cs, 1.0, "ka", As, "kb", Bs)
    plan.execute()
    torch.cuda.synchronize()
    assert status(lib, torch.cuda.current_stream()) == 0
    for A, B, C in zip(As, Bs, Cs):
        assert torch.allclose(C, A.T @ B, rtol=0, atol=1e-10)
    plan.close()
