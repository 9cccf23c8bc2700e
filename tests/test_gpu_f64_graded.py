"""FP64 contractions whose rows are graded against each other, so that nearly every output fails the
accuracy check of the tensor cores and is computed by the FMA kernel: correct, and never much slower
than without the tensor cores (a memory budget keeps them out)."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.fixture(scope="module")
def eg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import einsums_gb300
    from einsums_gb300 import build
    build.build()
    return einsums_gb300


def profiled(f):
    """{kernel: microseconds a launch} of three runs of f."""
    from einsums_gb300 import _lib
    lib = _lib.load()
    buf = ctypes.create_string_buffer(1 << 16)
    f()
    torch.cuda.synchronize()
    lib.eg_profile_enable(1)
    lib.eg_profile_reset()
    try:
        for _ in range(3):
            f()
        torch.cuda.synchronize()
        _lib.check(lib.eg_profile_summary(buf, len(buf)))
    finally:
        lib.eg_profile_enable(0)
    rows = (line.split(",") for line in buf.value.decode().split())
    return {name: float(ms) / 3 * 1e3 for name, _, ms in rows}


def without_scratch(f):
    """f() under a memory budget that leaves the library none to allocate."""
    from einsums_gb300 import _lib
    lib = _lib.load()
    used, p = ctypes.c_size_t(), ctypes.c_void_p()
    _lib.check(lib.eg_set_memory_budget(1))
    try:
        assert lib.eg_device_alloc(1 << 20, ctypes.byref(p)) != 0  # the shared scratch is given back
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        _lib.check(lib.eg_set_memory_budget(used.value + (1 << 20)))
        return f()
    finally:
        _lib.check(lib.eg_set_memory_budget(0))


def graded(gen, m, n, k):
    d = 10.0 ** torch.linspace(-9, 9, k, dtype=torch.float64, device="cuda")
    A = torch.randn((m, k), generator=gen, dtype=torch.float64, device="cuda") * d
    return A, torch.randn((k, n), generator=gen, dtype=torch.float64, device="cuda") / d[:, None]


@pytest.mark.parametrize("m,n,k", [(120000, 75, 75), (20000, 57, 130), (3000, 200, 500)])
def test_narrow_outputs(eg, m, n, k):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(m)
    A, B = graded(gen, m, n, k)
    C = torch.full((m, n), float("nan"), dtype=torch.float64, device="cuda")
    call = lambda: eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B)
    times = profiled(call)
    assert "k_tc_split_gemm_f64" in times
    rows = np.arange(0, m, m // 50)
    a, b = A[rows].cpu().numpy(), B.cpu().numpy()
    want = (a.astype(np.longdouble) @ b.astype(np.longdouble)).astype(float)
    assert np.all(np.abs(C[rows].cpu().numpy() - want) <= (k + 4) * U * (np.abs(a) @ np.abs(b)))
    plain = without_scratch(lambda: profiled(call))
    assert set(plain) == {"k_contract_f64"}
    # the listed blocks are all of the output, in tiles of as many outputs: a fifth more for their order
    assert times["k_contract_f64_listed"] <= 1.2 * plain["k_contract_f64"]
