"""Tiles cut along K: with and without the scratch for their slices (a memory budget that holds
the digit planes only) the split form gives the same bits, at output edges and with C_prefactor."""
import ctypes

import numpy as np
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
    return einsums_gb300


@pytest.mark.parametrize("m,n,k", [(256, 256, 4096), (255, 70, 4100), (129, 257, 2048)])
def test_without_room_for_slices(eg, m, n, k):
    from einsums_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(m + n)
    A, B, C0 = (torch.from_numpy(rng.standard_normal(s)).cuda() for s in ((m, k), (k, n), (m, n)))
    buf = ctypes.create_string_buffer(1 << 16)

    def run():  # on a stream of its own: its workspace is allocated in the call
        C, s = C0.clone(), torch.cuda.Stream()
        torch.cuda.synchronize()
        lib.eg_profile_enable(1)
        lib.eg_profile_reset()
        try:
            eg.einsum(0.5, "ij", C, -3.0, "ik", A, "kj", B, precision="split_bf16", stream=s)
            s.synchronize()
            _lib.check(lib.eg_profile_summary(buf, len(buf)))
        finally:
            lib.eg_profile_enable(0)
        return C.cpu().numpy(), buf.value.decode()

    want, kernels = run()
    assert "k_tc_finish_slices" in kernels
    used, p = ctypes.c_size_t(), ctypes.c_void_p()
    _lib.check(lib.eg_set_memory_budget(1))
    try:
        assert lib.eg_device_alloc(1 << 20, ctypes.byref(p)) != 0  # the shared scratch is given back
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        planes = 5 * 2 * (m + n + 256) * (k + 64)  # rows padded to 128
        _lib.check(lib.eg_set_memory_budget(used.value + planes + (26 << 20)))
        got, kernels = run()
    finally:
        _lib.check(lib.eg_set_memory_budget(0))
    assert "k_tc_split_gemm" in kernels and "k_tc_finish_slices" not in kernels
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
