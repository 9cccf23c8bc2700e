"""FP64 contractions that take scratch, on a stream the library has not seen, while another thread
captures a CUDA graph in the default (global) mode: the call runs and the capture stays valid."""
import ctypes
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.complex128])
def test_beside_a_capture(dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import einsums_gb300 as eg
    from einsums_gb300 import _lib
    lib = _lib.load()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    A, B = (torch.randn(s, generator=gen, dtype=dtype, device="cuda") for s in ((700, 600), (600, 500)))
    C = torch.zeros((700, 500), dtype=dtype, device="cuda")
    want = A @ B
    small = torch.randn((30, 30), generator=gen, dtype=torch.float64, device="cuda")
    out = torch.zeros_like(small)
    eg.einsum(0.0, "ij", out, 1.0, "ik", small, "kj", small)  # the library is loaded
    # the scratch has to be allocated anew
    p = ctypes.c_void_p()
    _lib.check(lib.eg_set_memory_budget(1))
    lib.eg_device_alloc(1 << 20, ctypes.byref(p))
    _lib.check(lib.eg_set_memory_budget(0))
    fresh = ctypes.c_ulonglong()
    torch.cuda.cudart().cudaStreamCreate(ctypes.addressof(fresh))
    torch.cuda.synchronize()
    before, after, fails = ctypes.c_uint64(), ctypes.c_uint64(), []

    def other():
        try:
            lib.eg_kernel_launches(ctypes.byref(before))
            eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B, stream=fresh.value)
            lib.eg_kernel_launches(ctypes.byref(after))
        except Exception as e:  # noqa: BLE001
            fails.append(e)

    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        eg.einsum(0.0, "ij", out, 2.0, "ik", small, "kj", small)
        t = threading.Thread(target=other)
        t.start()
        t.join()
    assert not fails
    out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.allclose(out, 2 * small @ small, rtol=0, atol=1e-11)
    assert torch.allclose(C, want, rtol=0, atol=1e-10)
    assert after.value - before.value >= 3  # split, tensor kernel, FMA kernel for what it leaves
    torch.cuda.cudart().cudaStreamDestroy(fresh.value)
