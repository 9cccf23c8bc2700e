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


def replay_us(plan):
    times = []
    for _ in range(9):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        plan.execute()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 1e3)
    return sorted(times)[4]


def test_lists(eg):
    """An uneven list: all graded, every second item, and magnitudes that are worth a try but fail."""
    from einsums_gb300 import _lib, workloads
    lib = _lib.load()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    normal = lambda *s: torch.randn(s, generator=gen, dtype=torch.float64, device="cuda")
    shapes = workloads.batched_shapes(512, seed=5)
    used = ctypes.c_size_t()
    for kind in ("graded", "half", "apart"):
        As, Bs = [], []
        for q, (i, j, a, b) in enumerate(shapes):
            A, B = normal(i, j, a), normal(i, j, b)
            if kind == "apart":  # two fifths of the summed indices each, elements of the other 1e-5
                at = torch.arange(i * j, device="cuda").view(i, j, 1) * 5 // (i * j)
                A, B = torch.where(at < 2, A, A * 1e-5), torch.where(at > 2, B, B * 1e-5)
            elif kind == "graded" or q % 2:
                d = 10.0 ** torch.linspace(-9, 9, i * j, dtype=torch.float64, device="cuda").view(i, j, 1)
                A, B = A * d, B / d
            As.append(A.contiguous()), Bs.append(B.contiguous())
        Cs = [torch.full((a, b), float("nan"), dtype=torch.float64, device="cuda") for i, j, a, b in shapes]
        plan = eg.GroupedPlan(0.0, "ab", Cs, 1.0, "ija", As, "ijb", Bs)
        plan.execute()
        torch.cuda.synchronize()
        for q in range(0, 512, 3):
            i, j, a, b = shapes[q]
            x, y = As[q].reshape(i * j, a).cpu().numpy(), Bs[q].reshape(i * j, b).cpu().numpy()
            want = (x.T.astype(np.longdouble) @ y.astype(np.longdouble)).astype(float)
            assert np.all(np.abs(Cs[q].cpu().numpy() - want) <= (i * j + 4) * U * (np.abs(x.T) @ np.abs(y))), (kind, q)
        ours = replay_us(plan)
        plan.close()
        _lib.check(lib.eg_memory_in_use(ctypes.byref(used)))
        try:
            _lib.check(lib.eg_set_memory_budget(used.value + (16 << 20)))
            plan = eg.GroupedPlan(0.0, "ab", Cs, 1.0, "ija", As, "ijb", Bs)
            plain = replay_us(plan)
            plan.close()
        finally:
            _lib.check(lib.eg_set_memory_budget(0))
        if kind != "apart":
            assert ours <= 1.1 * plain, (kind, ours, plain)
        print(kind, ours, plain)


@pytest.mark.parametrize("m,n,k", [(4000, 2100, 300), (300, 260, 4100), (100000, 24, 33)])
def test_not_tried_in_vain(eg, m, n, k):
    """Operands whose magnitudes say that nothing can pass are left to the FMA kernel at once, whole
    tiles and tiles cut along K; then ordinary and sparse ones with the same scratch are not."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(k)
    A, B = graded(gen, m, n, k)
    C = torch.full((m, n), float("nan"), dtype=torch.float64, device="cuda")
    call = lambda: eg.einsum(0.0, "ij", C, 1.0, "ik", A, "kj", B)
    tensor = {}
    for kind in ("graded", "ordinary", "sparse", "graded again"):
        if kind == "ordinary":
            gA, gB = A, B
            A, B = (torch.randn(x.shape, generator=gen, dtype=torch.float64, device="cuda") for x in (A, B))
        elif kind == "sparse":  # a tenth of A's elements
            A = A * (torch.rand(A.shape, generator=gen, device="cuda") < 0.1)
        elif kind == "graded again":
            A, B = gA, gB
        tensor[kind] = profiled(call)["k_tc_split_gemm_f64"]
        rows = np.arange(0, m, max(1, m // 40))
        a, b = A[rows].cpu().numpy(), B.cpu().numpy()
        want = (a.astype(np.longdouble) @ b.astype(np.longdouble)).astype(float)
        assert np.all(np.abs(C[rows].cpu().numpy() - want) <= (k + 4) * U * (np.abs(a) @ np.abs(b))), kind
    # without loads and products (an eighth and less of the time): the kernel's start and the listing
    assert max(tensor["graded"], tensor["graded again"]) <= 0.25 * tensor["ordinary"]
    assert tensor["sparse"] >= 0.5 * tensor["ordinary"]
